"""The tensor schedules with the last row groups' gene windows cut between CTAs, against the oracle and against themselves uncut."""
import numpy as np
import pytest
import torch

from cellerator_b200 import capi, ops
from conftest import random_csr
from gpu_util import dense, host_pack, row_l1, rows_of, to_dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("schedule,bits,n,dtype,multiply", [
    ("tensor_blocked", 8, 64, torch.bfloat16, capi.DTYPE_BF16), ("tensor_blocked", 8, 128, torch.bfloat16, capi.DTYPE_F32),
    ("tensor_blocked", 8, 32, torch.float32, capi.DTYPE_F32), ("tensor_blocked", 8, 64, torch.float32, capi.DTYPE_F32), ("tensor_dense", 4, 64, torch.bfloat16, capi.DTYPE_BF16),
    ("tensor_codes", 4, 128, torch.bfloat16, capi.DTYPE_BF16), ("tensor_codes", 4, 32, torch.bfloat16, capi.DTYPE_BF16)])
@pytest.mark.parametrize("rows,windows,density", [(200, 33, 40), (256 * 6 + 1, 12, 40), (256 * 6 + 1, 17, 400), (256 * 150 - 7, 9, 12)])
def test_cut_groups(cuda_device, oracle, monkeypatch, schedule, bits, n, dtype, multiply, rows, windows, density):
    """One group, a few (an even and an odd number of windows; short and long segments), two more than the SMs: whole groups first, the cut ones after."""
    monkeypatch.setitem(ops.SCHEDULE_REQUEST, capi.PROJECTION_CSR, schedule)
    rng = np.random.default_rng(rows + windows + n)
    cols = 128 * windows - 50
    c = host_pack(oracle, random_csr(rng, rows=rows, cols=cols, max_nnz=min(density, cols), bits=bits, policy=1))
    x = to_dev(c, cuda_device)
    w, w_host = dense(rng, cols, n, dtype, cuda_device)
    op = ops.PreparedSpmm(capi.PROJECTION_CSR, rows, cols, n, x.nnz, bits, 1, dtype, cuda_device, host_row_ptr=x.host_row_ptr,
                          multiply=multiply, device_matrix=x)
    assert op.schedule.startswith(schedule)
    ref = oracle.qcsr_forward(bits, 1, c["row_ptr"], c["packed_row_ptr"], c["col_idx"], c["packed"], c["scales"], c["offsets"], w_host, cols)
    # (a row of one entry can lie next to its zero-point's negative, and fp16 rounds both)
    scale = (row_l1(oracle, c)[0][:, None] + 0.1) * float(np.abs(w_host).max())
    bound = (1e-2 if multiply == capi.DTYPE_BF16 else 1e-4) * scale
    y = op.run(x, w, torch.full((rows, n), float("nan"), device=cuda_device))
    assert op.status() == 0
    assert np.all(np.abs(y.cpu().numpy() - ref) <= bound)
    assert torch.equal(y, op.run(x, w, torch.empty_like(y)))
    out = torch.full_like(y, -3.0)                                     # a shard cuts its groups as the whole launch does
    lo, hi = (rows // 512) * 256, rows - 5
    op.run(x, w, out, row_begin=lo, row_end=hi)
    assert torch.equal(out[lo:hi], y[lo:hi]) and torch.all(out[:lo] == -3.0) and torch.all(out[hi:] == -3.0)
    y0 = torch.from_numpy(rng.normal(size=(rows, n)).astype(np.float32)).to(cuda_device)
    assert torch.allclose(op.run(x, w, y0.clone(), alpha=2.0, beta=0.5), 2.0 * y + 0.5 * y0, rtol=1e-5, atol=1e-6)
    bias = torch.from_numpy(rng.normal(size=n).astype(np.float32)).to(cuda_device)
    relu = op.run(x, w, torch.empty_like(y), epilogue="bias_relu", bias=bias)
    assert torch.allclose(relu, torch.relu(y + bias), rtol=1e-5, atol=1e-6)
    op.workspace_bytes -= 1                                            # no room for the sums of parts: no group is cut
    uncut = op.run(x, w, torch.empty_like(y)).cpu().numpy()
    assert np.all(np.abs(uncut - y.cpu().numpy()) <= 1e-4 * scale)
    if schedule == "tensor_blocked":                                   # room for N columns of W: an fp32 W is multiplied in three passes
        op.workspace_bytes = 256 + windows * 128 * (2 * n + 8)
        narrow = op.run(x, w, torch.empty_like(y)).cpu().numpy()
        assert np.all(np.abs(narrow - y.cpu().numpy()) <= 1e-4 * scale)
    op.close()


@pytest.mark.parametrize("schedule,bits,n,dtype,multiply", [
    ("tensor_blocked", 8, 32, torch.bfloat16, capi.DTYPE_BF16), ("tensor_blocked", 8, 64, torch.bfloat16, capi.DTYPE_BF16),
    ("tensor_blocked", 4, 128, torch.bfloat16, capi.DTYPE_BF16), ("tensor_blocked", 8, 64, torch.bfloat16, capi.DTYPE_F32),
    ("tensor_blocked", 8, 32, torch.float32, capi.DTYPE_F32), ("tensor_blocked", 8, 64, torch.float32, capi.DTYPE_F32),
    ("tensor_blocked", 8, 128, torch.float32, capi.DTYPE_F32), ("tensor_dense", 8, 32, torch.bfloat16, capi.DTYPE_BF16),
    ("tensor_dense", 4, 64, torch.bfloat16, capi.DTYPE_BF16), ("tensor_dense", 8, 128, torch.bfloat16, capi.DTYPE_BF16),
    ("tensor_codes", 4, 32, torch.bfloat16, capi.DTYPE_BF16), ("tensor_codes", 4, 64, torch.bfloat16, capi.DTYPE_BF16),
    ("tensor_codes", 4, 128, torch.bfloat16, capi.DTYPE_BF16)])
@pytest.mark.parametrize("rows,windows,density", [(256 * 6 + 1, 7, 40), (256 * 6 + 1, 9, 300), (700, 17, 40), (256 * 150 - 7, 9, 12), (1800, 33, 1200),
                                                  (256 * 13, 64, 60), (256 * 47 + 3, 129, 15), (300, 200, 4000)])
def test_a_rows_bits_follow_from_its_entries(cuda_device, oracle, monkeypatch, schedule, bits, n, dtype, multiply, rows, windows, density):
    """The same bits in the whole matrix, in shards that are matrices of their own, and without room for the sums of parts: every
    number of parts and of parts to a CTA, whole groups beside cut ones, short and long segments."""
    monkeypatch.setitem(ops.SCHEDULE_REQUEST, capi.PROJECTION_CSR, schedule)
    rng = np.random.default_rng(rows + windows + n)
    cols = 128 * windows - 50
    c = host_pack(oracle, random_csr(rng, rows=rows, cols=cols, max_nnz=min(density, cols), bits=bits, policy=1))
    w, _ = dense(rng, cols, n, dtype, cuda_device)

    def project(c, uncut=False, narrow=False):
        x = to_dev(c, cuda_device)
        op = ops.PreparedSpmm(capi.PROJECTION_CSR, c["rows"], cols, n, x.nnz, bits, 1, dtype, cuda_device, host_row_ptr=x.host_row_ptr,
                              multiply=multiply, device_matrix=x)
        assert op.schedule.startswith(schedule)
        # the status block and the records of W, hi and lo of an fp32 W side by side; behind them the tables of the code tiles
        records = 256 + windows * 128 * (2 * n * (2 if dtype == torch.float32 and n <= 64 else 1) + 8) + (windows * 544 if schedule == "tensor_codes" else 0)
        if uncut and op.workspace_bytes > records:
            op.workspace_bytes = records
        if narrow:                                                     # room for N columns of W
            op.workspace_bytes = 256 + windows * 128 * (2 * n + 8)
        y = op.run(x, w, torch.empty(c["rows"], n, device=cuda_device))
        assert op.status() == 0
        op.close()
        return y

    y = project(c)
    assert torch.equal(project(c, uncut=True), y)
    if dtype == torch.float32:
        assert torch.equal(project(c, narrow=True), y)
    cuts = sorted({0, 1, 290, 556, rows // 2 + 100, rows} & set(range(rows + 1)))
    for lo, hi in zip(cuts[:-1], cuts[1:]):
        assert torch.equal(project(rows_of(c, lo, hi)), y[lo:hi])
