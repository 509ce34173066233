"""The split-product transpose whose passes over the hi words are one pass over [hi of G | lo of G], against the oracle and against
the three passes that run without room for both parts."""
import numpy as np
import pytest
import torch

from cellerator_b200 import capi, ops
from conftest import random_csr
from gpu_util import dense, host_pack, to_dev
from test_gpu_transpose import assert_transpose_close, col_l1_of

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [32, 64])
@pytest.mark.parametrize("rows,cols,max_nnz", [(256, 100, 30), (256 * 11, 128 * 3, 380), (256 * 40 - 5, 128 * 9 + 1, 60), (256 * 3, 128 * 5, 640)])
def test_pair_of_passes(cuda_device, oracle, monkeypatch, n, rows, cols, max_nnz):
    """One group and more than the ring of pieces of G holds, fewer windows than a set and a ragged last set, several runs
    per window, segments of several chunks, a row range, alpha / beta, repeated runs."""
    monkeypatch.setitem(ops.SCHEDULE_REQUEST, capi.PROJECTION_TRANSPOSE, "tensor_blocked")
    rng = np.random.default_rng(rows + n)
    c = host_pack(oracle, random_csr(rng, rows=rows, cols=cols, max_nnz=max_nnz, bits=8, policy=1))
    x = to_dev(c, cuda_device)
    g, g_host = dense(rng, rows, n, torch.float32, cuda_device, std=1.0, ld=n + 4)
    op = ops.PreparedSpmm(capi.PROJECTION_TRANSPOSE, rows, cols, n, x.nnz, 8, 1, g.dtype, cuda_device, device_matrix=x)
    assert op.schedule == "tensor_blocked_x3"
    cl1, gmax = col_l1_of(oracle, c), float(np.abs(g_host).max())
    init = torch.from_numpy(rng.normal(size=(cols, n)).astype(np.float32)).to(cuda_device)
    room = op.workspace_bytes
    for lo, hi in [(0, rows), (100, rows - 30)]:
        ref = oracle.qcsr_transpose(8, 1, c["row_ptr"], c["packed_row_ptr"], c["col_idx"], c["packed"], c["scales"], c["offsets"], g_host, cols, lo, hi)
        want = 2.0 * ref + 0.5 * init.cpu().numpy()
        got = []
        for op.workspace_bytes in (room, room, room - 1):
            got.append(op.run(x, g, init.clone(), alpha=2.0, beta=0.5, row_begin=lo, row_end=hi))
            assert op.status() == 0
            assert_transpose_close(got[-1].cpu().numpy(), want, 2.0 * cl1 + 1.0, gmax)
        assert torch.equal(got[0], got[1])
        assert float((got[0] - got[2]).abs().max()) <= 1e-4 * gmax * float(cl1.max() + 1.0)
    op.close()
