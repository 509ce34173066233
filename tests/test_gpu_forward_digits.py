"""GPU parity of the forward projection with exact integer sums, at the edges of its tiles, pieces, chunks and shares."""
import numpy as np
import pytest
import torch

from cellerator_b200 import capi, ops
from conftest import random_csr
from gpu_util import dense, host_pack, rows_of, to_dev

pytestmark = pytest.mark.gpu


def prepare(x, n, dtype, device):
    op = ops.PreparedSpmm(capi.PROJECTION_CSR, x.rows, x.cols, n, x.nnz, x.bits, x.policy, dtype, device, schedule="integer_windows")
    assert op.schedule == "integer_windows"
    return op


def reference(oracle, c, w):
    """Y in 64 bits and what bounds the kernel's difference from it.  Per entry: the operands of its gene are rounded to half a step,
    the code's counted up to 255 times, the constant's 127 times; a column's step is at most 2^-31 / 0.48 of its largest
    operand, max(|s|, (|o| + 128 |s|) / 127) |W|.  The oracle decodes with two roundings, at 2^-24 of |s c| <= |v| + |o| and of |v|.
    The sum, alpha and beta round at 2^-24 each."""
    dec = oracle.unpack_csr(c["bits"], c["policy"], c["row_ptr"], c["packed_row_ptr"], c["col_idx"], c["scales"], c["offsets"], c["packed"]).astype(np.float64)
    rows = np.repeat(np.arange(c["rows"]), np.diff(c["row_ptr"]))
    x, size, count = np.zeros((c["rows"], c["cols"])), np.zeros((c["rows"], c["cols"])), np.diff(c["row_ptr"])
    x[rows, c["col_idx"]] = dec
    size[rows, c["col_idx"]] = 2 * np.abs(dec) + np.abs(c["offsets"][c["col_idx"]])
    bias = 128.0 if c["bits"] == 8 else 0.0
    reach = np.maximum(np.abs(c["scales"]), (np.abs(c["offsets"]) + bias * np.abs(c["scales"])) / 127.0).astype(np.float64)
    step = (reach[:, None] * np.abs(w)).max(0) * 2.0 ** -31 / 0.48
    y = x @ w.astype(np.float64)
    return y, count[:, None] * (255 + 127) / 2 * step[None, :] + 2.0 ** -24 * (size @ np.abs(w).astype(np.float64)) + 3 * 2.0 ** -24 * np.abs(y) + 1e-30


@pytest.mark.parametrize("rows,cols,max_nnz", [(1, 100, 90), (31, 129, 60), (255, 1, 1), (257, 128, 90), (256 * 3 + 33, 383, 20), (700, 640, 640),
                                               (4100, 900, 90), (256 * 20 + 1, 1664, 300)])
@pytest.mark.parametrize("n,bits,dtype", [(64, 8, torch.bfloat16), (32, 4, torch.float32), (50, 8, torch.float32), (130, 4, torch.bfloat16), (1, 8, torch.float32)])
def test_against_64_bits(cuda_device, oracle, rows, cols, max_nnz, n, bits, dtype):
    """Fewer rows than a piece, a group and one row, one gene, tiles of several chunks (dense), sixteen and thirty-two rows to a piece,
    groups that several CTAs share and groups they have to themselves, column blocks with a remainder; alpha, beta, an
    epilogue; a row's bits do not follow from the row range, nor from the rows beside it."""
    rng = np.random.default_rng(rows + n + bits)
    c = host_pack(oracle, random_csr(rng, rows=rows, cols=cols, max_nnz=max_nnz, bits=bits, empty_rows=rows > 1))
    x = to_dev(c, cuda_device)
    w, w_host = dense(rng, cols, n, dtype, cuda_device, ld=n + 3)
    op = prepare(x, n, dtype, cuda_device)
    want, bound = reference(oracle, c, w_host)
    y = op.run(x, w, torch.full((rows, n), float("nan"), device=cuda_device))
    assert op.status() == 0
    worst = np.max(np.abs(y.cpu().numpy() - want) / bound)
    assert worst <= 1.0, worst
    lo, hi = rows // 3, max(rows // 3 + 1, rows - rows // 9)             # borders inside groups and pieces
    part = op.run(x, w, torch.full((rows, n), -3.0, device=cuda_device), row_begin=lo, row_end=hi)
    assert torch.equal(part[lo:hi], y[lo:hi]) and torch.all(part[:lo] == -3.0) and torch.all(part[hi:] == -3.0)
    shard = to_dev(rows_of(c, lo, hi), cuda_device)
    if shard.nnz > 0:
        op2 = prepare(shard, n, dtype, cuda_device)
        assert torch.equal(op2.run(shard, w, torch.empty(hi - lo, n, device=cuda_device)), y[lo:hi])
        op2.close()
    init, bias = rng.normal(size=(rows, n)).astype(np.float32), rng.normal(size=n).astype(np.float32)
    got = op.run(x, w, torch.from_numpy(init).to(cuda_device), alpha=2.0, beta=0.5, epilogue="bias_relu", bias=torch.from_numpy(bias).to(cuda_device)).cpu().numpy()
    full = 2.0 * want + 0.5 * init + bias
    assert np.all(np.abs(got - np.maximum(full, 0.0)) <= 2.0 * bound + 2.0 ** -22 * (np.abs(init) + np.abs(bias) + np.abs(full)))
    op.close()


def test_chosen_by_size(cuda_device):
    """From 2 million entries and 200 million products on, and only with zero-points per gene and 3 to 4 % density."""
    def schedule(rows, cols, n, nnz, bits=8, policy=1, dtype=torch.float32):
        op = ops.PreparedSpmm(capi.PROJECTION_CSR, rows, cols, n, nnz, bits, policy, dtype, cuda_device)
        name = op.schedule
        op.close()
        return name
    assert schedule(20_000, 2_000, 32, 6_800_000) == schedule(4_099, 33_538, 50, 7_400_000, dtype=torch.bfloat16) == "integer_windows"
    assert {schedule(20_000, 2_000, 16, 6_800_000), schedule(8_000, 2_000, 32, 2_700_000), schedule(4_099, 33_538, 50, 5_000_000),
            schedule(20_000, 2_000, 32, 6_800_000, policy=2), schedule(200_000, 2_000, 32, 68_000_000)} == {"warp_per_row"}


def test_what_integer_sums_do_not_cover(cuda_device, oracle):
    """Genes that a row holds twice count twice, rows may be in any order; a column with an outlier keeps the others' bits; infinities and
    NaNs reach the rows that hold their genes and no others; so do scales that are not finite."""
    rng = np.random.default_rng(8)
    rows, cols, n = 256 * 5 + 40, 1100, 64
    c = host_pack(oracle, random_csr(rng, rows=rows, cols=cols, max_nnz=100, bits=8))
    for r in range(200, rows, 41):
        lo, hi = c["row_ptr"][r], c["row_ptr"][r + 1]
        c["col_idx"][lo:hi] = rng.permutation(c["col_idx"][lo:hi])
    c["col_idx"][(c["col_idx"] == 300) & (np.arange(len(c["col_idx"])) > len(c["col_idx"]) // 2)] = 303
    w, w_host = dense(rng, cols, n, torch.float32, cuda_device)
    w_host = w_host.copy()

    def check():
        x = to_dev(c, cuda_device)
        op = prepare(x, n, torch.float32, cuda_device)
        got = op.run(x, torch.from_numpy(w_host).to(cuda_device), torch.full((rows, n), float("nan"), device=cuda_device)).cpu().numpy()
        assert op.status() == 0
        op.close()
        with np.errstate(invalid="ignore", over="ignore"):
            dec = oracle.unpack_csr(8, 1, c["row_ptr"], c["packed_row_ptr"], c["col_idx"], c["scales"], c["offsets"], c["packed"]).astype(np.float64)
            r = np.repeat(np.arange(rows), np.diff(c["row_ptr"]))
            want, scale = np.zeros((rows, n)), np.zeros((rows, n))
            for j in range(n):
                np.add.at(want[:, j], r, dec * w_host[c["col_idx"], j])
                np.add.at(scale[:, j], r, (2 * np.abs(dec) + np.abs(c["offsets"][c["col_idx"]])) * np.abs(w_host[c["col_idx"], j]))
            finite = np.isfinite(want)
            assert np.array_equal(np.isnan(got), np.isnan(want)) and np.array_equal(got[np.isinf(want)], want[np.isinf(want)])
            # fixed point: half a step, 2^-30.9 of the largest operand, counts up to 382 times an entry, and the average operand is not more than 2^6
            # below the largest: 2^-15 of it at worst, 2^-19 where, as here, only uniform scales and normal W spread them; else fp32 products,
            # in sums of up to 100: 100 * 2^-24 of them at worst
            assert np.all(np.abs(got[finite] - want[finite]) <= 2.0 ** -19 * scale[finite] + 1e-30)

    check()
    w_host[77, 5] = 1e6
    check()
    w_host[123, 9], w_host[400, 9], w_host[401, 11] = np.inf, -np.inf, np.nan
    check()
    w_host[:] = rng.normal(size=w_host.shape)
    c["scales"][500], c["offsets"][7] = np.nan, np.inf
    check()


@pytest.mark.parametrize("bits,n,dtype", [(8, 64, torch.float32), (4, 50, torch.bfloat16), (8, 33, torch.bfloat16), (4, 100, torch.float32), (8, 3, torch.float32)])
def test_a_wide_operand_gets_the_gather_kernels_bits(cuda_device, oracle, bits, n, dtype):
    """More groups of rows than are resident at a time, a last one that is not full, and a row range."""
    rng = np.random.default_rng(n)
    rows, cols = 8 * 2 * 148 * 2 + 5, 700
    x = to_dev(host_pack(oracle, random_csr(rng, rows=rows, cols=cols, max_nnz=300, bits=bits)), cuda_device)
    w, _ = dense(rng, cols, n, dtype, cuda_device)
    w[5] = 1e6
    gather = ops.PreparedSpmm(capi.PROJECTION_CSR, rows, cols, n, x.nnz, bits, 1, dtype, cuda_device, schedule="warp_per_row")
    op = prepare(x, n, dtype, cuda_device)
    y = gather.run(x, w, torch.empty(rows, n, device=cuda_device))
    assert torch.equal(op.run(x, w, torch.full_like(y, float("nan"))), y) and op.status() == 0
    part = op.run(x, w, torch.full_like(y, -3.0), row_begin=130, row_end=rows - 9)
    assert torch.equal(part[130:-9], y[130:-9]) and torch.all(part[:130] == -3.0) and torch.all(part[-9:] == -3.0)


def test_bounded_wait_path(cuda_device, oracle):
    """The loader of W withholds its copies and every wait gives up: the status says so, and the next launch is correct."""
    rng = np.random.default_rng(4)
    rows, cols, n = 256 * 6, 1000, 64
    c = host_pack(oracle, random_csr(rng, rows=rows, cols=cols, max_nnz=100, bits=8, empty_rows=False))
    x = to_dev(c, cuda_device)
    w, _ = dense(rng, cols, n, torch.bfloat16, cuda_device)
    op = prepare(x, n, torch.bfloat16, cuda_device)
    good = op.run(x, w, torch.empty(rows, n, device=cuda_device)).clone()
    assert op.status() == 0
    capi.lib().cb200_test_arm_wait_timeout(4096)
    try:
        op.run(x, w, torch.empty(rows, n, device=cuda_device))
    finally:
        capi.lib().cb200_test_disarm_wait_timeout()
    with pytest.raises(capi.Cb200Error) as e:
        op.status()
    assert e.value.status == capi.DEVICE_WAIT_TIMEOUT
    assert torch.equal(op.run(x, w, torch.full((rows, n), float("nan"), device=cuda_device)), good) and op.status() == 0
    op.close()
