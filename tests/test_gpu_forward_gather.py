"""GPU parity of the exact gather kernels at the edges of how they cut rows into parts, share them out and read W."""
import numpy as np
import pytest
import torch

from cellerator_b200 import capi, ops
from gpu_util import assert_forward_close, dense, host_pack, row_l1, rows_of, to_dev

pytestmark = pytest.mark.gpu

# around a segment (64), a part (128), the longest row of 16 parts of 128, and beyond it
EDGE_LENGTHS = [0, 1, 15, 16, 17, 63, 64, 65, 127, 128, 129, 255, 257, 2047, 2048, 2049, 3500, 0]


def matrix(oracle, lengths, cols, bits, policy, seed):
    rng = np.random.default_rng(seed)
    row_ptr = np.concatenate([[0], np.cumsum(lengths)]).astype(np.int64)
    col_idx = np.concatenate([np.sort(rng.choice(cols, size=k, replace=False)) for k in lengths]).astype(np.int32)
    offsets = rng.uniform(0.0, 1.0, size=cols if policy == 1 else len(lengths)).astype(np.float32)
    return host_pack(oracle, dict(rows=len(lengths), cols=cols, bits=bits, policy=policy, row_ptr=row_ptr, col_idx=col_idx,
                                  scales=rng.uniform(0.01, 0.05, size=cols).astype(np.float32), offsets=offsets,
                                  values=rng.uniform(0.0, 5.0, size=len(col_idx)).astype(np.float32)))


def check(oracle, device, c, n, dtype, bias=None):
    x = to_dev(c, device)
    w, w_host = dense(np.random.default_rng(n), c["cols"], n, dtype, device)
    op = ops.PreparedSpmm(capi.PROJECTION_CSR, c["rows"], c["cols"], n, x.nnz, c["bits"], c["policy"], dtype, device)
    assert op.schedule == "warp_per_row"
    y = op.run(x, w, torch.full((c["rows"], n), float("nan"), device=device))
    assert op.status() == 0
    ref = oracle.qcsr_forward(c["bits"], c["policy"], c["row_ptr"], c["packed_row_ptr"], c["col_idx"], c["packed"], c["scales"],
                              c["offsets"], w_host, c["cols"])
    l1, _ = row_l1(oracle, c)
    assert_forward_close(y.cpu().numpy(), ref, l1, float(np.abs(w_host).max()), bf16=dtype == torch.bfloat16)
    # a row's sum does not depend on the launch's row range
    lo, hi = c["rows"] // 5, c["rows"] - 2
    part = op.run(x, w, torch.full_like(y, -3.0), row_begin=lo, row_end=hi)
    assert torch.equal(part[lo:hi], y[lo:hi]) and torch.all(part[:lo] == -3.0) and torch.all(part[hi:] == -3.0)


@pytest.mark.parametrize("bits,policy", [(8, 1), (4, 2)])
@pytest.mark.parametrize("n,dtype", [(3, torch.bfloat16), (50, torch.bfloat16), (100, torch.float32), (256, torch.float32),
                                     (300, torch.bfloat16)])
def test_row_lengths_around_the_cuts(cuda_device, oracle, bits, policy, n, dtype):
    check(oracle, cuda_device, matrix(oracle, EDGE_LENGTHS, 4000, bits, policy, 7 * n + bits), n, dtype)


@pytest.mark.parametrize("mean,n", [(4, 64), (90, 16), (90, 50)])
def test_many_rows(cuda_device, oracle, mean, n):
    """a warp per row (short rows; narrow W) and several rows per CTA, with a last CTA that is not full"""
    rows = 64 * 160 + 3
    lengths = np.random.default_rng(mean).integers(0, 2 * mean, size=rows)
    lengths[77] = 700
    check(oracle, cuda_device, matrix(oracle, lengths, 900, 8, 1, mean), n, torch.bfloat16)


@pytest.mark.parametrize("n,dtype", [(50, torch.bfloat16), (50, torch.float32), (101, torch.bfloat16)])
def test_w_re_laid_with_aligned_rows(cuda_device, oracle, n, dtype):
    lengths = np.random.default_rng(1).integers(900, 1300, size=1001)
    c = matrix(oracle, lengths, 4000, 8, 1, n)
    assert c["row_ptr"][-1] >= 1 << 20
    op = ops.PreparedSpmm(capi.PROJECTION_CSR, c["rows"], c["cols"], n, int(c["row_ptr"][-1]), 8, 1, dtype, cuda_device)
    assert op.workspace_bytes > 256
    check(oracle, cuda_device, c, n, dtype)


@pytest.mark.parametrize("bits,policy", [(8, 1), (4, 2)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_a_rows_bits_follow_from_its_entries(cuda_device, oracle, bits, policy, dtype):
    """The same bits in the whole matrix, in shards that are matrices of their own, with and without room to re-lay W, from a W
    whose rows start anywhere, and through the routed call: every width of slices and number of sums per lane."""
    rng = np.random.default_rng(bits)
    lengths = np.concatenate([EDGE_LENGTHS, rng.integers(900, 1300, size=1001), rng.integers(0, 40, size=300)])
    c = matrix(oracle, lengths, 4000, bits, policy, 5)
    assert c["row_ptr"][-1] >= 1 << 20
    x = to_dev(c, cuda_device)
    shards = [(lo, hi, to_dev(rows_of(c, lo, hi), cuda_device)) for lo, hi in ((0, 40), (40, 700), (1019, c["rows"]))]
    for n in (1, 2, 3, 4, 6, 7, 12, 16, 20, 36, 49, 50, 64, 100, 101, 300):
        w, _ = dense(rng, 4000, n, dtype, cuda_device)
        y = ops.spmm_forward(x, w)
        op = ops.PreparedSpmm(capi.PROJECTION_CSR, c["rows"], 4000, n, x.nnz, bits, policy, dtype, cuda_device)
        op.workspace_bytes = 256
        assert torch.equal(op.run(x, w, torch.empty_like(y)), y), n
        op.close()
        odd, _ = dense(rng, 4000, n, dtype, cuda_device, ld=n + 3)
        odd.copy_(w)
        assert torch.equal(ops.spmm_forward(x, odd), y), n
        for lo, hi, part in shards:
            assert torch.equal(ops.spmm_forward(part, w), y[lo:hi]), (n, lo)
        if dtype == torch.float32:
            assert torch.equal(ops.public_projection(x, w), y), n


def test_chunks_of_a_host_call_have_the_matrixs_bits(cuda_device, oracle):
    """W is re-laid for the whole matrix, not for a chunk of it, nor for a chunk of 1,000 rows but for one of 1,300."""
    from test_gpu_fleet_host import _host_forward_all_forms
    c = matrix(oracle, np.random.default_rng(3).integers(900, 1300, size=1301), 4000, 8, 1, 9)
    w, _ = dense(np.random.default_rng(4), 4000, 50, torch.bfloat16, cuda_device)
    y = ops.spmm_forward(to_dev(c, cuda_device), w).cpu().numpy()
    for rows in (300, 1000, 1301):
        got = _host_forward_all_forms(cuda_device, c, w.cpu().pin_memory(), 50, (0,), chunk_rows=rows, chunk_nnz=1_700_000)
        assert np.array_equal(got[0][0].numpy(), y)


@pytest.mark.parametrize("mean", [40, 100])
def test_both_kernels_give_a_row_the_same_bits(cuda_device, oracle, mean):
    """Many short rows, or narrow operands, run with a warp per row (32 or 64 entries at a time); a shard of them by parts."""
    rng = np.random.default_rng(mean)
    c = matrix(oracle, np.concatenate([EDGE_LENGTHS, rng.integers(0, 2 * mean, size=64 * 160)]), 4000, 8, 1, mean)
    x, part = to_dev(c, cuda_device), to_dev(rows_of(c, 0, 600), cuda_device)
    for n, dtype in ((1, torch.float32), (5, torch.bfloat16), (8, torch.float32), (16, torch.bfloat16), (50, torch.bfloat16), (64, torch.float32)):
        w, _ = dense(rng, 4000, n, dtype, cuda_device)
        assert torch.equal(ops.spmm_forward(part, w), ops.spmm_forward(x, w)[:600]), n


@pytest.mark.parametrize("n,dtype", [(64, torch.bfloat16), (130, torch.float32)])
def test_a_rows_bits_in_matrices_of_any_size(cuda_device, oracle, n, dtype):
    """Millions of entries or thousands of them, dense rows, wide W: the whole matrix, shards of a few and of most of its rows, row ranges and a
    launch with the least workspace give a row the same bits."""
    rng = np.random.default_rng(n)
    c = matrix(oracle, rng.integers(300, 700, size=6500), 4000, 8, 1, n)
    x = to_dev(c, cuda_device)
    assert x.nnz >= 3_000_000
    w, _ = dense(rng, 4000, n, dtype, cuda_device)
    y = ops.spmm_forward(x, w)
    op = ops.PreparedSpmm(capi.PROJECTION_CSR, c["rows"], 4000, n, x.nnz, 8, 1, dtype, cuda_device)
    op.workspace_bytes = 256
    assert torch.equal(op.run(x, w, torch.empty_like(y)), y)
    assert torch.equal(op.run(x, w, torch.empty_like(y), row_begin=5, row_end=41)[5:41], y[5:41])
    op.close()
    for lo, hi in ((0, 7), (30, 1500), (1, 6499)):
        assert torch.equal(ops.spmm_forward(to_dev(rows_of(c, lo, hi), cuda_device), w), y[lo:hi]), (lo, hi)


def test_what_reaches_a_row(cuda_device, oracle):
    """Genes that a row holds twice count twice, rows may be in any order; outliers, infinities and NaNs reach the rows that hold their genes and
    no others; so do scales that are not finite."""
    rng = np.random.default_rng(8)
    rows, cols, n = 256 * 5 + 40, 1100, 64
    c = matrix(oracle, rng.integers(0, 101, size=rows), cols, 8, 1, 8)
    for r in range(200, rows, 41):
        lo, hi = c["row_ptr"][r], c["row_ptr"][r + 1]
        c["col_idx"][lo:hi] = rng.permutation(c["col_idx"][lo:hi])
    c["col_idx"][(c["col_idx"] == 300) & (np.arange(len(c["col_idx"])) > len(c["col_idx"]) // 2)] = 303
    w_host = dense(rng, cols, n, torch.float32, cuda_device)[1].copy()

    def compare():
        got = ops.spmm_forward(to_dev(c, cuda_device), torch.from_numpy(w_host).to(cuda_device)).cpu().numpy()
        with np.errstate(invalid="ignore", over="ignore"):
            dec = oracle.unpack_csr(8, 1, c["row_ptr"], c["packed_row_ptr"], c["col_idx"], c["scales"], c["offsets"], c["packed"]).astype(np.float64)
            r = np.repeat(np.arange(rows), np.diff(c["row_ptr"]))
            want, scale = np.zeros((rows, n)), np.zeros((rows, n))
            for j in range(n):
                np.add.at(want[:, j], r, dec * w_host[c["col_idx"], j])
                np.add.at(scale[:, j], r, (2 * np.abs(dec) + np.abs(c["offsets"][c["col_idx"]])) * np.abs(w_host[c["col_idx"], j]))
            finite = np.isfinite(want)
            assert np.array_equal(np.isnan(got), np.isnan(want)) and np.array_equal(got[np.isinf(want)], want[np.isinf(want)])
            # fp32 sums of up to 100 products, 2^-24 of the terms' magnitudes each; the oracle decodes with two roundings
            assert np.all(np.abs(got[finite] - want[finite]) <= 102 * 2.0 ** -24 * scale[finite] + 1e-30)

    compare()
    w_host[77, 5] = 1e6
    compare()
    w_host[123, 9], w_host[400, 9], w_host[401, 11] = np.inf, -np.inf, np.nan
    compare()
    w_host[:] = rng.normal(size=w_host.shape)
    c["scales"][500], c["offsets"][7] = np.nan, np.inf
    compare()
