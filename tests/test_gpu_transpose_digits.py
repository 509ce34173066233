"""GPU parity of the transpose with exact integer sums, at the edges of its tiles, pieces, chunks and runs."""
import numpy as np
import pytest
import torch

from cellerator_b200 import capi, ops
from conftest import random_csr
from gpu_util import dense, host_pack, to_dev

pytestmark = pytest.mark.gpu


def reference(oracle, c, g, lo=0, hi=None):
    """The sums over stored entries in 64 bits, and over their magnitudes; these with the zero-point's added, because the oracle decodes with
    two roundings, the product's and the sum's."""
    hi = c["rows"] if hi is None else hi
    dec = oracle.unpack_csr(c["bits"], c["policy"], c["row_ptr"], c["packed_row_ptr"], c["col_idx"], c["scales"], c["offsets"], c["packed"]).astype(np.float64)
    s, e = c["row_ptr"][lo], c["row_ptr"][hi]
    rows = np.repeat(np.arange(lo, hi), np.diff(c["row_ptr"][lo:hi + 1]))
    x = np.zeros((hi - lo, c["cols"]))
    x[rows - lo, c["col_idx"][s:e]] = dec[s:e]
    return x.T @ g[lo:hi].astype(np.float64), np.abs(x).sum(0) + np.bincount(c["col_idx"][s:e], minlength=c["cols"]) * np.abs(c["offsets"])


def assert_within(got, want, l1, g, slices):
    """G is rounded at 2 max|G| / 2^(8 S - 1) at most (max|G| of the column; 0.99 of the digits' range is used), the oracle's decoded value
    at 2^-24 of its terms; the sums are exact.  The end of a run, the sums of up to six runs, alpha and beta round at 2^-24 each."""
    most = np.abs(g).max(0, initial=0.0)
    bound = (1.02 * 2.0 ** (1 - 8 * slices) + 10 * 2.0 ** -24) * l1[:, None] * most[None, :] + 1e-30
    worst = np.max(np.abs(got.astype(np.float64) - want) / bound)
    assert worst <= 1.0, worst


def prepared(x, n, slices, device, **kw):
    """3 digits: fp32 products with the matrix in hand; 4: a request that has to be repeatable."""
    op = ops.PreparedSpmm(capi.PROJECTION_TRANSPOSE, x.rows, x.cols, n, x.nnz, x.bits, x.policy, torch.float32, device, device_matrix=x,
                          deterministic=slices == 4, schedule="tensor_blocked" if slices == 3 else None, **kw)
    assert op.schedule == ("tensor_blocked_x3" if slices == 3 else "gene_gather")
    return op


# fewer cells than a piece, a group and one cell, windows of one gene and of all but one, pieces without entries, tiles of several
# chunks (dense), and sizes from which on a repeatable request takes integer sums
@pytest.mark.parametrize("rows,cols,max_nnz,slices", [(31, 129, 60, 3), (257, 128, 90, 3), (256 * 3 + 33, 383, 20, 3), (700, 640, 640, 3),
                                                      (256 * 20 + 1, 1664, 120, 4), (256 * 17 - 1, 2047, 900, 4)])
@pytest.mark.parametrize("n,bits", [(64, 8), (32, 4), (32, 8)])
def test_prepared_against_64_bits(cuda_device, oracle, rows, cols, max_nnz, slices, n, bits):
    rng = np.random.default_rng(rows + n + bits)
    c = host_pack(oracle, random_csr(rng, rows=rows, cols=cols, max_nnz=max_nnz, bits=bits))
    x = to_dev(c, cuda_device)
    g, g_host = dense(rng, rows, n, torch.float32, cuda_device, std=1.0, ld=n + 3)
    op = prepared(x, n, slices, cuda_device)
    want, l1 = reference(oracle, c, g_host)
    first = op.run(x, g, torch.full((cols, n), float("nan"), device=cuda_device))
    assert op.status() == 0
    assert_within(first.cpu().numpy(), want, l1, g_host, slices)
    assert torch.equal(first, op.run(x, g, torch.full((cols, n), float("nan"), device=cuda_device)))
    lo, hi = rows // 7, rows - rows // 9                              # borders inside groups and pieces
    init = rng.normal(size=(cols, n)).astype(np.float32)
    want, l1 = reference(oracle, c, g_host, lo, hi)
    room = op.workspace_bytes
    for op.workspace_bytes in (room, room - 1 if rows < 4096 else room * 3 // 4):  # groups in slices
        part = op.run(x, g, torch.from_numpy(init).to(cuda_device), alpha=2.0, beta=0.5, row_begin=lo, row_end=hi).cpu().numpy()
        assert op.status() == 0
        assert_within(part, 2.0 * want + 0.5 * init, 2.0 * l1 + 1.0, np.maximum(np.abs(g_host[lo:hi]), 1.0), slices)
    op.close()


@pytest.mark.parametrize("n", [1, 33, 64, 100, 130])
@pytest.mark.parametrize("bits,ordered", [(8, True), (4, True), (8, False)])
def test_words_made_in_the_call(cuda_device, oracle, n, bits, ordered):
    """A matrix that is seen once, with enough entries; column blocks with a remainder; rows in any order, a row range."""
    rng = np.random.default_rng(n + bits)
    rows, cols = 2111, 1500
    c = random_csr(rng, rows=rows, cols=cols, max_nnz=3000, bits=bits)
    if not ordered:
        for r in range(3, rows, 41):
            lo, hi = c["row_ptr"][r], c["row_ptr"][r + 1]
            c["col_idx"][lo:hi] = rng.permutation(c["col_idx"][lo:hi])
    c = host_pack(oracle, c)
    x = to_dev(c, cuda_device)
    assert x.nnz >= 2_200_000
    g, g_host = dense(rng, rows, n, torch.float32, cuda_device, std=1.0, ld=n + 3)
    op = ops.PreparedSpmm(capi.PROJECTION_TRANSPOSE, rows, cols, n, x.nnz, bits, 1, torch.float32, cuda_device)
    assert op.schedule == "vector_reductions" and op.workspace_bytes > 4 * x.nnz
    for lo, hi in [(0, rows), (5, rows - 40)]:
        launches = capi.lib().cb200_kernel_launch_count()
        out = op.run(x, g, torch.full((cols, n), float("nan"), device=cuda_device), row_begin=lo, row_end=hi)
        assert capi.lib().cb200_kernel_launch_count() - launches == 5 and op.status() == 0
        want, l1 = reference(oracle, c, g_host, lo, hi)
        assert_within(out.cpu().numpy(), want, l1, g_host[lo:hi], 4)
    op.close()


def test_long_runs_stay_inside_32_bits(cuda_device):
    """140,000 cells: more than a run holds.  Every code is 0 (-128 as an operand) and G is the same everywhere: the largest sums there are."""
    rows, cols, n = 140_000, 40, 32
    row_ptr = np.arange(rows + 1, dtype=np.int64) * 20
    col_idx = (2 * np.tile(np.arange(20), rows) + np.repeat(np.arange(rows) & 1, 20)).astype(np.int32)
    c = dict(rows=rows, cols=cols, bits=8, policy=1, row_ptr=row_ptr, packed_row_ptr=row_ptr, col_idx=col_idx, packed=np.zeros(rows * 20, dtype=np.uint8),
             scales=np.full(cols, 0.25, dtype=np.float32), offsets=np.full(cols, 0.5, dtype=np.float32))
    x = to_dev(c, cuda_device)
    op = prepared(x, n, 3, cuda_device)
    for value in (0.99, -0.99):
        out = op.run(x, torch.full((rows, n), value, device=cuda_device), torch.empty(cols, n, device=cuda_device))
        assert op.status() == 0
        assert float((out / (np.float32(value).item() * 0.5 * rows / 2) - 1).abs().max()) <= 2.0 ** -22 + 8 * 2.0 ** -24
    op.close()


@pytest.mark.parametrize("slices", [3, 4])
def test_what_integer_sums_do_not_cover(cuda_device, oracle, slices):
    """Genes that a cell holds twice count twice; a column with an outlier keeps the others' bits; infinities and NaNs reach the genes of
    their cells and no others; so do scales that are not finite, of genes with and without entries."""
    rng = np.random.default_rng(slices)
    rows, cols, n = 256 * 20, 1664, 64
    c = host_pack(oracle, random_csr(rng, rows=rows, cols=cols, max_nnz=100, bits=8))
    c["col_idx"][c["col_idx"] == 300] = 303                           # gene 300 has no entries, rows may not ascend, cells may hold a gene twice
    assert any(np.any(np.diff(np.sort(c["col_idx"][a:b])) == 0) for a, b in zip(c["row_ptr"][:-1], c["row_ptr"][1:]))
    x = to_dev(c, cuda_device)
    g, g_host = dense(rng, rows, n, torch.float32, cuda_device, std=1.0)
    g_host = g_host.copy()
    op = prepared(x, n, slices, cuda_device)

    def entry_by_entry():
        dec = oracle.unpack_csr(8, 1, c["row_ptr"], c["packed_row_ptr"], c["col_idx"], c["scales"], c["offsets"], c["packed"]).astype(np.float64)
        r = np.repeat(np.arange(rows), np.diff(c["row_ptr"]))
        want, scale = np.zeros((cols, n)), np.zeros((cols, n))
        with np.errstate(invalid="ignore"):
            for j in range(n):
                np.add.at(want[:, j], c["col_idx"], dec * g_host[r, j])
                np.add.at(scale[:, j], c["col_idx"], (np.abs(dec) + np.abs(c["offsets"][c["col_idx"]])) * np.abs(g_host[r, j]))
        return want, scale

    def check():
        out = op.run(x, torch.from_numpy(g_host).to(cuda_device), torch.empty(cols, n, device=cuda_device))
        assert op.status() == 0 and torch.equal(out.view(torch.int32), op.run(x, torch.from_numpy(g_host).to(cuda_device), torch.empty(cols, n, device=cuda_device)).view(torch.int32))
        got, (want, scale) = out.cpu().numpy(), entry_by_entry()
        finite = np.isfinite(want)
        assert np.array_equal(np.isnan(got), np.isnan(want)) and np.array_equal(got[np.isinf(want)], want[np.isinf(want)])
        # an entry's value v = s c + o: rounded once here, at 2^-24 |v|, twice by the oracle, at 2^-24 |s c| <= 2^-24 (|v| + |o|) and 2^-24 |v|;
        # the sum once at the end, at 2^-24 of itself: four times 2^-24 (|v| + |o|) |g| in all
        assert np.all(np.abs(got[finite] - want[finite]) <= 2.0 ** -22 * scale[finite] + 1e-30)

    check()
    g_host[77, 5] = 1e6                                               # a second pass of digits
    check()
    g_host[123, 9], g_host[4000, 9], g_host[4001, 11] = np.inf, -np.inf, np.nan
    check()
    g_host[:] = rng.normal(size=g_host.shape)
    c["scales"][300], c["offsets"][7] = np.nan, np.inf
    x.scales.copy_(torch.from_numpy(c["scales"])), x.offsets.copy_(torch.from_numpy(c["offsets"]))
    out = op.run(x, torch.from_numpy(g_host).to(cuda_device), torch.empty(cols, n, device=cuda_device)).cpu().numpy()
    assert np.all(out[300] == 0.0) and not np.any(np.isfinite(out[7])) and np.all(np.isfinite(np.delete(out, 7, axis=0)))
    op.close()


def test_bounded_wait_path(cuda_device, oracle):
    """The loader of G withholds its copies and every wait gives up: the status says so, and the next launch is correct."""
    rng = np.random.default_rng(4)
    rows, cols, n = 256 * 6, 1000, 64
    c = host_pack(oracle, random_csr(rng, rows=rows, cols=cols, max_nnz=100, bits=8, empty_rows=False))
    x = to_dev(c, cuda_device)
    g, _ = dense(rng, rows, n, torch.float32, cuda_device, std=1.0)
    op = prepared(x, n, 3, cuda_device)
    good = op.run(x, g, torch.empty(cols, n, device=cuda_device)).clone()
    assert op.status() == 0
    capi.lib().cb200_test_arm_wait_timeout(4096)
    try:
        op.run(x, g, torch.empty(cols, n, device=cuda_device))
    finally:
        capi.lib().cb200_test_disarm_wait_timeout()
    with pytest.raises(capi.Cb200Error) as e:
        op.status()
    assert e.value.status == capi.DEVICE_WAIT_TIMEOUT
    assert torch.equal(op.run(x, g, torch.full((cols, n), float("nan"), device=cuda_device)), good) and op.status() == 0
    op.close()


@pytest.mark.parametrize("slices,room", [(3, 1.0), (3, 0.8), (4, 1.0), (4, 0.3), (0, 1.0)])
def test_sums_are_whole_when_a_wait_ran_out(cuda_device, oracle, slices, room):
    """The status word is set, and the launch's last kernel has added the entries up by itself: a call that keeps no handle to ask has its result.
    Slices of the groups; a row range; 0 digits: the words made in the call, and the one-call function."""
    rng = np.random.default_rng(slices)
    rows, cols, n = (2111, 1500, 50) if slices == 0 else (256 * 20 + 9, 1664, 64)
    c = host_pack(oracle, random_csr(rng, rows=rows, cols=cols, max_nnz=3000 if slices == 0 else 120, bits=8))
    x = to_dev(c, cuda_device)
    g, g_host = dense(rng, rows, n, torch.float32, cuda_device, std=1.0)
    op = prepared(x, n, slices, cuda_device) if slices else ops.PreparedSpmm(capi.PROJECTION_TRANSPOSE, rows, cols, n, x.nnz, 8, 1, torch.float32, cuda_device)
    op.workspace_bytes = int(op.workspace_bytes * room)
    init = rng.normal(size=(cols, n)).astype(np.float32)
    for lo, hi in ((0, rows), (5, rows - 40)):
        want, l1 = reference(oracle, c, g_host, lo, hi)
        outs = []
        for polls in (4096, 4096, 0):
            out = torch.from_numpy(init).to(cuda_device)
            if polls:
                capi.lib().cb200_test_arm_wait_timeout(polls)
            try:
                op.run(x, g, out, alpha=2.0, beta=0.5, row_begin=lo, row_end=hi)
            finally:
                capi.lib().cb200_test_disarm_wait_timeout()
            if polls:
                with pytest.raises(capi.Cb200Error) as e:
                    op.status()
                assert e.value.status == capi.DEVICE_WAIT_TIMEOUT
            else:
                assert op.status() == 0
            outs.append(out.cpu().numpy())
            # in 64 bits where the wait ran out: inside the bound of the digits
            assert_within(outs[-1], 2.0 * want + 0.5 * init, 2.0 * l1 + 1.0, np.maximum(np.abs(g_host[lo:hi]), 1.0), 3 if polls == 0 and slices == 3 else 4)
        assert np.array_equal(outs[0], outs[1])
    op.close()
    if slices == 0:
        want, l1 = reference(oracle, c, g_host)
        capi.lib().cb200_test_arm_wait_timeout(4096)
        try:
            out = ops.spmm_transpose(x, g)
        finally:
            capi.lib().cb200_test_disarm_wait_timeout()
        assert_within(out.cpu().numpy(), want, l1, g_host, 4)


@pytest.mark.parametrize("n,bits,outlier", [(64, 8, 1.0), (32, 4, 1.0), (128, 8, 1e6)])
def test_repeatable_bits_do_not_follow_from_the_workspace(cuda_device, oracle, n, bits, outlier):
    """Row groups in slices, windows in chunks, one pass of digits and two: whatever the room is, down to the least that is accepted."""
    rng = np.random.default_rng(n)
    rows, cols = 256 * 22 + 7, 128 * 37 - 5
    x = to_dev(host_pack(oracle, random_csr(rng, rows=rows, cols=cols, max_nnz=400, bits=bits)), cuda_device)
    g, _ = dense(rng, rows, n, torch.float32, cuda_device, std=1.0)
    g[77, 5] *= outlier
    op = prepared(x, n, 4, cuda_device)
    room = op.workspace_bytes
    for lo, hi in ((0, rows), (100, rows - 300)):
        op.workspace_bytes = room
        want, refused, accepted = op.run(x, g, torch.empty(cols, n, device=cuda_device), row_begin=lo, row_end=hi).clone(), 0, []
        for part in (0.99, 0.75, 0.5, 0.35, 0.25, 0.18, 0.12, 0.08, 0.05, 0.02):
            op.workspace_bytes = int(room * part)
            try:
                got = op.run(x, g, torch.full((cols, n), float("nan"), device=cuda_device), row_begin=lo, row_end=hi)
            except capi.Cb200Error as e:
                assert e.status == capi.INSUFFICIENT_WORKSPACE
                refused += 1
                continue
            assert refused == 0 and op.status() == 0 and torch.equal(got, want), part
            accepted.append(part)
        assert refused > 0 and min(accepted) < 0.75
    op.close()


def mode_of(op):
    """Digits, passes and whether the last launch went entry by entry: the word behind the workspace's status word."""
    mode = op.workspace[4:8].view(torch.int32).item()
    return mode >> 4 & 15, mode & 15, bool(mode & 256)


# cells scaled down (share, binary orders, all columns or every fifth alone), and how many digits and passes that takes from three and from four
@pytest.mark.parametrize("share,orders,column,from3,from4", [
    (0.0, 0, None, (3, 1, False), (4, 1, False)), (0.3, 7, None, (4, 1, False), (4, 2, False)), (0.1, 20, None, (3, 2, False), (4, 2, False)),
    (0.02, 36, None, (4, 2, False), (4, 2, False)), (0.05, 30, None, (4, 2, False), (4, 2, False)), (0.1, 70, None, (4, 2, True), (4, 2, True)),
    (0.3, 22, 5, (3, 2, False), (4, 2, False))])
@pytest.mark.parametrize("slices,n,bits", [(3, 64, 8), (3, 32, 4), (4, 64, 8), (4, 32, 8), (4, 128, 4)])
def test_few_small_cells_keep_their_bits(cuda_device, oracle, share, orders, column, from3, from4, slices, n, bits):
    """A gene that only cells with a small G hold has the precision of its own products, whatever the rest of G's columns hold.  No cell holds a
    gene twice: nothing here goes entry by entry but numbers beyond two passes.  Row ranges; slices of the groups."""
    rng = np.random.default_rng(int(100 * share) + orders)
    rows, cols = 256 * 20 + 3, 1664
    c = random_csr(rng, rows=rows, cols=cols - 1, max_nnz=120, bits=bits)
    small = rng.permutation(rows)[:int(share * rows)]
    is_small = np.zeros(rows, dtype=bool)
    is_small[small] = True
    c["col_idx"][c["col_idx"] >= 7] += 1                              # gene 7: held by the small cells alone
    at = np.repeat(np.arange(rows), np.diff(c["row_ptr"]))
    keys = np.concatenate([at.astype(np.int64) * cols + c["col_idx"], small.astype(np.int64) * cols + 7])
    order = np.argsort(keys)
    values = np.concatenate([c["values"], rng.uniform(-2.0, 40.0, size=len(small)).astype(np.float32)])[order]
    c.update(cols=cols, col_idx=(keys[order] % cols).astype(np.int32), values=values, row_ptr=np.searchsorted(keys[order], np.arange(rows + 1) * cols).astype(np.int64),
             scales=np.append(c["scales"], np.float32(0.3)), offsets=np.append(c["offsets"], np.float32(-0.7)))
    c = host_pack(oracle, c)
    x = to_dev(c, cuda_device)
    g_host = rng.normal(size=(rows, n)).astype(np.float32)
    if column is None:
        g_host[is_small] *= np.float32(2.0 ** -orders)
    else:
        g_host[np.ix_(is_small, np.arange(0, n, column))] *= np.float32(2.0 ** -orders)
    g = torch.from_numpy(g_host).to(cuda_device)
    # what a number's rounding is measured against: the cell's largest of sixteen neighbouring columns, or the number itself
    reach = np.abs(g_host).astype(np.float64) if column is not None else np.repeat(np.abs(g_host).reshape(rows, n // 16, 16).max(2), 16, axis=1).astype(np.float64)
    op = prepared(x, n, slices, cuda_device)
    dec = oracle.unpack_csr(bits, 1, c["row_ptr"], c["packed_row_ptr"], c["col_idx"], c["scales"], c["offsets"], c["packed"]).astype(np.float64)
    at, room = np.repeat(np.arange(rows), np.diff(c["row_ptr"])), op.workspace_bytes
    for lo, hi, part in ((0, rows, 1.0), (0, rows, 0.8), (300, rows - 100, 1.0)):
        op.workspace_bytes = int(room * part)
        out = op.run(x, g, torch.full((cols, n), float("nan"), device=cuda_device), row_begin=lo, row_end=hi)
        assert op.status() == 0
        if part == 1.0 and lo == 0:
            assert mode_of(op) == (from3 if slices == 3 else from4)
        sel = (at >= lo) & (at < hi)
        value, size = np.zeros((rows, cols)), np.zeros((rows, cols))
        value[at[sel], c["col_idx"][sel]] = dec[sel]
        size[at[sel], c["col_idx"][sel]] = np.abs(dec[sel]) + np.abs(c["offsets"][c["col_idx"][sel]])
        want, scale = value.T @ g_host.astype(np.float64), size.T @ reach
        # half a step: 1.02 * 2^(1 - 8 S) of a column's largest, which the launch's spread makes 2^-23 (from 4 digits) or 2^-18 (from 3) of `reach`; for a
        # column by itself the mean over its numbers is bounded, and with a third of them small theirs by ten times that (1 / 0.3^2); the oracle's
        # decoding and the roundings of up to eight runs at 2^-24 each
        half = 1.02 * (2.0 ** -23 if slices == 4 else 2.0 ** -18) * (1.0 if column is None else 12.0)
        assert np.all(np.abs(out.cpu().numpy() - want) <= (half + 10 * 2.0 ** -24) * scale + 1e-37), np.max(np.abs(out.cpu().numpy() - want) / (scale + 1e-37))
    op.close()


def test_more_genes_than_one_round_of_windows(cuda_device, oracle):
    """The places of more than 98,304 genes' windows are added up in two rounds; prepared and with words made in the call."""
    rng = np.random.default_rng(11)
    rows, cols, n = 300, 120_000, 32
    lengths = np.full(rows, 7200)
    row_ptr = np.concatenate([[0], np.cumsum(lengths)]).astype(np.int64)
    col_idx = np.concatenate([np.sort(rng.permutation(cols)[:k]) for k in lengths]).astype(np.int32)
    c = host_pack(oracle, dict(rows=rows, cols=cols, bits=8, policy=1, row_ptr=row_ptr, col_idx=col_idx, scales=rng.uniform(0.01, 0.5, size=cols).astype(np.float32),
                               offsets=rng.uniform(-1.0, 1.0, size=cols).astype(np.float32), values=rng.uniform(-2.0, 40.0, size=len(col_idx)).astype(np.float32)))
    x = to_dev(c, cuda_device)
    g, g_host = dense(rng, rows, n, torch.float32, cuda_device, std=1.0)
    want, l1 = reference(oracle, c, g_host)
    op = prepared(x, n, 4, cuda_device)
    assert mode_of_run(op, x, g, cols) == (4, 1, False)
    assert_within(op.run(x, g, torch.empty(cols, n, device=cuda_device)).cpu().numpy(), want, l1, g_host, 4)
    op.close()
    op = ops.PreparedSpmm(capi.PROJECTION_TRANSPOSE, rows, cols, n, x.nnz, 8, 1, torch.float32, cuda_device)
    assert x.nnz >= 2_000_000 and mode_of_run(op, x, g, cols) == (4, 1, False)
    assert_within(op.run(x, g, torch.empty(cols, n, device=cuda_device)).cpu().numpy(), want, l1, g_host, 4)
    op.close()


def mode_of_run(op, x, g, cols):
    op.run(x, g, torch.empty(cols, g.shape[1], device=g.device))
    assert op.status() == 0
    return mode_of(op)


@pytest.mark.parametrize("slices,n,bits,outlier", [(3, 64, 8, 1.0), (3, 32, 4, 1e6), (4, 64, 8, 1e6), (4, 32, 8, 1.0), (4, 128, 4, 1.0), (0, 50, 8, 1.0), (0, 130, 4, 1e6)])
def test_a_gene_held_again_changes_no_others(cuda_device, oracle, slices, n, bits, outlier):
    """A cell that holds genes twice and three times, one that holds a gene a hundred times: these genes count as often, and all others keep the bits that they have without
    them.  0 digits: the words made in the call."""
    rng = np.random.default_rng(n)
    rows, cols = (2111, 1500) if slices == 0 else (256 * 20, 1664)
    c = random_csr(rng, rows=rows, cols=cols, max_nnz=3000 if slices == 0 else 200, bits=bits)
    again = {77: [100, 101, 101, 600], rows - 1: [5], 256 * 3 + 31: [1400] * 100}
    keys = np.repeat(np.arange(rows), np.diff(c["row_ptr"])).astype(np.int64) * cols + c["col_idx"]
    keep = np.isin(keys, [r * cols + g for r, genes in again.items() for g in genes], invert=True)
    keys, values = keys[keep], c["values"][keep]
    once = np.array([r * cols + g for r, genes in again.items() for g in sorted(set(genes))])
    more = np.array([r * cols + g for r, genes in again.items() for g in genes])

    def matrix(extra):
        all_keys = np.concatenate([keys, extra])
        order = np.argsort(all_keys, kind="stable")
        k = all_keys[order]
        v = np.concatenate([values, np.linspace(1.0, 30.0, len(extra), dtype=np.float32)])[order]
        return host_pack(oracle, dict(c, row_ptr=np.searchsorted(k, np.arange(rows + 1) * cols).astype(np.int64), col_idx=(k % cols).astype(np.int32), values=v))

    g_host = rng.normal(size=(rows, n)).astype(np.float32)
    g_host[9, n - 1] = outlier
    g = torch.from_numpy(g_host).to(cuda_device)
    outs = []
    for m in (matrix(once), matrix(np.concatenate([once, more])), matrix(np.concatenate([once, more]))):
        x = to_dev(m, cuda_device)
        op = prepared(x, n, slices, cuda_device) if slices else ops.PreparedSpmm(capi.PROJECTION_TRANSPOSE, rows, cols, n, x.nnz, bits, 1, torch.float32, cuda_device)
        out = op.run(x, g, torch.full((cols, n), float("nan"), device=cuda_device))
        assert op.status() == 0 and not mode_of(op)[2] and (outlier == 1.0) == (mode_of(op)[1] == 1)
        outs.append(out.cpu().numpy())
        op.close()
    held = sorted({g for genes in again.values() for g in genes})
    others = np.delete(np.arange(cols), held)
    assert np.array_equal(outs[0][others], outs[1][others]) and np.array_equal(outs[1], outs[2])
    dec = oracle.unpack_csr(bits, 1, m["row_ptr"], m["packed_row_ptr"], m["col_idx"], m["scales"], m["offsets"], m["packed"]).astype(np.float64)
    at = np.repeat(np.arange(rows), np.diff(m["row_ptr"]))
    for gene in held:
        sel = m["col_idx"] == gene
        want, size = dec[sel] @ g_host[at[sel]].astype(np.float64), (np.abs(dec[sel]) + abs(m["offsets"][gene])).sum() * np.abs(g_host).max(0)
        # as in assert_within, two passes as four digits at least
        assert np.all(np.abs(outs[1][gene] - want) <= (1.02 * 2.0 ** (1 - 8 * (3 if slices == 3 else 4)) + 10 * 2.0 ** -24) * size), gene


@pytest.mark.parametrize("slices,n,bits", [(3, 64, 8), (3, 32, 4), (4, 64, 8), (4, 32, 8), (4, 128, 4), (0, 50, 8), (0, 130, 4)])
def test_infinities_and_nans_reach_their_genes_alone(cuda_device, oracle, slices, n, bits):
    """Every sum that no infinity or NaN is part of has the bits it has with zeroes in their place; the others are what 64 bits make of them.  Few cells,
    all cells, cells outside the row range; genes held again; slices of the groups; alpha and beta.  0 digits: the words made in the call."""
    rng = np.random.default_rng(n)
    rows, cols = (2111, 1500) if slices == 0 else (256 * 20 + 9, 1664)
    c = host_pack(oracle, random_csr(rng, rows=rows, cols=cols, max_nnz=3000 if slices == 0 else 120, bits=bits))
    if bits == 4:
        c["col_idx"][c["col_idx"] == 300] = 303                       # gene 300 is in no cell, some cells hold 303 twice
    x = to_dev(c, cuda_device)
    dec = oracle.unpack_csr(bits, 1, c["row_ptr"], c["packed_row_ptr"], c["col_idx"], c["scales"], c["offsets"], c["packed"]).astype(np.float64)
    at = np.repeat(np.arange(rows), np.diff(c["row_ptr"]))
    op = prepared(x, n, slices, cuda_device) if slices else ops.PreparedSpmm(capi.PROJECTION_TRANSPOSE, rows, cols, n, x.nnz, bits, 1, torch.float32, cuda_device)
    room = op.workspace_bytes
    base = rng.normal(size=(rows, n)).astype(np.float32)
    few = base.copy()
    few[[5, 400, 401, rows - 1], [0, 31, n - 1, n - 1]] = [np.inf, -np.inf, np.nan, np.inf]
    few[700:703, :] = np.inf
    many = np.where(rng.random(base.shape) < 0.5, np.inf, base).astype(np.float32)
    many[::3, 7] = -np.inf
    for g_host in (few, many, np.full_like(base, np.nan)):
        for lo, hi, part in ((0, rows, 1.0), (6, rows - 1, 1.0)) + (((0, rows, 0.8),) if slices else ()):
            op.workspace_bytes = int(room * part)
            init = torch.from_numpy(rng.normal(size=(cols, n)).astype(np.float32)).to(cuda_device)
            def run(g):
                out = op.run(x, torch.from_numpy(g).to(cuda_device), init.clone(), alpha=2.0, beta=0.5, row_begin=lo, row_end=hi)
                assert op.status() == 0 and not mode_of(op)[2]
                return out.cpu().numpy()
            got, zeroed = run(g_host), run(np.where(np.isfinite(g_host), g_host, 0.0).astype(np.float32))
            sel = (at >= lo) & (at < hi)
            want = np.zeros((cols, n))
            with np.errstate(invalid="ignore"):
                for j in range(n):                                    # what the sums are made of, not their rounding
                    odd = sel & ~np.isfinite(g_host[at, j])
                    np.add.at(want[:, j], c["col_idx"][odd], 2.0 * dec[odd] * g_host[at[odd], j])
            touched = ~np.isfinite(want)
            assert touched.any() and np.array_equal(got[~touched], zeroed[~touched])
            assert np.array_equal(got[touched], want[touched].astype(np.float32), equal_nan=True)
            assert np.array_equal(run(g_host).view(np.int32), got.view(np.int32))
    op.close()


@pytest.mark.parametrize("gene", [-1, 1664, 2 ** 31 - 1])
def test_a_gene_outside_the_matrix_is_refused(cuda_device, oracle, gene):
    """Preparing a repeatable transpose refuses it whatever kernel is chosen; the other requests leave its entry out."""
    rng = np.random.default_rng(5)
    rows, cols, n = 256 * 20, 1664, 64
    c = host_pack(oracle, random_csr(rng, rows=rows, cols=cols, max_nnz=100, bits=8, empty_rows=False))
    x = to_dev(c, cuda_device)
    at = int(c["row_ptr"][1234])
    x.col_idx[at] = gene
    for hint in (None, "gene_gather"):
        with pytest.raises(capi.Cb200Error) as e:
            ops.PreparedSpmm(capi.PROJECTION_TRANSPOSE, rows, cols, n, x.nnz, 8, 1, torch.float32, cuda_device, device_matrix=x, deterministic=True, schedule=hint)
        assert e.value.status == capi.INVALID_SHAPE
    g, g_host = dense(rng, rows, n, torch.float32, cuda_device, std=1.0)
    op = prepared(x, n, 3, cuda_device)
    got = op.run(x, g, torch.empty(cols, n, device=cuda_device)).cpu().numpy()
    assert op.status() == 0
    op.close()
    want, l1 = reference(oracle, c, g_host)                           # with the entry's own gene in place
    held = c["col_idx"][at]
    dec = oracle.unpack_csr(8, 1, c["row_ptr"], c["packed_row_ptr"], c["col_idx"], c["scales"], c["offsets"], c["packed"])
    want[held] -= float(dec[at]) * g_host[1234].astype(np.float64)
    assert_within(got, want, l1, g_host, 3)


@pytest.mark.parametrize("n,multiply", [(1, capi.DTYPE_F32), (50, capi.DTYPE_F32), (100, capi.DTYPE_BF16), (128, capi.DTYPE_F32)])
def test_handing_the_matrix_over_takes_nothing_away(cuda_device, oracle, n, multiply):
    """Widths that no prepared schedule serves: the same kernels, workspace and bits as without the matrix in hand."""
    rng = np.random.default_rng(n)
    rows, cols = 4500, 1400
    x = to_dev(host_pack(oracle, random_csr(rng, rows=rows, cols=cols, max_nnz=1300, bits=8)), cuda_device)
    assert x.nnz >= 2_000_000
    g, _ = dense(rng, rows, n, torch.float32, cuda_device, std=1.0)
    outs = []
    for matrix in (None, x):
        op = ops.PreparedSpmm(capi.PROJECTION_TRANSPOSE, rows, cols, n, x.nnz, 8, 1, torch.float32, cuda_device, device_matrix=matrix, multiply=multiply)
        launches = capi.lib().cb200_kernel_launch_count()
        out = op.run(x, g, torch.empty(cols, n, device=cuda_device))
        assert op.status() == 0
        outs.append((op.schedule, op.workspace_bytes, capi.lib().cb200_kernel_launch_count() - launches, out.cpu().numpy().tobytes()))
        op.close()
    assert outs[0] == outs[1] and outs[0][0] == "vector_reductions"


def test_names_and_digits(cuda_device, oracle):
    """The integer kernel of a repeatable request by its name, at a size that would not choose it, and which kernel a name that two share stands for."""
    rng = np.random.default_rng(6)
    rows, cols, n = 700, 640, 64
    c = host_pack(oracle, random_csr(rng, rows=rows, cols=cols, max_nnz=200, bits=8))
    x = to_dev(c, cuda_device)
    g, g_host = dense(rng, rows, n, torch.float32, cuda_device, std=1.0)
    want, l1 = reference(oracle, c, g_host)

    def make(hint, deterministic=True, matrix=x, nnz=x.nnz, rows=rows, cols=cols):
        return ops.PreparedSpmm(capi.PROJECTION_TRANSPOSE, rows, cols, n, nnz, 8, 1, torch.float32, cuda_device, device_matrix=matrix, deterministic=deterministic, schedule=hint)
    for hint, name, digits in ((None, "gene_gather", 0), ("gene_gather", "gene_gather", 0), ("integer_windows", "integer_windows", 4)):
        op = make(hint)
        assert (op.schedule, op.digits) == (name, digits)
        got = op.run(x, g, torch.empty(cols, n, device=cuda_device)).cpu().numpy()
        assert op.status() == 0
        if digits:
            assert_within(got, want, l1, g_host, 4)
        op.close()
    for op, name, digits in ((make("tensor_blocked", False), "tensor_blocked_x3", 3), (make(None, False, None, 5_000_000, 8_000, 4_000), "vector_reductions", 4),
                             (make(None, False, None, 100_000, 8_000, 4_000), "vector_reductions", 0)):
        assert (op.schedule, op.digits) == (name, digits)
        op.close()
