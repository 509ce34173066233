"""GPU parity of the fp32-FMA transpose that sorts entries by gene in shared memory, at the edges of its tiles, ranges and batches."""
import numpy as np
import pytest
import torch

from cellerator_b200 import capi, ops
from conftest import random_csr
from gpu_util import dense, host_pack, to_dev
from test_gpu_transpose import assert_transpose_close, col_l1_of

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,cols,max_nnz", [(512, 1500, 900), (513, 700, 700), (1030, 513, 513), (300, 1024, 1000)])
@pytest.mark.parametrize("n,bits,policy", [(64, 8, 1), (50, 8, 2), (32, 4, 1), (7, 4, 2), (130, 8, 1)])
def test_against_oracle(cuda_device, oracle, rows, cols, max_nnz, n, bits, policy):
    """One and several row tiles, ranges of genes that end inside a gene tile, batches of one and of several (dense rows),
    column tiles with a remainder, alpha / beta, a row range, rows that do not ascend."""
    rng = np.random.default_rng(rows + cols + n)
    c = random_csr(rng, rows=rows, cols=cols, max_nnz=max_nnz, bits=bits, policy=policy)
    for r in range(3, rows, 41):                                       # any order inside a row
        lo, hi = c["row_ptr"][r], c["row_ptr"][r + 1]
        c["col_idx"][lo:hi] = rng.permutation(c["col_idx"][lo:hi])
    c = host_pack(oracle, c)
    x = to_dev(c, cuda_device)
    assert x.nnz >= 50_000
    g, g_host = dense(rng, rows, n, torch.float32, cuda_device, std=1.0, ld=n + 3)
    op = ops.PreparedSpmm(capi.PROJECTION_TRANSPOSE, rows, cols, n, x.nnz, bits, policy, torch.float32, cuda_device)
    assert op.schedule == "vector_reductions" and op.workspace_bytes > 256
    cl1, gmax = col_l1_of(oracle, c), float(np.abs(g_host).max())
    args = (bits, policy, c["row_ptr"], c["packed_row_ptr"], c["col_idx"], c["packed"], c["scales"], c["offsets"], g_host, cols)
    out = op.run(x, g, torch.full((cols, n), float("nan"), device=cuda_device))
    assert op.status() == 0
    assert_transpose_close(out.cpu().numpy(), oracle.qcsr_transpose(*args), cl1, gmax)
    lo, hi = 5, rows - 9
    init = torch.from_numpy(rng.normal(size=(cols, n)).astype(np.float32)).to(cuda_device)
    part = op.run(x, g, init.clone(), alpha=2.0, beta=0.5, row_begin=lo, row_end=hi).cpu().numpy()
    want = 2.0 * oracle.qcsr_transpose(*args, lo, hi) + 0.5 * init.cpu().numpy()
    assert_transpose_close(part, want, 2.0 * cl1 + 1.0, gmax)
    # without a workspace the entries are added one by one
    op.workspace, op.workspace_bytes = None, 0
    assert_transpose_close(op.run(x, g, torch.empty(cols, n, device=cuda_device)).cpu().numpy(), oracle.qcsr_transpose(*args), cl1, gmax)


def test_workspace_does_not_grow_with_the_matrix(cuda_device):
    """1,000,000 x 33,538, 1.8e9 entries: the rows are taken in slices."""
    op = ops.PreparedSpmm(capi.PROJECTION_TRANSPOSE, 1_000_000, 33_538, 64, 1_800_000_000, 8, 1, torch.float32, cuda_device)
    assert op.schedule == "vector_reductions" and 256 < op.workspace_bytes <= 40 << 20
    op.close()


@pytest.mark.parametrize("rows", [4096 * 2, 4096 * 3 + 77])
def test_slices_against_oracle(cuda_device, oracle, rows):
    """A workspace for the starts of 4,096 rows at a time; alpha / beta count once; a row range cut into slices of its own."""
    rng = np.random.default_rng(rows)
    cols, n, bits, policy = 1025, 36, 8, 1
    c = host_pack(oracle, random_csr(rng, rows=rows, cols=cols, max_nnz=60, bits=bits, policy=policy))
    x = to_dev(c, cuda_device)
    g, g_host = dense(rng, rows, n, torch.float32, cuda_device, std=1.0)
    op = ops.PreparedSpmm(capi.PROJECTION_TRANSPOSE, rows, cols, n, x.nnz, bits, policy, torch.float32, cuda_device)
    sms = torch.cuda.get_device_properties(cuda_device).multi_processor_count
    op.workspace_bytes = 256 + 4 * ((3 + 1) * 4096 + 512 * sms)
    cl1, gmax = col_l1_of(oracle, c), float(np.abs(g_host).max())
    args = (bits, policy, c["row_ptr"], c["packed_row_ptr"], c["col_idx"], c["packed"], c["scales"], c["offsets"], g_host, cols)
    init = torch.from_numpy(rng.normal(size=(cols, n)).astype(np.float32)).to(cuda_device)
    launches = capi.lib().cb200_kernel_launch_count()
    out = op.run(x, g, init.clone(), alpha=2.0, beta=0.5).cpu().numpy()
    assert capi.lib().cb200_kernel_launch_count() - launches == 2 * -(-rows // 4096) and op.status() == 0
    assert_transpose_close(out, 2.0 * oracle.qcsr_transpose(*args) + 0.5 * init.cpu().numpy(), 2.0 * cl1 + 1.0, gmax)
    lo, hi = 5, rows - 9
    part = op.run(x, g, torch.full_like(init, float("nan")), row_begin=lo, row_end=hi).cpu().numpy()
    assert_transpose_close(part, oracle.qcsr_transpose(*args, lo, hi), cl1, gmax)
