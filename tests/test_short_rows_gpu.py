"""GPU: SpMM of matrices with many short rows: results at the edges of spmm_gather_half's range, bit for bit, and the
choice between gathering X and staging it block by block where rows have few entries per block."""
import numpy as np
import pytest
import torch

import spx_ctypes as sx
from conftest import assert_bit_equal

pytestmark = pytest.mark.gpu


def rows_of(rng, m, n, lengths):
    """CSR of m rows with the given lengths at random columns."""
    rowptr = np.concatenate([[0], np.cumsum(lengths)]).astype(np.uint64)
    col = np.concatenate([np.sort(rng.choice(n, k, replace=False)) for k in lengths] + [np.empty(0, int)]).astype(np.uint32)
    return rowptr, col, rng.standard_normal(len(col)).astype(np.float32)


@pytest.mark.parametrize("C", [40, 44, 48, 60, 64, 68, 100, 124, 128, 132])
@pytest.mark.parametrize("m", [2367, 2368, 4737])
def test_widths_and_row_counts(lib, orc, cuda, m, C):
    import workloads as wl
    from oracle import EllArrays
    rng = np.random.default_rng([m, C])
    n = 700
    lengths = rng.integers(0, 40, m)
    lengths[[0, m // 2, m - 1]] = [0, 127, 17]
    rowptr, col, val = rows_of(rng, m, n, lengths)
    h = lib.ell_create_csr(m, n, rowptr, col, val)
    Wd, idx, nnz = wl.csr_to_ell(m, rowptr, col, val)
    E = EllArrays(m, n, Wd.shape[1], Wd, idx, nnz)
    X = rng.uniform(-1, 1, (n, C)).astype(np.float32)
    b = rng.standard_normal(m).astype(np.float32)
    dX, dB = torch.from_numpy(X).to(cuda), torch.from_numpy(b).to(cuda)
    for bias, act in ((b, 1), (None, 0)):
        want = orc.spmm(E, X, bias, act=act)
        for call in range(3):
            dY = torch.full((m, C), float("nan"), device=cuda)
            h.spmm(dX.data_ptr(), C, C, 0 if bias is None else dB.data_ptr(), act, dY.data_ptr(), C)
            torch.cuda.synchronize()
            assert_bit_equal(dY.cpu().numpy(), want, f"call {call}")


@pytest.mark.parametrize("m,n,d,C", [(60000, 4000, 8, 33), (60000, 4000, 8, 250), (60000, 4000, 16, 130), (60000, 4000, 3, 127)])
def test_rows_with_few_entries_per_block_are_gathered(lib, cuda, m, n, d, C):
    """Staging X took 2 to 3.3 times as long as gathering it here: no later call on a handle may take longer than the
    first one, which gathers."""
    rng = np.random.default_rng(1)
    rowptr = np.arange(m + 1, dtype=np.uint64) * d
    col = (rng.integers(0, n // d, (m, d)) + np.arange(d) * (n // d)).astype(np.uint32).reshape(-1)
    h = lib.ell_create_csr(m, n, rowptr, col, np.ones(m * d, np.float32))
    X, Y = torch.rand((n, C), device=cuda), torch.zeros((m, C), device=cuda)
    before = lib.spx_launch_count()
    for k in range(3):
        h.spmm(X.data_ptr(), C, C, 0, 0, Y.data_ptr(), C)
    torch.cuda.synchronize()
    assert lib.spx_launch_count() - before == 3, "the block form was built"
