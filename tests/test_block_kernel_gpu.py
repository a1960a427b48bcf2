"""GPU tests of the SpMM kernel that stages X block by block (spmm_tile.cu): how its warps share the stages,
what a call costs and leaves behind.  Results are compared with the oracle bit for bit."""
import os
import subprocess
import sys

import numpy as np
import pytest
import torch

import spx_ctypes as sx
from conftest import assert_bit_equal

pytestmark = pytest.mark.gpu


def sparse(rng, m, n, p):
    W = rng.standard_normal((m, n)).astype(np.float32)
    W[rng.random((m, n)) >= p] = 0
    return W


def in_child(name, **env):
    """Runs the test called `name` of this file in a process of its own: switches are read once per process."""
    cmd = [sys.executable, "-m", "pytest", "-q", "-x", "-m", "gpu", "-p", "no:cacheprovider", os.path.abspath(__file__), "-k", name]
    r = subprocess.run(cmd, env={**os.environ, **env}, capture_output=True, text=True, timeout=900)
    assert r.returncode == 0 and " passed" in r.stdout, r.stdout[-3000:] + r.stderr[-2000:]


@pytest.mark.parametrize("m,n,C,p", [
    # a stage is refilled many times (chunks of 256 columns, three staged), by CTAs of 1, a few and all 28 warps,
    # with rows long enough that the warps of a CTA drift apart
    (4, 20000, 64, 0.05), (1500, 12000, 64, 0.05), (5000, 6000, 128, 0.1), (16576, 3000, 64, 0.1)])
def test_stage_refills(lib, orc, cuda, m, n, C, p):
    """A chunk of X is overwritten by a later one once every warp of the CTA has read it.  Rows differ widely in
    length, X carries its row number, so an operand of the wrong chunk shows in any output it reaches."""
    if os.environ.get("SPX_SPMM_TILE") != "2":
        pytest.skip("runs in a child process of test_stage_refills_forced")
    rng = np.random.default_rng([m, n, C])
    W = sparse(rng, m, n, p)
    W[rng.random(m) < 0.3] *= (rng.random(n) < 0.2)       # a third of the rows a fifth as long
    W[m // 2] = 0
    E = orc.encode(W)
    X = (np.arange(n, dtype=np.float32)[:, None] + rng.uniform(-1, 1, (n, C))).astype(np.float32)
    rows = np.unique(np.concatenate([np.arange(0, m, max(1, m // 64)), [m // 2, m - 1], np.argsort(E.nnz)[-8:]]))
    from oracle import EllArrays
    want = orc.spmm(EllArrays(len(rows), n, E.r, E.Wd[rows], E.idx[rows], E.nnz[rows]), X, None)
    h = lib.ell_create(E.Wd, E.idx, E.nnz, E.n)
    dX = torch.from_numpy(X).to(cuda)
    first = None
    for call in range(12):
        dY = torch.full((m, C), float("nan"), device=cuda)
        h.spmm(dX.data_ptr(), C, C, 0, sx.ACT_NONE, dY.data_ptr(), C)
        torch.cuda.synchronize()
        if first is None:
            first = dY
            assert_bit_equal(dY[torch.from_numpy(rows).to(cuda)].cpu().numpy(), want, "sampled rows")
        assert torch.equal(dY.view(torch.int32), first.view(torch.int32)), f"call {call} differs from the first (gathered) one"


def test_stage_refills_forced():
    in_child("test_stage_refills and not forced", SPX_SPMM_TILE="2")
