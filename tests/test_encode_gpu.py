"""GPU: the device encoder around its limits -- units with as many entries as the counter keeps, one more, full and empty
ones in one matrix; row counts (and widths) on both sides of what the device ranks; ties -- against the oracle's arrays,
and a product through the row schedule."""
import os
import subprocess
import sys

import numpy as np
import pytest
import torch

import spx_ctypes as sx
from conftest import assert_bit_equal
from test_conv_tmem_gpu import fill_device, waits_for_the_device
from test_parity_gpu import dev, gpu_spmm

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n", [(1, 3), (5, 4096), (300, 2050), (1200, 512), (8192, 40), (8193, 40), (4099, 4100), (4800, 4100), (9473, 2050), (16385, 2050),
                                 (3, 300000), (7, 5000), (8, 5000), (2, 8191), (2, 8192), (900, 9000), (9, 262143), (28, 131000), (1300, 7000)])
@pytest.mark.parametrize("offset", [0, 1])
def test_units_around_what_is_kept(lib, orc, cuda, m, n, offset):
    rng = np.random.default_rng([m, n])
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    segs = min(max(1, n // 1024), max(1, -(-sms * 64 // m)))        # as the encoder cuts rows: where its limits lie
    seg = -(-(-(-n // segs)) // 4) * 4
    W = np.zeros((m, n), np.float32)
    for lo in range(0, n, seg):
        w = min(seg, n - lo)
        cap = seg // 64 * 17 + 16
        lens = rng.choice([0, 1, min(w, cap), min(w, cap + 1), w // 10, w], m, p=[.1, .1, .3, .2, .2, .1])
        order = np.argsort(rng.random((m, w), dtype=np.float32), axis=1)
        order[::3] = np.arange(w)[::-1]                             # at the end: kept up to the last place
        order[1::6] = np.arange(w)                                  # at the front: given up where they are many
        W[:, lo:lo + w][order < lens[:, None]] = 1
    W *= rng.standard_normal((m, n), dtype=np.float32)
    flat = torch.zeros(m * n + 1, device=cuda)
    flat[offset:offset + m * n] = dev(W, cuda).reshape(-1)
    E = orc.encode(W)
    for _ in range(2):                                              # the second time in memory that the first used
        h = lib.ell_encode_device(flat.data_ptr() + 4 * offset, m, n)
        Wd, idx, nnz = h.download()
        assert h.r == E.r and h.nnz_total == int(E.nnz.sum()) and np.array_equal(nnz, E.nnz) and np.array_equal(idx, E.idx)
        assert_bit_equal(Wd, E.Wd, "Wd")
    X = rng.uniform(-1, 1, (n, 12)).astype(np.float32)
    assert_bit_equal(gpu_spmm(h, X, None, sx.ACT_NONE, cuda), orc.spmm(E, X, None, act=0), "product")


@pytest.mark.parametrize("m,n", [(4800, 4100), (4799, 4101), (9000, 2048), (15104, 4096), (15105, 4096), (15105, 4608)])
def test_large_matrices(lib, cuda, m, n):
    """Rows in one and two segments, ranked and sorted by the host, with pairs and without, some too dense for them: the
    arrays against the same ones made with torch, and the schedule by a product of small whole numbers, which is exact."""
    g = torch.Generator(device=cuda).manual_seed(m + n)
    share = torch.tensor([0.0, 0.02, 0.1, 0.1, 0.24, 0.3], device=cuda)[torch.randint(0, 6, (m, 1), device=cuda, generator=g)]
    share = share.repeat(1, n)
    share[::7, n // 2:] = 0.4                               # rows whose second half is too dense
    W = torch.randint(1, 9, (m, n), device=cuda, generator=g).float()
    W[torch.rand((m, n), device=cuda, generator=g) >= share] = 0
    del share
    h = lib.ell_encode_device(W.data_ptr(), m, n)
    Wd, idx, nnz = (torch.from_numpy(a.view(np.int32)).to(cuda) for a in h.download())
    cnt = (W != 0).sum(1)
    assert torch.equal(nnz.long(), cnt) and h.r == int(cnt.max()) and h.nnz_total == int(cnt.sum())
    rows, cols = W.nonzero(as_tuple=True)
    place = torch.arange(len(rows), device=cuda) - (torch.cumsum(cnt, 0) - cnt)[rows]
    want = torch.zeros((m, h.r), dtype=torch.int32, device=cuda)
    want[rows, place] = cols.int()
    assert torch.equal(idx.view(m, h.r), want)
    want[rows, place] = W[rows, cols].view(torch.int32)
    assert torch.equal(Wd.view(m, h.r), want)
    X = torch.randint(-4, 5, (n, 4), device=cuda, generator=g).float()
    Y = torch.full((m, 4), float("nan"), device=cuda)
    h.spmm(X.data_ptr(), 4, 4, 0, sx.ACT_NONE, Y.data_ptr(), 4)
    assert torch.equal(Y.double(), W.double() @ X.double())


def test_without_room_for_the_pairs(lib, cuda):
    """Pairs that do not fit (39 MB) are gone without at once: the call waits for its own stream and for no other."""
    if os.environ.get("SPX_TEST_FULL_DEVICE") != "1":
        pytest.skip("runs in a child process, whose pool of freed memory is empty")
    m, n = 4800, 4100
    W = torch.zeros((m, n), device=cuda)
    W[:, ::20] = torch.arange(m, device=cuda)[:, None] + 1.0
    want = [a.copy() for a in lib.ell_encode_device(W[:2].contiguous().data_ptr(), 2, n).download()]
    assert not waits_for_the_device(lambda: None)           # (makes the stream while there is room)
    made = []
    held = fill_device(lib, 24 << 20, 8 << 20)
    try:
        for again in (False, True):
            waited = waits_for_the_device(lambda: made.append(lib.ell_encode_device(W.data_ptr(), m, n)))
            assert not (again and waited), "an encode waited for another stream's work"
            Wd, idx, nnz = made[-1].download()
            assert (nnz == want[2][0]).all() and (idx == want[1][0]).all() and (Wd[1] == want[0][1]).all() and Wd[-1, 0] == m
            made.pop().close()
    finally:
        for p in held:
            lib.spx_free(p)


def test_without_room_for_the_pairs_alone():
    cmd = [sys.executable, "-m", "pytest", "-q", "-x", "-m", "gpu", "-p", "no:cacheprovider", os.path.abspath(__file__) + "::test_without_room_for_the_pairs"]
    r = subprocess.run(cmd, env={**os.environ, "SPX_TEST_FULL_DEVICE": "1"}, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and " passed" in r.stdout, r.stdout[-3000:] + r.stderr[-2000:]
