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


@pytest.mark.parametrize("m,n", [(1, 3), (5, 4096), (300, 2050), (1200, 512), (8192, 40), (8193, 40), (4099, 4100), (9473, 2050), (16385, 2050),
                                 (3, 300000), (7, 5000), (8, 5000), (9, 262143), (28, 131000), (1300, 7000)])
@pytest.mark.parametrize("offset", [0, 1])
def test_units_around_what_is_kept(lib, orc, cuda, m, n, offset):
    rng = np.random.default_rng([m, n])
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    segs = min(max(1, n // 1024), max(1, -(-sms * 64 // m)))        # as the encoder cuts rows: where its limits lie
    seg = -(-(-(-n // segs)) // 4) * 4
    W = np.zeros((m, n), np.float32)
    for lo in range(0, n, seg):
        w = min(seg, n - lo)
        cap = seg // 4
        lens = rng.choice([0, 1, min(w, cap), min(w, cap + 1), w // 10, w], m, p=[.1, .1, .3, .2, .2, .1])
        order = np.argsort(rng.random((m, w), dtype=np.float32), axis=1)
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


def test_without_room_for_the_pairs(lib, cuda):
    """Pairs that do not fit (39 MB) are gone without at once: the call waits for its own stream and for no other."""
    if os.environ.get("SPX_TEST_FULL_DEVICE") != "1":
        pytest.skip("runs in a child process, whose pool of freed memory is empty")
    m, n = 9473, 2050
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
