"""GPU tests of the host-buffer calls and copies: what they do under stream capture, from several threads, in order
with other work, and on every route that an operand's size and kind of memory selects."""
import ctypes as C
import threading

import numpy as np
import pytest
import torch

import spx_ctypes as sx
from conftest import assert_bit_equal

pytestmark = pytest.mark.gpu


def vp(a):
    return a.ctypes.data_as(C.c_void_p)


def sparse(rng, m, n, p):
    W = rng.standard_normal((m, n)).astype(np.float32)
    W[rng.random((m, n)) >= p] = 0
    return W


class Stream:
    """A stream of the library's own (non-blocking)."""

    def __init__(self, lib):
        self.lib, self.h = lib, C.c_void_p()
        lib.spx_stream_create(C.byref(self.h))

    def __enter__(self):
        return self.h

    def __exit__(self, *exc):
        self.lib.spx_stream_sync(self.h)
        self.lib.spx_stream_destroy(self.h)


def test_copies_under_capture(lib, cuda):
    """A captured copy of pageable memory reads that memory when the graph runs, whatever was copied since, and
    copies outside the capture go on as before -- the same thread's on another stream too, while it captures."""
    rng = np.random.default_rng(1)
    src, other = rng.random(1 << 18, dtype=np.float32), rng.random(3 << 20, dtype=np.float32)
    dst = torch.zeros(1 << 18, device=cuda)
    elsewhere = torch.zeros(3 << 20, device=cuda)
    torch.cuda.synchronize()
    with Stream(lib) as st, Stream(lib) as free:
        for warm in range(2):                   # the second time the staging ring has been used before
            lib.spx_graph_capture_begin(st)
            lib.spx_memcpy_h2d(dst.data_ptr(), vp(src), src.nbytes, st)
            lib.spx_memcpy_h2d(elsewhere.data_ptr(), vp(other), other.nbytes, free)
            graph = C.c_void_p()
            lib.spx_graph_capture_end(st, C.byref(graph))
            for k in range(3):
                lib.spx_memcpy_h2d(elsewhere.data_ptr(), vp(other), other.nbytes, free)
            lib.spx_stream_sync(free)
            assert_bit_equal(elsewhere.cpu().numpy(), other, "ordinary copies")
            src[:] = rng.random(1 << 18, dtype=np.float32)
            lib.spx_graph_launch(graph, st)
            lib.spx_stream_sync(st)
            assert_bit_equal(dst.cpu().numpy(), src, "captured copy")
            lib.spx_graph_destroy(graph)
