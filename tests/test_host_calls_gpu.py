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


def together(*jobs):
    """Runs the jobs in threads of their own and raises what any of them raised."""
    errors = []

    def guard(job):
        try:
            torch.cuda.set_device(0)
            job()
        except BaseException as e:      # noqa: BLE001 - reported below
            errors.append(e)
    threads = [threading.Thread(target=guard, args=(j,)) for j in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    if errors:
        raise errors[0]


def test_launches_of_one_kernel_from_several_threads(lib, orc, cuda):
    """The same kernels with different amounts of shared memory at the same time: no launch is refused, and results
    are those of one thread."""
    rng = np.random.default_rng(3)
    jobs = []
    for i, (m, n, Cc) in enumerate([(300, 100, 64), (300, 500, 64), (400, 300, 32), (256, 1000, 32)]):
        E = orc.encode(sparse(rng, m, n, 0.9))
        X = rng.uniform(-1, 1, (n, Cc)).astype(np.float32)
        x = rng.uniform(-1, 1, (n, 1)).astype(np.float32)
        h = lib.ell_create(E.Wd, E.idx, E.nnz, E.n)
        dX, dx = torch.from_numpy(X).to(cuda), torch.from_numpy(x).to(cuda)
        dY, dy, dz = torch.zeros((m, Cc), device=cuda), torch.zeros((m, 1), device=cuda), torch.zeros(m, device=cuda)
        want, want1 = orc.spmm(E, X, None), orc.spmm(E, x, None)

        def job(h=h, dX=dX, dx=dx, dY=dY, dy=dy, dz=dz, Cc=Cc, want=want, want1=want1):
            with Stream(lib) as st:
                for k in range(1500):
                    h.spmm(dX.data_ptr(), Cc, Cc, 0, 0, dY.data_ptr(), Cc, st)
                    h.spmm(dx.data_ptr(), 1, 1, 0, 0, dy.data_ptr(), 1, st)
                    h.spmv(dx.data_ptr(), 0, dz.data_ptr(), st)
                lib.spx_stream_sync(st)
            assert_bit_equal(dY.cpu().numpy(), want, "wide")
            assert_bit_equal(dy.cpu().numpy(), want1, "one column")
        jobs.append(job)
    torch.cuda.synchronize()
    together(*jobs)


def test_encoding_beside_products_on_one_stream(lib, orc, cuda):
    """Handles are made and destroyed on a stream on which another thread queues products that use scratch of the
    library's pool (X re-pitched for bulk copies): neither disturbs the other."""
    rng = np.random.default_rng(4)
    m, n, Cc = 1201, 1100, 77                   # the block kernel, with a copy of X in rows of 16-byte multiples
    E = orc.encode(sparse(rng, m, n, 0.5))
    X = rng.uniform(-1, 1, (n, Cc)).astype(np.float32)
    W = sparse(rng, 3000, 200, 0.3)
    E2 = orc.encode(W)
    h = lib.ell_create(E.Wd, E.idx, E.nnz, E.n)
    dX, dW = torch.from_numpy(X).to(cuda), torch.from_numpy(W).to(cuda)
    dY = [torch.zeros((m, Cc), device=cuda) for _ in range(300)]
    dx, dy = torch.ones((200, 1), device=cuda), torch.zeros((3000, 1), device=cuda)
    want, want2 = orc.spmm(E, X, None), orc.spmm(E2, np.ones((200, 1), np.float32), None)
    torch.cuda.synchronize()
    with Stream(lib) as st:
        def products():
            for y in dY:
                h.spmm(dX.data_ptr(), Cc, Cc, 0, 0, y.data_ptr(), Cc, st)

        def handles():
            for k in range(40):
                h2 = lib.ell_encode_device(dW.data_ptr(), 3000, 200, st)
                h2.spmm(dx.data_ptr(), 1, 1, 0, 0, dy.data_ptr(), 1, st)
                lib.spx_stream_sync(st)
                assert_bit_equal(dy.cpu().numpy(), want2, f"handle {k}")
                h2.close()
        together(products, handles)
        lib.spx_stream_sync(st)
        for k, y in enumerate(dY):
            assert_bit_equal(y.cpu().numpy(), want, f"product {k}")


def test_handles_come_and_go_beside_another_threads_capture(lib, orc, cuda):
    """A graph that one thread records survives another thread making, using and destroying handles and growing their
    scratch (spx_graph_capture_begin keeps other threads' calls apart)."""
    rng = np.random.default_rng(6)
    E = orc.encode(sparse(rng, 300, 400, 0.2))
    X = rng.uniform(-1, 1, (400, 48)).astype(np.float32)
    want = orc.spmm(E, X, None)
    h = lib.ell_create(E.Wd, E.idx, E.nnz, E.n)
    dX, dY = torch.from_numpy(X).to(cuda), torch.zeros((300, 48), device=cuda)
    begun, done = threading.Event(), threading.Event()
    torch.cuda.synchronize()

    def records():
        with Stream(lib) as st:
            try:
                h.spmm(dX.data_ptr(), 48, 48, 0, 0, dY.data_ptr(), 48, st)
                lib.spx_stream_sync(st)
                lib.spx_graph_capture_begin(st)
                h.spmm(dX.data_ptr(), 48, 48, 0, 0, dY.data_ptr(), 48, st)
            finally:
                begun.set()
            done.wait(60)
            h.spmm(dX.data_ptr(), 48, 48, 0, 0, dY.data_ptr(), 48, st)
            graph = C.c_void_p()
            lib.spx_graph_capture_end(st, C.byref(graph))
            lib.spx_memset(dY.data_ptr(), 0, dY.numel() * 4, st)
            lib.spx_graph_launch(graph, st)
            lib.spx_stream_sync(st)
            lib.spx_graph_destroy(graph)
        assert_bit_equal(dY.cpu().numpy(), want, "replay")

    def others():
        begun.wait(60)
        try:
            for k in range(3):
                h2 = lib.ell_create(E.Wd, E.idx, E.nnz, E.n)
                assert_bit_equal(h2.spmm_host(X[:, :8].copy(), None), want[:, :8], "host call")
                assert_bit_equal(h2.spmm_host(X, None), want, "host call, more scratch")
                h2.close()
        finally:
            done.set()
    together(records, others)


@pytest.mark.parametrize("m,n,Cc", [(200, 300, 1), (200, 300, 8), (300, 2000, 17), (700, 3000, 48), (4096, 4100, 64)])
def test_host_calls_follow_the_default_stream(lib, orc, cuda, m, n, Cc):
    """Operands in page-locked memory that a copy on the default stream is still to fill: the call comes after it,
    as it does when it runs on that stream itself.  The result's old contents are still being read, too."""
    rng = np.random.default_rng([m, n, Cc])
    E = orc.encode(sparse(rng, m, n, 0.1))
    X = rng.uniform(-1, 1, (n, Cc)).astype(np.float32)
    b = rng.standard_normal(m).astype(np.float32)
    h = lib.ell_create(E.Wd, E.idx, E.nnz, E.n)
    want = orc.spmm(E, X, b)
    hX, hB, hY = torch.zeros((n, Cc)).pin_memory(), torch.zeros(m).pin_memory(), torch.full((m, Cc), 5.0).pin_memory()
    dX, dB, old = torch.from_numpy(X).to(cuda), torch.from_numpy(b).to(cuda), torch.zeros((m, Cc), device=cuda)
    hog = torch.empty(1 << 30, dtype=torch.uint8, device=cuda)
    h.spmm_host(X, b)
    torch.cuda.synchronize()
    for _ in range(40):                     # some milliseconds on the default stream
        lib.spx_memset(hog.data_ptr(), 1, hog.numel(), 0)
    lib.spx_memcpy_d2h(hX.data_ptr(), dX.data_ptr(), X.nbytes, 0)
    lib.spx_memcpy_d2h(hB.data_ptr(), dB.data_ptr(), b.nbytes, 0)
    lib.spx_memcpy_h2d(old.data_ptr(), hY.data_ptr(), hY.numel() * 4, 0)
    if Cc == 1:
        lib.spx_spmv_host(h.h, hX.data_ptr(), hB.data_ptr(), hY.data_ptr())
        bound = orc.absbound(E, X[:, 0].copy(), b)
        assert (np.abs(hY.numpy()[:, 0] - want[:, 0]) <= 1e-5 * bound).all()
    else:
        lib.spx_spmm_host(h.h, hX.data_ptr(), Cc, hB.data_ptr(), 0, hY.data_ptr())
        assert_bit_equal(hY.numpy(), want, "host call")
    assert bool((old == 5.0).all())


@pytest.mark.parametrize("Cc", [160, 77])
def test_products_beside_the_same_threads_capture(lib, orc, cuda, Cc):
    """While a thread records a graph on one stream, its products on another stream may build the block kernel's form of
    a matrix and take scratch: the graph survives that."""
    rng = np.random.default_rng(8)
    m, n = 1312, 2080                           # takes the block kernel at both widths, from the second call on
    E = orc.encode(sparse(rng, m, n, 0.5))
    X = rng.uniform(-1, 1, (n, Cc)).astype(np.float32)
    want = orc.spmm(E, X, None)
    h, small = lib.ell_create(E.Wd, E.idx, E.nnz, E.n), lib.ell_create(E.Wd, E.idx, E.nnz, E.n)
    dX, dY, dZ = torch.from_numpy(X).to(cuda), torch.zeros((m, Cc), device=cuda), torch.zeros((m, Cc), device=cuda)
    torch.cuda.synchronize()
    with Stream(lib) as st, Stream(lib) as free:
        lib.spx_graph_capture_begin(st)
        small.spmm(dX.data_ptr(), Cc, Cc, 0, 0, dZ.data_ptr(), Cc, st)
        for k in range(3):
            h.spmm(dX.data_ptr(), Cc, Cc, 0, 0, dY.data_ptr(), Cc, free)
        small.spmm(dX.data_ptr(), Cc, Cc, 0, 0, dZ.data_ptr(), Cc, st)
        graph = C.c_void_p()
        lib.spx_graph_capture_end(st, C.byref(graph))
        lib.spx_graph_launch(graph, st)
        lib.spx_stream_sync(st)
        lib.spx_stream_sync(free)
        lib.spx_graph_destroy(graph)
    assert_bit_equal(dY.cpu().numpy(), want, "beside the capture")
    assert_bit_equal(dZ.cpu().numpy(), want, "replay")


@pytest.mark.parametrize("memory", ["pageable", "pinned", "pinned X", "pinned Y"])
@pytest.mark.parametrize("m,n,Cc", [(4100, 4100, 64), (1500, 1400, 192), (1031, 1500, 256), (4096, 1024, 320)])
def test_host_product_in_two_panels(lib, orc, cuda, m, n, Cc, memory):
    """Operands of 1 MB and more whose width is a multiple of 64 go in two column panels: every kind of memory, with and
    without bias, several calls with changing operands."""
    rng = np.random.default_rng([m, n, Cc])
    E = orc.encode(sparse(rng, m, n, 0.03))
    h = lib.ell_create(E.Wd, E.idx, E.nnz, E.n)
    hX = torch.zeros((n, Cc))
    hY = torch.zeros((m, Cc))
    if memory in ("pinned", "pinned X"):
        hX = hX.pin_memory()
    if memory in ("pinned", "pinned Y"):
        hY = hY.pin_memory()
    before = lib.spx_launch_count()
    for k in range(4):
        hX.numpy()[:] = rng.uniform(-1, 1, (n, Cc))
        b = rng.standard_normal(m).astype(np.float32) if k % 2 else None
        hY.fill_(float("nan"))
        lib.spx_spmm_host(h.h, hX.data_ptr(), Cc, vp(b) if k % 2 else 0, k % 2, hY.data_ptr())
        assert_bit_equal(hY.numpy(), orc.spmm(E, hX.numpy(), b, act=k % 2), f"call {k}")
    assert lib.spx_launch_count() - before >= 8, "not in two panels"


def test_host_product_into_pageable_memory_keeps_up(lib, cuda):
    """A result in ordinary memory costs a copy more than one in page-locked memory, not a copy per row: 0.7 ms against
    0.5 here, 5 ms when it was fetched row by row."""
    import time
    m, n, Cc = 20000, 3000, 128
    g = torch.Generator(device="cuda").manual_seed(3)
    W = torch.rand((m, n), device=cuda, generator=g)
    W[torch.rand((m, n), device=cuda, generator=g) >= 0.02] = 0
    h = lib.ell_encode_device(W.data_ptr(), m, n)
    hX, hY, pY = torch.rand((n, Cc)), torch.zeros((m, Cc)), torch.zeros((m, Cc)).pin_memory()

    def least(y):
        t = []
        for k in range(12):
            t0 = time.perf_counter()
            lib.spx_spmm_host(h.h, hX.data_ptr(), Cc, 0, 0, y.data_ptr())
            t.append(time.perf_counter() - t0)
        return min(t)
    pinned, pageable = least(pY), least(hY)
    assert pageable < 4 * pinned, (pageable, pinned)


def test_two_threads_make_host_calls(lib, orc, cuda):
    """Host calls on different handles from two threads, on every route: small, medium, two panels, one column."""
    rng = np.random.default_rng(9)
    jobs = []
    for i in range(2):
        cases = []
        for (m, n, Cc) in [(300, 400, 8), (500, 900, 30), (2000, 3000, 100), (2200, 2100, 128), (700, 5000, 1)]:
            E = orc.encode(sparse(rng, m, n, 0.05))
            X = rng.uniform(-1, 1, (n, Cc)).astype(np.float32)
            cases.append((lib.ell_create(E.Wd, E.idx, E.nnz, E.n), X, orc.spmm(E, X, None)))

        def job(cases=cases):
            for k in range(25):
                for h, X, want in cases:
                    assert_bit_equal(h.spmm_host(X, None), want, f"call {k}")
        jobs.append(job)
    together(*jobs)


@pytest.mark.parametrize("slices", [1, 4, 16])
def test_slices_are_complete_on_a_stream_of_the_callers(lib, orc, cuda, slices):
    """The first exchange call makes the slices and multiplies them at once, here on a non-blocking stream."""
    rng = np.random.default_rng(12)
    m, n, Cc = 900, 700, 64
    E = orc.encode(sparse(rng, m, n, 0.1))
    X = rng.uniform(-1, 1, (n, Cc)).astype(np.float32)
    want = orc.spmm(E, X, None)
    dX = torch.from_numpy(X).to(cuda)
    torch.cuda.synchronize()
    for k in range(20):
        h = lib.ell_create(E.Wd, E.idx, E.nnz, E.n)
        dY = torch.zeros((m, Cc), device=cuda)
        torch.cuda.synchronize()
        with Stream(lib) as st:
            one = (C.c_void_p * 1)(dY.data_ptr())
            lib.spx_spmm_exchange(h.h, dX.data_ptr(), Cc, Cc, 0, 0, one, 1, 0, 0, Cc, slices, st)
        assert_bit_equal(dY.cpu().numpy(), want, f"handle {k}")
