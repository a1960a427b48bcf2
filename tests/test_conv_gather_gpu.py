"""GPU: the convolution that gathers its operands (conv_gather.cu), forced, against the oracle bit for bit: edges of its tiles of
positions, of batches of 32 entries and groups of 8 and 4, both widths of operands, all layouts; and when it is chosen.  The
switch is read once per process, so the forced cases run in a child."""
import ctypes
import os
import threading

import numpy as np
import pytest
import torch

import spx_ctypes as sx
from conftest import assert_bit_equal
from test_conv_tmem_gpu import assert_ran, child, fill_device, kernels_of, waits_for_the_device
from test_parity_gpu import as_layout, dev, gpu_ell, ptr, sparse

pytestmark = pytest.mark.gpu
forced = pytest.mark.skipif(os.environ.get("SPX_CONV_GATHER") != "2", reason="runs in a child process")
chosen = pytest.mark.skipif(any(k.startswith("SPX_CONV") for k in os.environ), reason="the choice is forced")

# B, Cin, Cout, H, W, (kH, kW), (sH, sW), (dH, dW), density
CASES = [(1, 3, 8, 4, 8, (3, 3), (1, 1), (1, 1), 0.5),          # one tile of 32 positions
         (1, 5, 9, 3, 11, (3, 3), (1, 1), (1, 1), 1.0),         # a channel and a position over; rows of 45 entries
         (3, 16, 33, 13, 12, (1, 1), (2, 2), (1, 1), 0.4),      # a tap, a stride
         (5, 33, 7, 7, 6, (1, 1), (1, 1), (1, 1), 1.0),         # rows of 33 entries, fewer channels than warps
         (4, 32, 24, 9, 9, (1, 1), (2, 1), (1, 1), 1.0),        # of 32, four batch entries a lane
         (12, 4, 40, 17, 5, (5, 5), (2, 2), (1, 1), 0.2),
         (32, 3, 65, 21, 20, (3, 3), (2, 1), (1, 1), 0.3),
         (8, 6, 16, 15, 14, (3, 3), (1, 2), (2, 3), 0.4),       # dilated
         (2, 3, 17, 9, 10, (4, 8), (1, 1), (1, 1), 0.5),        # 32 taps
         (2, 3, 17, 9, 14, (3, 11), (1, 1), (1, 1), 0.5),       # 33: not for this kernel
         (1, 2, 130, 66, 65, (3, 3), (1, 1), (1, 1), 0.6),      # many positions and channels, short rows
         (32, 3, 200, 30, 31, (1, 1), (2, 2), (1, 1), 0.7),
         (4, 64, 24, 17, 13, (3, 3), (1, 1), (1, 1), 0.3),      # one batch entry a lane although four are contiguous
         (28, 24, 104, 14, 14, (3, 3), (1, 1), (1, 1), 0.3)]    # and of four positions


@forced
@pytest.mark.parametrize("off", [0, 1])
@pytest.mark.parametrize("layout", [sx.LAYOUT_PF, sx.LAYOUT_NCHW, sx.LAYOUT_FMAJOR])
@pytest.mark.parametrize("B,Cin,Cout,H,W,k,s,d,density", CASES)
def test_forced_gather(lib, orc, cuda, layout, off, B, Cin, Cout, H, W, k, s, d, density):
    """off: the tensors start a float off 16 bytes.  The first tap of the first output meets padding; weights there are
    infinite in one row, so that w * 0 shows as it does in the reference."""
    (kH, kW), (sH, sW), (dH, dW) = k, s, d
    rng = np.random.default_rng([B, Cin, Cout, H, W, kH])
    wt = sparse(rng, Cout, Cin * kH * kW, density)
    wt[Cout // 2] = 0
    wt[0, 0] = np.inf
    x = rng.standard_normal((B, Cin, H, W)).astype(np.float32)
    x[-1, -1, -1, -1] = np.nan
    bias = rng.standard_normal(Cout).astype(np.float32)
    pH, pW = (kH // 2) * dH, (kW // 2) * dW
    src, E = as_layout(x, layout), orc.encode(wt)
    want = orc.conv2d(E, dict(Cin=Cin, kH=kH, kW=kW, sH=sH, sW=sW, pH=pH, pW=pW, dH=dH, dW=dW, H=H, W=W), layout, src, B, bias, 1).reshape(-1)
    h, g = gpu_ell(lib, E), sx.conv_geom(Cin, Cout, kH, kW, H, W, sH, sW, pH, pW, dH, dW)
    dX = torch.empty(src.size + 4, device=cuda)
    dX[off:off + src.size] = dev(src.reshape(-1), cuda)
    dB = dev(bias, cuda)
    out = torch.full((want.size + 8,), 7.0, device=cuda)
    call = lambda: h.conv2d(g, layout, dX.data_ptr() + 4 * off, B, ptr(dB), sx.ACT_RELU, out.data_ptr() + 16 + 4 * off)
    call()
    names = kernels_of(call)
    if kH * kW > 32:
        assert names is None or "conv_gather_kernel" not in names
    elif not (k == (1, 1) and s == (1, 1)):                 # such a one is an SpMM
        assert_ran(names, "conv_gather_kernel")
    got = out.cpu().numpy()
    y, nan = got[4 + off:4 + off + want.size], np.isnan(want)
    assert (np.isnan(y) == nan).all()
    assert_bit_equal(np.where(nan, 0, y).astype(np.float32), np.where(nan, 0, want).astype(np.float32), "conv")
    assert (got[:4 + off] == 7.0).all() and (got[4 + off + want.size:] == 7.0).all()


@forced
@pytest.mark.parametrize("B,layout", [(1, sx.LAYOUT_NCHW), (8, sx.LAYOUT_PF)])
def test_forced_gather_any_column_order(lib, orc, cuda, B, layout):
    """Rows whose columns do not ascend (only raw arrays have such): entries are added in storage order."""
    rng = np.random.default_rng(4)
    Cin, Cout, H = 6, 20, 9
    E = orc.encode(sparse(rng, Cout, Cin * 9, 0.4))
    for i in range(Cout):
        p = rng.permutation(E.nnz[i])
        E.idx[i, :E.nnz[i]], E.Wd[i, :E.nnz[i]] = E.idx[i, :E.nnz[i]][p], E.Wd[i, :E.nnz[i]][p]
    src = as_layout(rng.standard_normal((B, Cin, H, H)).astype(np.float32), layout)
    want = orc.conv2d(E, dict(Cin=Cin, kH=3, kW=3, sH=1, sW=1, pH=1, pW=1, dH=1, dW=1, H=H, W=H), layout, src, B, None, 0)
    h, dX, dY = gpu_ell(lib, E), dev(src, cuda), torch.empty(want.shape, device=cuda)
    h.conv2d(sx.conv_geom(Cin, Cout, 3, 3, H, H, 1, 1, 1, 1), layout, ptr(dX), B, None, 0, ptr(dY))
    assert_bit_equal(dY.cpu().numpy(), want, "permuted rows")


@chosen
@pytest.mark.parametrize("shared,kernel", [(False, "conv_gather_kernel"), (True, "conv_rbm_tile_kernel")])
def test_choice_of_gathering(lib, orc, cuda, shared, kernel):
    """Rows that share all their columns are merged at a quarter of the work: 54 -> 100 channels, 5 x 5, batch 2 23 us against 34
    gathered; of rows that share nothing the merged kernel takes longer."""
    rng = np.random.default_rng(13)
    Cin, Cout, H, W, B = 54, 100, 8, 63, 2
    wt = rng.standard_normal((Cout, Cin * 25)).astype(np.float32)
    wt[np.broadcast_to(rng.random((1 if shared else Cout, Cin * 25)) >= 0.436, wt.shape)] = 0
    E = orc.encode(wt)
    src = as_layout(rng.standard_normal((B, Cin, H, W)).astype(np.float32), sx.LAYOUT_PF)
    want = orc.conv2d(E, dict(Cin=Cin, kH=5, kW=5, sH=1, sW=1, pH=2, pW=2, dH=1, dW=1, H=H, W=W), sx.LAYOUT_PF, src, B, None, 0)
    h, dX, dY = gpu_ell(lib, E), dev(src, cuda), torch.empty(want.shape, device=cuda)
    g = sx.conv_geom(Cin, Cout, 5, 5, H, W, 1, 1, 2, 2)
    for _ in range(2):
        dY.fill_(float("nan"))
        assert_ran(kernels_of(lambda: h.conv2d(g, sx.LAYOUT_PF, ptr(dX), B, None, 0, ptr(dY))), kernel)
        assert_bit_equal(dY.cpu().numpy(), want, kernel)


@chosen
@pytest.mark.parametrize("B,Cin,Cout,H,k,s,density", [(4, 19, 70, 84, 3, 12, 0.05), (1, 28, 158, 61, 4, 14, 0.23),      # 39 and 80 us against 4 and 7
                                                      (3, 14700, 40, 6, 3, 1, 0.004), (16, 5300, 33, 5, 5, 2, 0.004)])  # 132300 columns and more
def test_choice_where_nothing_is_merged(lib, orc, cuda, B, Cin, Cout, H, k, s, density):
    """Strides that leave no patch to the merged kernel, and more columns than it takes: the call is compared with the per-row kernel,
    and no columns are counted."""
    rng = np.random.default_rng([B, Cin])
    E = orc.encode(sparse(rng, Cout, Cin * k * k, density))
    src = as_layout(rng.standard_normal((B, Cin, H, H)).astype(np.float32), sx.LAYOUT_PF)
    want = orc.conv2d(E, dict(Cin=Cin, kH=k, kW=k, sH=s, sW=s, pH=k // 2, pW=k // 2, dH=1, dW=1, H=H, W=H), sx.LAYOUT_PF, src, B, None, 0)
    h, g, dX, dY = gpu_ell(lib, E), sx.conv_geom(Cin, Cout, k, k, H, H, s, s, k // 2, k // 2), dev(src, cuda), torch.empty(want.shape, device=cuda)
    names = kernels_of(lambda: h.conv2d(g, sx.LAYOUT_PF, ptr(dX), B, None, 0, ptr(dY)))
    assert_ran(names, "conv_gather_kernel")
    assert names is None or "union_count_kernel" not in names
    assert_bit_equal(dY.cpu().numpy(), want, "gathered")


@chosen
def test_tiled_call_recorded_after_gathered_ones(lib, orc, cuda):
    """Calls that gather need no merged weights; a later one that is recorded does, and has them: in the graph, and in an
    eager call before the graph is launched."""
    rng = np.random.default_rng(14)
    C, H = 40, 12
    E = orc.encode(sparse(rng, C, C * 9, 0.3))
    gd = dict(Cin=C, kH=3, kW=3, sH=1, sW=1, pH=1, pW=1, dH=1, dW=1, H=H, W=H)
    h, g = gpu_ell(lib, E), sx.conv_geom(C, C, 3, 3, H, H, 1, 1, 1, 1)
    x = rng.standard_normal((32, C, H, H)).astype(np.float32)
    one, many = as_layout(x[:1], sx.LAYOUT_PF), as_layout(x, sx.LAYOUT_PF)
    w1, w32 = orc.conv2d(E, gd, sx.LAYOUT_PF, one, 1, None, 0), orc.conv2d(E, gd, sx.LAYOUT_PF, many, 32, None, 0)
    d1, d32, y1, y32, z32 = dev(one, cuda), dev(many, cuda), torch.empty(w1.shape, device=cuda), torch.empty(w32.shape, device=cuda), torch.empty(w32.shape, device=cuda)
    assert_ran(kernels_of(lambda: h.conv2d(g, sx.LAYOUT_PF, ptr(d1), 1, None, 0, ptr(y1))), "conv_gather_kernel")
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        h.conv2d(g, sx.LAYOUT_PF, ptr(d32), 32, None, 0, ptr(y32), torch.cuda.current_stream().cuda_stream)
    h.conv2d(g, sx.LAYOUT_PF, ptr(d32), 32, None, 0, ptr(z32))
    assert_bit_equal(z32.cpu().numpy(), w32, "eager, before the graph")
    graph.replay()
    torch.cuda.synchronize()
    assert_bit_equal(y32.cpu().numpy(), w32, "replayed")
    assert_bit_equal(y1.cpu().numpy(), w1, "gathered")


def merged_after_gathered(lib, orc, cuda, batches):
    """A handle whose first call gathers (so that nothing is merged yet), and a call per batch size; 32 is merged."""
    rng, C, H = np.random.default_rng(15), 64, 28
    E = orc.encode(sparse(rng, C, C * 9, 0.3))
    gd = dict(Cin=C, kH=3, kW=3, sH=2, sW=2, pH=1, pW=1, dH=1, dW=1, H=H, W=H)
    h, g = gpu_ell(lib, E), sx.conv_geom(C, C, 3, 3, H, H, 2, 2, 1, 1)
    x = rng.standard_normal((max(batches), C, H, H)).astype(np.float32)
    runs = []
    for B in batches:
        src = as_layout(x[:B], sx.LAYOUT_PF)
        want = orc.conv2d(E, gd, sx.LAYOUT_PF, src, B, None, 0)
        dX, dY = dev(src, cuda), torch.full(want.shape, float("nan"), device=cuda)
        runs.append((B, dX, dY, want, torch.cuda.Stream()))
    one, y1 = dev(as_layout(x[:1], sx.LAYOUT_PF), cuda), torch.empty((C, H // 2, H // 2, 1), device=cuda)
    assert_ran(kernels_of(lambda: h.conv2d(g, sx.LAYOUT_PF, ptr(one), 1, None, 0, ptr(y1))), "conv_gather_kernel")
    torch.cuda.synchronize()
    return h, g, runs, lambda run: h.conv2d(g, sx.LAYOUT_PF, ptr(run[1]), run[0], None, 0, ptr(run[2]), run[4].cuda_stream)


@chosen
def test_merged_weights_for_two_streams(lib, orc, cuda):
    """The first merged call waits behind a long kernel, one on another stream does not: it has the weights all the same."""
    h, g, runs, call = merged_after_gathered(lib, orc, cuda, [32, 32])

    def both():
        with torch.cuda.stream(runs[0][4]):
            torch.cuda._sleep(200_000_000)
        for run in runs:
            call(run)

    assert_ran(kernels_of(both), "conv_rbm_tile_kernel")
    for B, _, dY, want, _ in runs:
        assert_bit_equal(dY.cpu().numpy(), want, f"batch {B}")


@chosen
def test_merged_weights_for_several_threads(lib, orc, cuda):
    """A handle's first merged calls, made by eight threads on streams of their own at once."""
    for _ in range(4):
        h, g, runs, call = merged_after_gathered(lib, orc, cuda, [32, 64, 36, 32, 40, 32, 64, 32])
        start, errors = threading.Barrier(len(runs)), []

        def work(run):
            try:
                start.wait()
                for _ in range(3):
                    call(run)
            except Exception as e:      # noqa: BLE001
                errors.append(e)

        threads = [threading.Thread(target=work, args=(run,)) for run in runs]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        torch.cuda.synchronize()
        assert not errors, errors
        for B, _, dY, want, _ in runs:
            assert_bit_equal(dY.cpu().numpy(), want, f"batch {B}")


@chosen
@pytest.mark.parametrize("B", [1, 3, 32])
def test_eager_call_between_recording_and_replay(lib, orc, cuda, B):
    """A handle's very first call is recorded; an eager one before the graph has run finds what it needs all the same, and so
    does one on another stream behind which a long kernel is queued."""
    rng, C, H = np.random.default_rng(16), 64, 28
    E = orc.encode(sparse(rng, C, C * 9, 0.3))
    src = as_layout(rng.standard_normal((B, C, H, H)).astype(np.float32), sx.LAYOUT_PF)
    want = orc.conv2d(E, dict(Cin=C, kH=3, kW=3, sH=2, sW=2, pH=1, pW=1, dH=1, dW=1, H=H, W=H), sx.LAYOUT_PF, src, B, None, 0)
    h, g, dX = gpu_ell(lib, E), sx.conv_geom(C, C, 3, 3, H, H, 2, 2, 1, 1), dev(src, cuda)
    Y = [torch.full(want.shape, float("nan"), device=cuda) for _ in range(4)]
    other, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    call = lambda y, stream=0: h.conv2d(g, sx.LAYOUT_PF, ptr(dX), B, None, 0, ptr(y), stream)
    with torch.cuda.graph(graph):
        call(Y[0], torch.cuda.current_stream().cuda_stream)
    call(Y[1])
    with torch.cuda.stream(other):
        torch.cuda._sleep(100_000_000)
    call(Y[2], other.cuda_stream)
    call(Y[3])
    graph.replay()
    torch.cuda.synchronize()
    for k, y in enumerate(Y):
        assert_bit_equal(y.cpu().numpy(), want, f"call {k}")


def two_kernel_shapes(lib, orc, cuda, Cin, Cout, H, B, density, full_row=False):
    """A handle, and what a 3 x 3 and a 1 x 9 kernel over its columns give: (geometry, batch, input, result) each."""
    rng = np.random.default_rng(17)
    wt = sparse(rng, Cout, Cin * 9, density)
    if full_row:
        wt[0] = 1
    E = orc.encode(wt)
    x = rng.standard_normal((max(B), Cin, H, H)).astype(np.float32)
    runs = []
    for b in B:
        for kH, kW in ((3, 3), (1, 9)):
            src = as_layout(x[:b], sx.LAYOUT_PF)
            gd = dict(Cin=Cin, kH=kH, kW=kW, sH=2, sW=2, pH=kH // 2, pW=kW // 2, dH=1, dW=1, H=H, W=H)
            runs.append((sx.conv_geom(Cin, Cout, kH, kW, H, H, 2, 2, kH // 2, kW // 2), b, dev(src, cuda), orc.conv2d(E, gd, sx.LAYOUT_PF, src, b, None, 0)))
    return gpu_ell(lib, E), runs


@chosen
def test_two_kernel_shapes_of_a_handle(lib, orc, cuda):
    """Graphs of one kernel shape keep theirs when another one is recorded and called; calls of both alternate on two streams,
    one of which is held up."""
    h, runs = two_kernel_shapes(lib, orc, cuda, 64, 64, 28, [1, 32], 0.3)
    graphs, outs = [], [torch.full(want.shape, float("nan"), device=cuda) for *_, want in runs]
    for (g, B, dX, want), dY in zip(runs, outs):
        graphs.append(torch.cuda.CUDAGraph())
        with torch.cuda.graph(graphs[-1]):
            h.conv2d(g, sx.LAYOUT_PF, ptr(dX), B, None, 0, ptr(dY), torch.cuda.current_stream().cuda_stream)
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    with torch.cuda.stream(streams[0]):
        torch.cuda._sleep(100_000_000)
    eager = []
    for _ in range(2):
        for k, (g, B, dX, want) in enumerate(runs):
            eager.append((torch.full(want.shape, float("nan"), device=cuda), want))
            torch.cuda.current_stream().synchronize()
            h.conv2d(g, sx.LAYOUT_PF, ptr(dX), B, None, 0, ptr(eager[-1][0]), streams[k % 2].cuda_stream)
    torch.cuda.synchronize()
    for graph in graphs:
        graph.replay()
    torch.cuda.synchronize()
    for dY, want in eager + [(dY, run[3]) for dY, run in zip(outs, runs)]:
        assert_bit_equal(dY.cpu().numpy(), want, "two kernel shapes")


no_memory = pytest.mark.skipif(os.environ.get("SPX_TEST_NO_MEMORY") != "1", reason="runs in a child process")


@no_memory
def test_second_kernel_shape_without_memory(lib, orc, cuda):
    """There is no room for another kernel shape's tables: the ids are decoded by the general kernel, and no call waits for the
    device to look for memory again."""
    h, runs = two_kernel_shapes(lib, orc, cuda, 512, 2048, 4, [4], 0.01, full_row=True)     # a tap table is 38 MB
    outs = [torch.full(want.shape, float("nan"), device=cuda) for *_, want in runs]
    call = lambda k: h.conv2d(runs[k][0], sx.LAYOUT_PF, ptr(runs[k][2]), runs[k][1], None, 0, ptr(outs[k]))
    call(0)
    assert not waits_for_the_device(lambda: None)           # (makes the stream while there is room)
    held = fill_device(lib, 4 << 20, 16 << 20)
    try:
        for again in (False, True):
            outs[1].fill_(float("nan"))
            waited = waits_for_the_device(lambda: call(1))
            assert not (again and waited), "waited for another stream's work"
            assert_bit_equal(outs[1].cpu().numpy(), runs[1][3], "no room")
            call(0)
            assert_bit_equal(outs[0].cpu().numpy(), runs[0][3], "the first kernel shape")
    finally:
        for p in held:
            lib.spx_free(p)
    call(1)
    assert_bit_equal(outs[1].cpu().numpy(), runs[1][3], "room again")


def exhaust(lib):
    """Takes all device memory, what the library's pool has left included."""
    held, handles = fill_device(lib, 64 << 20, 16 << 20), []
    for m in (1 << 22, 1 << 20, 1 << 16, 1 << 12, 1 << 8, 1 << 6):   # 12 bytes a row
        nnz = np.zeros(m, np.uint32)
        try:
            while True:
                handles.append(lib.ell_create(np.zeros((m, 0), np.float32), np.zeros((m, 0), np.uint32), nnz, 1))
        except sx.SpxError as e:
            assert e.status == 3, e
    return held, handles


@no_memory
def test_calls_that_are_sure_to_gain_without_memory(lib, orc, cuda):
    """A call that would count the shared columns finds no memory for it: from then on the calls that depend on the count take
    the tiled kernels, and those that are faster gathered whatever it says still are."""
    rng, C, H = np.random.default_rng(18), 1024, 14         # the count takes 2 KB
    E = orc.encode(sparse(rng, C, 64 * 9, 0.3))
    g, outs = sx.conv_geom(64, C, 3, 3, H, H, 2, 2, 1, 1), {}
    gd = dict(Cin=64, kH=3, kW=3, sH=2, sW=2, pH=1, pW=1, dH=1, dW=1, H=H, W=H)
    x = rng.standard_normal((32, 64, H, H)).astype(np.float32)
    for B in (1, 32):
        src = as_layout(x[:B], sx.LAYOUT_PF)
        want = orc.conv2d(E, gd, sx.LAYOUT_PF, src, B, None, 0)
        outs[B] = dev(src, cuda), torch.full(want.shape, float("nan"), device=cuda), want

    def call(h, B, stream=0):
        h.conv2d(g, sx.LAYOUT_PF, ptr(outs[B][0]), B, None, 0, ptr(outs[B][1]), stream)

    def check(B):
        assert_bit_equal(outs[B][1].cpu().numpy(), outs[B][2], f"batch {B}")
        outs[B][1].fill_(float("nan"))

    other, h = gpu_ell(lib, E), gpu_ell(lib, E)             # (the other one: kernels are loaded while there is room)
    assert_ran(kernels_of(lambda: call(other, 1)), "conv_gather_kernel")
    assert_ran(kernels_of(lambda: call(other, 32)), "union_count_kernel")
    call(h, 1)
    with torch.cuda.graph(torch.cuda.CUDAGraph()):          # builds the merged weights without a count
        call(h, 32, torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    before = lib.spx_launch_count()
    held, handles = exhaust(lib)
    try:
        call(h, 32)
        assert lib.spx_launch_count() == before + 1, "there was memory for the count"
        check(32)
    finally:
        for p in held:
            lib.spx_free(p)
        handles.clear()
    for B, kernel in ((1, "conv_gather_kernel"), (32, "conv_rbm_tile_kernel")):
        assert_ran(kernels_of(lambda: call(h, B)), kernel)
        check(B)


def test_without_memory():
    child(["test_conv_gather_gpu.py"], "second_kernel_shape_without or sure_to_gain_without", {"SPX_TEST_NO_MEMORY": "1"})


@chosen
@pytest.mark.parametrize("first", [1, 16])
def test_recorded_calls_that_need_more_scratch(lib, orc, cuda, first):
    """NCHW calls copy their input: one that is recorded after smaller ones (gathered, or with less scratch) gets what it needs, and
    its graph keeps that when a later call needs more."""
    rng, C, H = np.random.default_rng(19), 128, 14
    E = orc.encode(sparse(rng, C, C * 9, 0.5))
    h, g, x = gpu_ell(lib, E), sx.conv_geom(C, C, 3, 3, H, H, 1, 1, 1, 1), rng.standard_normal((64, C, H, H)).astype(np.float32)
    runs = {}
    for B in (first, 32, 48, 64):
        want = orc.conv2d(E, dict(Cin=C, kH=3, kW=3, sH=1, sW=1, pH=1, pW=1, dH=1, dW=1, H=H, W=H), sx.LAYOUT_NCHW, x[:B], B, None, 0)
        runs[B] = dev(x[:B], cuda), torch.full(want.shape, float("nan"), device=cuda), want
    call = lambda B: h.conv2d(g, sx.LAYOUT_NCHW, ptr(runs[B][0]), B, None, 0, ptr(runs[B][1]), torch.cuda.current_stream().cuda_stream)
    call(first)
    graphs = []
    for B in (32, 48):
        graphs.append(torch.cuda.CUDAGraph())
        with torch.cuda.graph(graphs[-1]):
            call(B)
    assert_ran(kernels_of(lambda: call(64)), "transpose2d_kernel")
    for graph in graphs * 2:
        graph.replay()
    torch.cuda.synchronize()
    for B, (_, dY, want) in runs.items():
        assert_bit_equal(dY.cpu().numpy(), want, f"batch {B}")


@chosen
def test_recording_while_a_table_is_being_built(lib, orc, cuda):
    """The build of the tables is queued behind a long kernel when the same stream begins to record calls that need them: those
    wait for it, and calls on another stream come behind it."""
    rng, C, H = np.random.default_rng(20), 64, 28
    E = orc.encode(sparse(rng, C, C * 9, 0.3))
    h, g, x = gpu_ell(lib, E), sx.conv_geom(C, C, 3, 3, H, H, 2, 2, 1, 1), rng.standard_normal((32, C, H, H)).astype(np.float32)
    stream, other, graph, runs = torch.cuda.Stream(), torch.cuda.Stream(), ctypes.c_void_p(), []
    for B in (1, 32):
        src = as_layout(x[:B], sx.LAYOUT_PF)
        want = orc.conv2d(E, dict(Cin=C, kH=3, kW=3, sH=2, sW=2, pH=1, pW=1, dH=1, dW=1, H=H, W=H), sx.LAYOUT_PF, src, B, None, 0)
        runs.append((B, dev(src, cuda), want, [torch.full(want.shape, float("nan"), device=cuda) for _ in range(3)]))
    call = lambda run, k, st: h.conv2d(g, sx.LAYOUT_PF, ptr(run[1]), run[0], None, 0, ptr(run[3][k]), st.cuda_stream)
    torch.cuda.synchronize()
    with torch.cuda.stream(stream):
        torch.cuda._sleep(200_000_000)
    call(runs[0], 0, stream)                                # batch 1: the tap table alone
    call(runs[0], 1, other)
    lib.spx_graph_capture_begin(stream.cuda_stream)
    for run in runs:
        call(run, 2, stream)
    lib.spx_graph_capture_end(stream.cuda_stream, ctypes.byref(graph))
    call(runs[1], 0, other)
    call(runs[1], 1, stream)
    lib.spx_graph_launch(graph, stream.cuda_stream)
    torch.cuda.synchronize()
    for B, _, want, outs in runs:
        for k, y in enumerate(outs):
            assert_bit_equal(y.cpu().numpy(), want, f"batch {B}, call {k}")
    lib.spx_graph_destroy(graph)


@chosen
def test_recording_a_merged_call_waits_for_no_other_work(lib, orc, cuda):
    """Recording a call that lacks the merged weights builds them at once, beside what other streams do: that kernel is no part
    of the graph."""
    h, g, runs, call = merged_after_gathered(lib, orc, cuda, [32])
    (B, _, dY, want, stream), graph = runs[0], ctypes.c_void_p()
    assert not waits_for_the_device(lambda: None)           # (makes the stream)

    def record():
        lib.spx_graph_capture_begin(stream.cuda_stream)
        call(runs[0])
        lib.spx_graph_capture_end(stream.cuda_stream, ctypes.byref(graph))

    before = lib.spx_launch_count()
    assert not waits_for_the_device(record)
    assert lib.spx_launch_count() == before + 1
    for _ in range(2):
        lib.spx_graph_launch(graph, stream.cuda_stream)
    torch.cuda.synchronize()
    assert lib.spx_launch_count() == before + 3
    assert_bit_equal(dY.cpu().numpy(), want, "replayed")
    lib.spx_graph_destroy(graph)


def test_forced_kernel():
    child(["test_conv_gather_gpu.py", "test_parity_gpu.py", "test_fuzz_gpu.py"],
          "forced_gather or conv_bit_exact or conv_views or conv_random or golden_conv", {"SPX_CONV_GATHER": "2"})
