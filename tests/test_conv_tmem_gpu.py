"""GPU: the convolution with its patch in tensor memory (conv_tmem.cu), forced, against the oracle bit for bit: edges of
tiles, chunks and batch segments, few and many output channels, full and empty rows, infinities under taps that a row
does not store.  The switch is read once per process, so the cases run in a child."""
import ctypes
import os
import subprocess
import sys

import numpy as np
import pytest
import torch

import spx_ctypes as sx
from conftest import assert_bit_equal
from test_parity_gpu import as_layout, dev, gpu_ell, ptr, sparse

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))
forced = pytest.mark.skipif(os.environ.get("SPX_CONV_TMEM") != "2", reason="runs in a child process")

def kernels_of(f):
    """Names of the kernels that f() launches; None where the profiler sees none at all."""
    probe = torch.empty(1000, device="cuda")
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA], acc_events=True) as p:
        probe.sin_()
        f()
        torch.cuda.synchronize()
    names = " ".join(e.key for e in p.key_averages())
    return names.replace("sin_kernel", "") if "sin_kernel" in names else None


def assert_ran(names, kernel):
    assert names is None or kernel in names, names


# B, Cin, Cout, H, W, (kH, kW), (sH, dH, dW), density
CASES = [(32, 6, 64, 6, 8, (3, 3), (1, 1, 1), 0.3),         # one chunk, one unit
         (32, 7, 65, 7, 9, (3, 3), (1, 1, 1), 0.3),         # a chunk of one channel; a block and a position over
         (32, 13, 33, 5, 17, (3, 3), (1, 1, 1), 1.0),       # dense: the most entries a chunk can hold
         (48, 19, 29, 4, 7, (3, 3), (1, 1, 1), 0.2),        # segments of 32 and 16, two patches per CTA
         (60, 5, 40, 9, 9, (3, 3), (1, 1, 1), 0.2),         # all segment widths
         (4, 30, 132, 3, 40, (3, 3), (1, 1, 1), 0.1),       # eight lane groups
         (16, 9, 70, 11, 8, (5, 5), (1, 1, 1), 0.15),
         (8, 8, 36, 12, 12, (7, 7), (1, 1, 1), 0.1),
         (12, 10, 32, 14, 10, (3, 3), (1, 2, 2), 0.3),      # dilated
         (32, 8, 31, 9, 8, (3, 2), (2, 1, 3), 0.3),         # stride along the rows only
         (32, 600, 29, 2, 3, (3, 3), (1, 1, 1), 0.02),      # many chunks, most rows' runs empty
         (64, 12, 256, 56, 56, (3, 3), (1, 1, 1), 0.05)]    # several waves and a tail of half units


@forced
@pytest.mark.parametrize("layout", [sx.LAYOUT_PF, sx.LAYOUT_NCHW, sx.LAYOUT_FMAJOR])
@pytest.mark.parametrize("B,Cin,Cout,H,W,k,sd,density", CASES)
def test_forced_cases(lib, orc, cuda, layout, B, Cin, Cout, H, W, k, sd, density):
    (kH, kW), (sH, dH, dW) = k, sd
    if layout != sx.LAYOUT_PF and H > 50:
        pytest.skip("once is enough at this size")
    rng = np.random.default_rng([B, Cin, Cout, H, W, kH])
    wt = sparse(rng, Cout, Cin * kH * kW, density) * np.float32(0.3)
    wt[Cout // 2] = 0                                       # an empty row
    wt[:, 4 % wt.shape[1]] = 0                              # nobody stores this tap ...
    x = rng.standard_normal((B, Cin, H, W)).astype(np.float32)
    if kH * kW > 4 and H <= 20:
        x[0, 0, 0, 0], x[-1, -1, -1, -1] = np.inf, np.nan   # ... and what others meet comes out as it is
    bias = rng.standard_normal(Cout).astype(np.float32)
    src = as_layout(x, layout)
    E = orc.encode(wt)
    pH, pW = (kH // 2) * dH, (kW // 2) * dW
    gd = dict(Cin=Cin, kH=kH, kW=kW, sH=sH, sW=1, pH=pH, pW=pW, dH=dH, dW=dW, H=H, W=W)
    want = orc.conv2d(E, gd, layout, src, B, bias, 0)
    h = gpu_ell(lib, E)
    g = sx.conv_geom(Cin, Cout, kH, kW, H, W, sH, 1, pH, pW, dH, dW)
    dX, dB = dev(src, cuda), dev(bias, cuda)
    out = torch.full((want.size + 8,), 7.0, device=cuda, dtype=torch.float32)
    call = lambda: h.conv2d(g, layout, ptr(dX), B, ptr(dB), sx.ACT_NONE, out.data_ptr() + 16)
    call()
    assert_ran(kernels_of(call), "conv_tmem_kernel")
    got = out.cpu().numpy()
    nan = np.isnan(want.reshape(-1))
    assert (np.isnan(got[4:-4]) == nan).all()
    assert_bit_equal(np.where(nan, 0, got[4:-4]).astype(np.float32), np.where(nan, 0, want.reshape(-1)).astype(np.float32), "conv")
    assert (got[:4] == 7.0).all() and (got[-4:] == 7.0).all()


@forced
def test_forced_more_shapes_than_forms_and_capture(lib, orc, cuda):
    """One handle under six kernel shapes, the first call of each but one on a stream that records a graph: results are
    the same whether a form could be built or not, also when graphs are replayed after others were built."""
    rng = np.random.default_rng(3)
    Cin, Cout, B, H, W = 8, 32, 32, 12, 12
    wt = sparse(rng, Cout, Cin * 9, 0.3)
    E = orc.encode(wt)
    h = gpu_ell(lib, E)
    x = rng.standard_normal((B, Cin, H, W)).astype(np.float32)
    src = as_layout(x, sx.LAYOUT_PF)
    dX = dev(src, cuda)
    runs = []
    for dil in range(1, 7):
        gd = dict(Cin=Cin, kH=3, kW=3, sH=1, sW=1, pH=0, pW=0, dH=1, dW=1, H=H, W=W)
        gd.update(dH=dil if dil < 6 else 1, dW=1, sH=1 if dil < 6 else 2)
        want = orc.conv2d(E, gd, sx.LAYOUT_PF, src, B, None, 0)
        g = sx.conv_geom(Cin, Cout, 3, 3, H, W, gd["sH"], 1, 0, 0, gd["dH"], 1)
        dY = torch.empty(want.shape, device=cuda)
        if dil == 1:
            # allocates what any kernel needs
            assert_ran(kernels_of(lambda: h.conv2d(g, sx.LAYOUT_PF, ptr(dX), B, None, 0, ptr(dY))), "conv_tmem_kernel")
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            h.conv2d(g, sx.LAYOUT_PF, ptr(dX), B, None, 0, ptr(dY), torch.cuda.current_stream().cuda_stream)
        dZ = torch.empty(want.shape, device=cuda)
        # four forms, the first shapes'; the rest goes without
        assert_ran(kernels_of(lambda: h.conv2d(g, sx.LAYOUT_PF, ptr(dX), B, None, 0, ptr(dZ))), "conv_tmem_kernel" if dil < 5 else "conv_rbm_tile_kernel")
        assert_bit_equal(dZ.cpu().numpy(), want, f"eager {dil}")
        runs.append((graph, dY, want))
    for graph, dY, want in runs:
        dY.fill_(float("nan"))
        graph.replay()
        torch.cuda.synchronize()
        assert_bit_equal(dY.cpu().numpy(), want, "replayed")


def fill_device(lib, leave, step):
    """Takes device memory until at most `leave` + `step` bytes are free."""
    held = []
    for s in (4 << 30, 256 << 20, step):
        while torch.cuda.mem_get_info()[0] > leave + s:
            p = ctypes.c_void_p()
            lib.spx_malloc(ctypes.byref(p), s)
            held.append(p)
    return held


def waits_for_the_device(f):
    """Whether f() returns only after what is queued on another stream."""
    torch.cuda.synchronize()
    with torch.cuda.stream(torch.cuda.Stream()):
        torch.cuda._sleep(1_000_000_000)                    # 0.5 s and more
        done = torch.cuda.Event()
        done.record()
    f()
    waited = done.query()
    torch.cuda.synchronize()
    return waited


@forced
@pytest.mark.parametrize("act", [sx.ACT_RELU, sx.ACT_SIGMOID, sx.ACT_TANH])
@pytest.mark.parametrize("B,Cin,Cout,H,W", [(32, 9, 37, 7, 8), (20, 7, 66, 5, 11), (8, 12, 32, 6, 20)])
@pytest.mark.parametrize("layout", [sx.LAYOUT_PF, sx.LAYOUT_NCHW, sx.LAYOUT_FMAJOR])
def test_forced_cases_activations(lib, orc, cuda, layout, B, Cin, Cout, H, W, act):
    """Activations in the epilogue, whole and partial tiles, single stores and (NCHW, a width of 4 k) quads: ReLU bit for bit,
    sigmoid and tanh within the library's bound, and all of them the bits of the kernel that computes one result a thread."""
    rng = np.random.default_rng([B, Cout, act])
    wt = sparse(rng, Cout, Cin * 9, 0.3) * np.float32(0.7)
    x = rng.standard_normal((B, Cin, H, W)).astype(np.float32)
    x[0] *= 40                                              # saturated results among them
    bias = rng.standard_normal(Cout).astype(np.float32)
    src = as_layout(x, layout)
    E = orc.encode(wt)
    gd = dict(Cin=Cin, kH=3, kW=3, sH=1, sW=1, pH=1, pW=1, dH=1, dW=1, H=H, W=W)
    want = orc.conv2d(E, gd, layout, src, B, bias, act)
    h = gpu_ell(lib, E)
    g = sx.conv_geom(Cin, Cout, 3, 3, H, W, 1, 1, 1, 1)
    dX, dB = dev(src, cuda), dev(bias, cuda)
    dY, dZ = torch.full(want.shape, float("nan"), device=cuda), torch.full(want.shape, float("nan"), device=cuda)
    assert_ran(kernels_of(lambda: h.conv2d(g, layout, ptr(dX), B, ptr(dB), act, ptr(dY))), "conv_tmem_kernel")
    got = dY.cpu().numpy()
    if act == sx.ACT_RELU:
        assert_bit_equal(got, want, "relu")
    else:
        assert np.abs(got - want).max() <= 4e-7             # expf and tanhf of CUDA and of the C library: a few ulp below 1
    if layout != sx.LAYOUT_FMAJOR:
        lib.spx_conv2d_static(h.h, ctypes.byref(g), layout, ptr(dX), B, ptr(dB), act, ptr(dZ), 0)
        assert_bit_equal(got, dZ.cpu().numpy(), "against one result a thread")


@forced
def test_forced_cases_two_streams(lib, orc, cuda):
    """Two handles on two streams at once, whose CTAs take all of an SM's tensor memory each."""
    rng = np.random.default_rng(4)
    runs = []
    for B, Cin, Cout, H, W in ((32, 20, 64, 28, 28), (16, 33, 96, 30, 21)):
        E = orc.encode(sparse(rng, Cout, Cin * 9, 0.2))
        src = as_layout(rng.standard_normal((B, Cin, H, W)).astype(np.float32), sx.LAYOUT_PF)
        want = orc.conv2d(E, dict(Cin=Cin, kH=3, kW=3, sH=1, sW=1, pH=1, pW=1, dH=1, dW=1, H=H, W=W), sx.LAYOUT_PF, src, B, None, 0)
        runs.append((gpu_ell(lib, E), sx.conv_geom(Cin, Cout, 3, 3, H, W, 1, 1, 1, 1), dev(src, cuda), B, want,
                     [torch.full(want.shape, float("nan"), device=cuda) for _ in range(8)], torch.cuda.Stream()))
    torch.cuda.synchronize()

    def all_calls():
        for i in range(8):
            for h, g, dX, B, _, out, stream in runs:
                h.conv2d(g, sx.LAYOUT_PF, ptr(dX), B, None, 0, ptr(out[i]), stream.cuda_stream)

    assert_ran(kernels_of(all_calls), "conv_tmem_kernel")
    for _, _, _, _, want, out, _ in runs:
        for y in out:
            assert_bit_equal(y.cpu().numpy(), want, "two streams")


@pytest.mark.skipif(os.environ.get("SPX_CONV_TMA_TEST_TIMEOUT") != "1" or os.environ.get("SPX_CONV_TMEM") != "2", reason="runs in a child process")
def test_timeout_of_this_kernel(lib, orc, cuda):
    """The waits for its bulk copies run out: that call returns, the next says so, the one after does without and is right."""
    rng = np.random.default_rng(6)
    B, Cin, Cout, H = 16, 40, 48, 12
    E = orc.encode(sparse(rng, Cout, Cin * 9, 0.25))
    src = as_layout(rng.standard_normal((B, Cin, H, H)).astype(np.float32), sx.LAYOUT_PF)
    want = orc.conv2d(E, dict(Cin=Cin, kH=3, kW=3, sH=1, sW=1, pH=1, pW=1, dH=1, dW=1, H=H, W=H), sx.LAYOUT_PF, src, B, None, 0)
    h, g, dX, dY = gpu_ell(lib, E), sx.conv_geom(Cin, Cout, 3, 3, H, H, 1, 1, 1, 1), dev(src, cuda), torch.full(want.shape, float("nan"), device=cuda)
    call = lambda: h.conv2d(g, sx.LAYOUT_PF, ptr(dX), B, None, 0, ptr(dY))
    assert_ran(kernels_of(call), "conv_tmem_kernel")
    with pytest.raises(sx.SpxError, match="bulk tensor copy"):
        call()
    dY.fill_(float("nan"))
    names = kernels_of(call)
    assert names is None or "conv_tmem_kernel" not in names
    assert_bit_equal(dY.cpu().numpy(), want, "after the reported timeout")


@pytest.mark.skipif(any(k.startswith("SPX_CONV") for k in os.environ), reason="the choice is forced")
@pytest.mark.parametrize("shared,density,kernel", [(False, 0.2, "conv_tmem_kernel"), (True, 0.05, "conv_rbm_tile_kernel"), (True, 0.5, "conv_tmem_kernel")])
def test_choice_follows_the_entries(lib, orc, cuda, shared, density, kernel):
    """The merged kernel does a column once for four rows: where rows share theirs it is the faster one at low density (128 ->
    128, 28 x 28, batch 32, 5 %: 29 us against 41), and has to be taken although the density alone speaks for the other
    (45 and 37)."""
    rng = np.random.default_rng(12)
    C, H, B = 128, 28, 32
    wt = rng.standard_normal((C, C * 9)).astype(np.float32)
    wt[np.broadcast_to(rng.random((1 if shared else C, C * 9)) >= density, wt.shape)] = 0
    E = orc.encode(wt)
    src = as_layout(rng.standard_normal((B, C, H, H)).astype(np.float32), sx.LAYOUT_PF)
    want = orc.conv2d(E, dict(Cin=C, kH=3, kW=3, sH=1, sW=1, pH=1, pW=1, dH=1, dW=1, H=H, W=H), sx.LAYOUT_PF, src, B, None, 0)
    dX, dY = dev(src, cuda), torch.empty(want.shape, device=cuda)
    h = gpu_ell(lib, E)
    g = sx.conv_geom(C, C, 3, 3, H, H, 1, 1, 1, 1)
    for _ in range(2):
        dY.fill_(float("nan"))
        names = kernels_of(lambda: h.conv2d(g, sx.LAYOUT_PF, ptr(dX), B, None, 0, ptr(dY)))
        assert_ran(names, kernel)
        assert_bit_equal(dY.cpu().numpy(), want, kernel)


@forced
def test_no_room_for_a_form(lib, orc, cuda):
    """The form does not fit: the merged kernel takes the call, and the next one does not try again (which would wait for
    the whole device each time)."""
    rng = np.random.default_rng(8)
    Cin, Cout, B, H = 512, 2048, 32, 4
    wt = sparse(rng, Cout, Cin * 9, 0.01)
    wt[0] = 1                                               # a full row: the form's capacity is for rows like it, 77 MB
    E = orc.encode(wt)
    src = as_layout(rng.standard_normal((B, Cin, H, H)).astype(np.float32), sx.LAYOUT_PF)
    want = orc.conv2d(E, dict(Cin=Cin, kH=3, kW=3, sH=1, sW=1, pH=1, pW=1, dH=1, dW=1, H=H, W=H), sx.LAYOUT_PF, src, B, None, 0)
    dX, dY = dev(src, cuda), torch.empty(want.shape, device=cuda)
    g = sx.conv_geom(Cin, Cout, 3, 3, H, H, 1, 1, 1, 1)

    def call(h):
        dY.fill_(float("nan"))
        h.conv2d(g, sx.LAYOUT_PF, ptr(dX), B, None, 0, ptr(dY))

    h = gpu_ell(lib, E)
    h.conv2d(sx.conv_geom(Cin, Cout, 3, 3, H, H, 2, 2, 1, 1), sx.LAYOUT_PF, ptr(dX), B, None, 0, ptr(dY))   # merged weights only
    dY.fill_(0.0)
    assert not waits_for_the_device(lambda: None)           # (makes the stream while there is room)
    held = fill_device(lib, 32 << 20, 16 << 20)
    try:
        for again in (False, True):
            waited = waits_for_the_device(lambda: call(h))
            assert not (again and waited), "a call after the failed one waited for another stream's work"
            assert_bit_equal(dY.cpu().numpy(), want, "short of memory")
    finally:
        for p in held:
            lib.spx_free(p)
    other = gpu_ell(lib, E)
    assert_ran(kernels_of(lambda: call(other)), "conv_tmem_kernel")
    assert_ran(kernels_of(lambda: call(h)), "conv_rbm_tile_kernel")
    assert_bit_equal(dY.cpu().numpy(), want, "room again")


def child(files, select, env):
    cmd = [sys.executable, "-m", "pytest", "-q", "-x", "-m", "gpu", "-p", "no:cacheprovider", *[os.path.join(HERE, f) for f in files], "-k", select]
    r = subprocess.run(cmd, env={**os.environ, **env}, capture_output=True, text=True, timeout=900)
    assert r.returncode == 0 and " passed" in r.stdout, r.stdout[-3000:] + r.stderr[-2000:]


def test_forced_kernel():
    child(["test_conv_tmem_gpu.py", "test_parity_gpu.py", "test_fuzz_gpu.py"],
          "forced_cases or forced_more or conv_bit_exact or conv_views or conv_random or golden_conv", {"SPX_CONV_TMEM": "2"})


def test_timeout_is_reported():
    """The waits for its bulk copies are bounded: they are made to run out, the next call says so, the one after works."""
    child(["test_conv_tmem_gpu.py", "test_parity_gpu.py"], "timeout_of_this_kernel or bulk_copy_timeout_child", {"SPX_CONV_TMEM": "2", "SPX_CONV_TMA_TEST_TIMEOUT": "1"})


def test_forced_without_memory():
    child(["test_conv_tmem_gpu.py"], "no_room_for_a_form", {"SPX_CONV_TMEM": "2"})
