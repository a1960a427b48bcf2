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
from test_conv_tmem_gpu import kernels_of

pytestmark = pytest.mark.gpu


def sparse(rng, m, n, p):
    W = rng.standard_normal((m, n)).astype(np.float32)
    W[rng.random((m, n)) >= p] = 0
    return W


def in_child(name, **env):
    """Runs the test `name` of this file in a process of its own: switches are read once per process."""
    cmd = [sys.executable, "-m", "pytest", "-q", "-x", "-m", "gpu", "-p", "no:cacheprovider", os.path.abspath(__file__) + "::" + name]
    r = subprocess.run(cmd, env={**os.environ, **env}, capture_output=True, text=True, timeout=300)
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
    in_child("test_stage_refills", SPX_SPMM_TILE="2")


def check_slices(lib, orc, cuda, m, n, C, p, kernel):
    rng = np.random.default_rng([m, C])
    E = orc.encode(sparse(rng, m, n, p))
    b = rng.standard_normal(m).astype(np.float32)
    X = rng.uniform(-1, 1, (n, C)).astype(np.float32)
    want = orc.spmm(E, X, b, act=1)
    h = lib.ell_create(E.Wd, E.idx, E.nnz, E.n)
    dX, dB = torch.from_numpy(X).to(cuda), torch.from_numpy(b).to(cuda)
    dY = torch.full((m, C), float("nan"), device=cuda)
    call = lambda: h.spmm(dX.data_ptr(), C, C, dB.data_ptr(), sx.ACT_RELU, dY.data_ptr(), C)
    for k in range(3):                      # the first one gathers
        dY.fill_(float("nan"))
        names = kernels_of(call)
        assert names is None or (kernel in names) == (k > 0), names
        assert_bit_equal(dY.cpu().numpy(), want, f"call {k}")


slices = pytest.mark.skipif(os.environ.get("SPX_SPMM_SLICES") not in ("32", "64"), reason="runs in a child process of test_slices_forced")


@slices
@pytest.mark.parametrize("C", [9, 32, 33, 63, 64, 65, 95, 96, 97, 128, 130, 352])
@pytest.mark.parametrize("m", [5, 300, 1300])
def test_slices(lib, orc, cuda, m, C):
    """Slices of 32 and of 64 columns, whole, cut short and with a single column, of aligned rows and of a copy.  (X is larger than
    shared memory: the kernels that hold it whole do not take these.)"""
    nv = int(os.environ["SPX_SPMM_SLICES"]) // 32
    n = 1900 if C > 30 else 6500
    check_slices(lib, orc, cuda, m, n, C, 0.2 if n < 2000 else 0.06, f"spmm_tile_kernel<{nv}, ")


@slices
@pytest.mark.parametrize("width,m,C,kernel", [
    (32, 1300, 130, "<1, 20>"), (32, 2604, 130, "<1, 24>"), (32, 3197, 130, "<1, 28>"), (32, 3196, 131, "<1, 28>"),
    (64, 1300, 130, "<2, 16>"), (64, 4200, 130, "<2, 28>"), (64, 4201, 131, "<2, 28>")])
def test_slices_of_each_kernel(lib, orc, cuda, width, m, C, kernel):
    """Several slices, the last one of two and three columns, in the kernels for few and for many warps."""
    if os.environ["SPX_SPMM_SLICES"] != str(width):
        pytest.skip("in the other child")
    check_slices(lib, orc, cuda, m, 1900, C, 0.1, "spmm_tile_kernel" + kernel)


@pytest.mark.parametrize("width", [32, 64])
def test_slices_forced(width):
    in_child("test_slices", SPX_SPMM_TILE="2", SPX_SPMM_SLICES=str(width))
    in_child("test_slices_of_each_kernel", SPX_SPMM_TILE="2", SPX_SPMM_SLICES=str(width))


@pytest.mark.skipif(any(k.startswith("SPX_SPMM") for k in os.environ), reason="the choice is forced")
@pytest.mark.parametrize("m,n,C,p", [(1344, 2176, 240, 0.0426), (644, 1051, 452, 0.0919)])
def test_choice_with_little_more_than_a_cta_per_sm(lib, orc, cuda, m, n, C, p):
    """Gathering takes as long as the SMs with two CTAs: 12.2 and 11.8 us, where X staged takes 8.9 and 7.8."""
    check_slices(lib, orc, cuda, m, n, C, p, "spmm_tile_kernel")


# ---- a bounded wait that runs out -----------------------------------------------------------------
def small_case(orc, seed=5):
    rng = np.random.default_rng(seed)
    m, n, C = 300, 1500, 64
    W = sparse(rng, m, n, 0.1)
    X = rng.uniform(-1, 1, (n, C)).astype(np.float32)
    b = rng.standard_normal(m).astype(np.float32)
    E = orc.encode(W)
    return m, n, C, W, X, b, E, orc.spmm(E, X, b, act=1)


def test_timeout_of_a_call(lib, orc, cuda):
    if os.environ.get("SPX_SPMM_TMA_TEST_TIMEOUT") != "1":
        pytest.skip("runs in a child process of test_timeouts_are_reported")
    m, n, C, W, X, b, E, want = small_case(orc)
    h = lib.ell_create(E.Wd, E.idx, E.nnz, E.n)
    dX, dB, dY = torch.from_numpy(X).to(cuda), torch.from_numpy(b).to(cuda), torch.zeros((m, C), device=cuda)
    run = lambda: h.spmm(dX.data_ptr(), C, C, dB.data_ptr(), sx.ACT_RELU, dY.data_ptr(), C)
    run()                                   # gathered
    run()                                   # enqueued fine; on the GPU a wait gives up after a second
    torch.cuda.synchronize()                # the context is still usable
    y1 = torch.zeros(m, device=cuda)
    with pytest.raises(sx.SpxError, match="bulk tensor copy") as err:       # any width reports it, whichever kernel it would take
        h.spmm(dX.data_ptr(), 1, C, dB.data_ptr(), 0, y1.data_ptr(), 1)
    assert err.value.status == 2
    for k in range(3):                      # no bulk copies from here on
        dY.fill_(float("nan"))
        run()
        torch.cuda.synchronize()
        assert_bit_equal(dY.cpu().numpy(), want, "after the report")
    lib.spx_ell_status(h.h)


def test_timeout_of_a_host_call(lib, orc, cuda):
    if os.environ.get("SPX_SPMM_TMA_TEST_TIMEOUT") != "1":
        pytest.skip("runs in a child process of test_timeouts_are_reported")
    m, n, C, W, X, b, E, want = small_case(orc)
    h = lib.ell_create(E.Wd, E.idx, E.nnz, E.n)
    assert_bit_equal(h.spmm_host(X, b, sx.ACT_RELU), want, "gathered")
    with pytest.raises(sx.SpxError, match="bulk tensor copy"):
        h.spmm_host(X, b, sx.ACT_RELU)
    assert_bit_equal(h.spmm_host(X, b, sx.ACT_RELU), want, "after the report")


@pytest.mark.parametrize("how", ["run", "resident"])
def test_timeout_of_a_replay(lib, orc, backend, cuda, tmp_path, how):
    """The graph's kernel waits in vain: run() fails instead of handing over a stale output, run_resident() fails on its
    next call; both work after that."""
    if os.environ.get("SPX_SPMM_TMA_TEST_TIMEOUT") != "2":
        pytest.skip("runs in a child process of test_timeouts_are_reported")
    import onnx_wire
    m, n, C, W, X, b, E, want = small_case(orc)
    path = tmp_path / "one.onnx"
    path.write_bytes(onnx_wire.mlp_model([W], [b], ["Relu"], C))
    model = backend.SparseOnnxModel(str(path))
    model.resize_buffers(C)                 # first launch: the warm-up pass; second: the captured one, which fails
    out = None
    if how == "run":
        with pytest.raises(RuntimeError, match="bulk tensor copy"):
            model.run(X.reshape(C, n))
        for k in range(2):
            out = np.asarray(model.run(X.reshape(C, n)))
            assert_bit_equal(out.reshape(m, C), want, "after the report")
        return
    dX, dY = torch.from_numpy(X).to(cuda), torch.full((m, C), 7.0, device=cuda)
    lib.spx_memcpy_d2d(model.device_input_ptr(), dX.data_ptr(), dX.numel() * 4, 0)
    torch.cuda.synchronize()
    model.run_resident(0)
    torch.cuda.synchronize()
    with pytest.raises(RuntimeError, match="bulk tensor copy"):
        model.run_resident(0)
    model.run_resident(0)
    torch.cuda.synchronize()
    lib.spx_memcpy_d2d(dY.data_ptr(), model.device_output_ptr(), dY.numel() * 4, 0)
    torch.cuda.synchronize()
    assert_bit_equal(dY.cpu().numpy(), want, "after the report")


@pytest.mark.parametrize("name,launch", [("test_timeout_of_a_call", "1"), ("test_timeout_of_a_host_call", "1"),
                                         ("test_timeout_of_a_replay[run]", "2"), ("test_timeout_of_a_replay[resident]", "2")])
def test_timeouts_are_reported(name, launch):
    """With the switch a barrier expects more bytes than its copy brings, so the kernel's bounded wait runs out (nothing
    faults, nothing hangs): an error, never a stale result."""
    in_child(name, SPX_SPMM_TILE="2", SPX_SPMM_TMA_TEST_TIMEOUT=launch)


def test_large_unaligned_operand_is_only_enqueued(lib, cuda):
    """The copy of an X whose rows are no multiple of 16 bytes is scratch of the call, 165 MB here: the call returns
    while the product runs."""
    m, n, C = 8192, 8192, 5033
    g = torch.Generator(device="cuda").manual_seed(7)
    W = torch.rand((m, n), device=cuda, generator=g)
    W[torch.rand((m, n), device=cuda, generator=g) >= 0.1] = 0
    X, Y = torch.rand((n, C), device=cuda, generator=g), torch.zeros((m, C), device=cuda)
    h = lib.ell_encode_device(W.data_ptr(), m, n)
    run = lambda: h.spmm(X.data_ptr(), C, C, 0, 0, Y.data_ptr(), C)
    for k in range(3):
        run()
    torch.cuda.synchronize()
    before = lib.spx_launch_count()
    run()
    ended = torch.cuda.Event()
    ended.record()
    still_running = not ended.query()
    assert lib.spx_launch_count() == before + 2, "not the route with a copy of X"
    assert still_running
    torch.cuda.synchronize()
    cols = [0, 1, 2517, C - 1]
    want = W.double() @ X[:, cols].double()
    got = Y[:, cols].double()
    assert float((got - want).norm() / want.norm()) < 1e-5      # 32-bit sums of about 800 terms


def test_one_call_in_parts_builds_nothing(lib, orc, cuda):
    """A matrix gets its block form when it is multiplied again.  A host call in column panels and a 1 x 1 convolution
    of several images are one call: the second one builds (two more kernels), the first and third do not."""
    rng = np.random.default_rng(11)
    m, n, C = 2048, 2048, 256
    E = orc.encode(sparse(rng, m, n, 0.2))
    X = rng.uniform(-1, 1, (n, C)).astype(np.float32)
    h = lib.ell_create(E.Wd, E.idx, E.nnz, E.n)
    counts = []
    for k in range(3):
        before = lib.spx_launch_count()
        h.spmm_host(X, None)
        counts.append(lib.spx_launch_count() - before)
    assert counts == [2, 4, 2]
    g = sx.conv_geom(n, m, 1, 1, 16, 16)
    h = lib.ell_create(E.Wd, E.idx, E.nnz, E.n)
    dX, dY = torch.rand((3, n, 256), device=cuda), torch.zeros((3, m, 256), device=cuda)
    counts = []
    for k in range(3):
        before = lib.spx_launch_count()
        h.conv2d(g, sx.LAYOUT_NCHW, dX.data_ptr(), 3, 0, 0, dY.data_ptr())
        counts.append(lib.spx_launch_count() - before)
    torch.cuda.synchronize()
    assert counts == [3, 5, 3]


@pytest.mark.gpu
@pytest.mark.parametrize("m,C", [
    # CTAs of 1, 20, 21, 24 and 25 warps for slices of 32 columns (9, 23: X moves into rows of 32 floats), and of 16 and 17
    # for slices of 64: where the kernels with two steps' operands in registers begin and end
    (4, 32), (7, 9), (11840, 32), (12000, 23), (14208, 32), (14400, 32), (9472, 64), (9600, 61), (592, 256), (600, 274)])
def test_phases(lib, orc, cuda, m, C):
    """Blocks of 256 columns that some rows do not use and others are full of: phases of no step, of one, of a few that
    begin or end inside a block of four, and of many."""
    if os.environ.get("SPX_SPMM_TILE") != "2":
        pytest.skip("runs in a child process of test_phases_forced")
    rng = np.random.default_rng([m, C])
    n = 1800
    share = rng.choice([0.0, 0.004, 0.02, 0.06, 0.3], (m, 8), p=[0.3, 0.2, 0.2, 0.2, 0.1]).astype(np.float32)
    W = rng.standard_normal((m, n), dtype=np.float32)
    W[rng.random((m, n), dtype=np.float32) >= np.repeat(share, 256, axis=1)[:, :n]] = 0
    W[m // 2] = 0
    E = orc.encode(W)
    X = (np.arange(n, dtype=np.float32)[:, None] + rng.uniform(-1, 1, (n, C))).astype(np.float32)
    rows = np.unique(np.concatenate([np.arange(0, m, max(1, m // 200)), [m // 2, m - 1], np.argsort(E.nnz)[-8:]]))
    from oracle import EllArrays
    want = orc.spmm(EllArrays(len(rows), n, E.r, E.Wd[rows], E.idx[rows], E.nnz[rows]), X, None)
    h = lib.ell_create(E.Wd, E.idx, E.nnz, E.n)
    dX = torch.from_numpy(X).to(cuda)
    first = None
    for call in range(6):
        dY = torch.full((m, C), float("nan"), device=cuda)
        h.spmm(dX.data_ptr(), C, C, 0, sx.ACT_NONE, dY.data_ptr(), C)
        torch.cuda.synchronize()
        if first is None:
            first = dY
            assert_bit_equal(dY[torch.from_numpy(rows).to(cuda)].cpu().numpy(), want, "sampled rows")
        assert torch.equal(dY.view(torch.int32), first.view(torch.int32)), f"call {call} differs from the first (gathered) one"


@pytest.mark.gpu
def test_phases_forced():
    in_child("test_phases", SPX_SPMM_TILE="2")
