"""The work this library is used for, as cases that can be timed one by one.

Every case is one call (or one forward pass) through the public entry points: the drop-in Python
module `sparseops_backend` on NumPy arrays, and the C ABI (`spx_ctypes`) or the module's `*_device`
calls on CUDA tensors.  A case is a dict of plain values; `kind` names the call:

  matvec   ellpack_matvec on host arrays            spmv   spx_spmv on device arrays
  matmul   ellpack_matmul on host arrays            spmm   spx_spmm on device arrays
  conv     spx_conv2d on device tensors, in the three layouts
  mlp      SparseOnnxModel: `host` -> run() on arrays, otherwise run_device() on tensors
  codec    spx_ell_encode_device of a dense matrix and spx_ell_decode_device back

Values follow the repository's workloads: weights N(0, sigma) kept iid with probability `density`,
operands U(-1, 1) (U(0, 1) into the MLP, N(0, 1) into the convolution), row lengths of the skewed
matrices from a power law with mean 64 and maximum 2048.  All arithmetic is float32.
"""
import math
import os
import sys
import tempfile

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.abspath(os.getcwd()), "sparse-ops_b200"))

import onnx_wire  # noqa: E402
import sparseops_backend as sb  # noqa: E402
import spx_ctypes as sx  # noqa: E402
import workloads  # noqa: E402

_ACTS = (sx.ACT_NONE, sx.ACT_RELU, sx.ACT_SIGMOID, sx.ACT_TANH)
_LAYOUTS = {"chwb": sx.LAYOUT_PF, "nchw": sx.LAYOUT_NCHW, "fmajor": sx.LAYOUT_FMAJOR}
_MEAN, _KMAX = 64.0, 2048        # skewed rows
_lib = None


def _spx():
    global _lib
    if _lib is None:
        _lib = sx.Lib()
    return _lib


def listed():
    return [
        # the smallest call: one pruned layer at batch 1 from NumPy, all latency
        dict(name="matvec_2048_host", kind="matvec", m=2048, n=2048, density=0.1, bias=True),
        # a small layer at a small batch, one of the published shapes (512 x 512, 80 % sparse, 64 columns)
        dict(name="spmm_512", kind="spmm", m=512, n=512, density=0.2, C=64, act=0, bias=True, rows="iid"),
        # a 4096-wide layer at batch 256
        dict(name="spmm_4096", kind="spmm", m=4096, n=4096, density=0.1, C=256, act=0, bias=True, rows="iid"),
        # sizes that are multiples of nothing, the last batch of an epoch: C is odd, no bias
        dict(name="spmm_ragged", kind="spmm", m=3001, n=4999, density=0.06, C=77, act=1, bias=False, rows="iid"),
        # the largest SpMM: a graph-like matrix with power-law rows, wide operand
        dict(name="spmm_skewed", kind="spmm", m=262144, n=65536, density=_MEAN / 65536, C=1024, act=0, bias=True, rows="power"),
        # the same layer as spmm_4096 as the Python API offers it: NumPy in, NumPy out
        dict(name="matmul_4096_host", kind="matmul", m=4096, n=4096, density=0.1, C=256, bias=True),
        # the largest SpMV of the batch-1 sweep that is not dense-ish: 65536 x 65536, 95 % sparse
        dict(name="spmv_65536", kind="spmv", m=65536, n=65536, density=0.05, bias=True),
        # one sample through a sparse MLP whose activations live on the device: serving at batch 1
        dict(name="mlp_1", kind="mlp", width=4096, depth=4, out=1000, density=0.1, batch=1, host=False),
        # the MLP at its benchmark batch through the unchanged Python API
        dict(name="mlp_256_host", kind="mlp", width=4096, depth=4, out=1000, density=0.1, batch=256, host=True),
        # the benchmark convolution: 256 -> 256 channels, 3 x 3, 56 x 56, batch 32, 80 % sparse
        dict(name="conv_256", kind="conv", Cin=256, Cout=256, k=3, stride=1, pad=1, H=56, W=56, B=32, density=0.2,
             layout="chwb", act=1, bias=True),
        # a downsampling layer at a small odd batch, in the layout images come in
        dict(name="conv_nchw_odd", kind="conv", Cin=64, Cout=128, k=3, stride=2, pad=1, H=57, W=57, B=3, density=0.1,
             layout="nchw", act=1, bias=True),
        # encode a pruned weight that lives on the device, and decode it again
        dict(name="codec_8192", kind="codec", m=8192, n=8192, density=0.1),
    ]


def _size(rng, lo, hi):
    """Log-uniform; every other one rounded to a multiple of 32 (never below lo), the rest as they fall."""
    v = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    if rng.random() < 0.5:
        v = max(32, (v + 16) // 32 * 32)
    return max(lo, min(hi, v))


def _density(rng, lo, hi):
    return round(math.exp(rng.uniform(math.log(lo), math.log(hi))), 4)


def draw(rng):
    kind = rng.choice(("spmm", "spmm", "spmm", "spmv", "spmv", "conv", "conv", "mlp", "mlp", "matmul", "matvec", "codec"))
    bias = rng.random() < 0.8
    if kind == "spmm" and rng.random() < 0.25:
        m, n = _size(rng, 16384, 262144), _size(rng, 4096, 65536)
        return dict(kind=kind, m=m, n=n, density=_MEAN / n, C=_size(rng, 32, 1024), act=rng.choice((0, 0, 1)), bias=bias, rows="power")
    if kind == "spmm":
        m, n, d = _size(rng, 256, 8192), _size(rng, 256, 8192), _density(rng, 0.02, 0.5)
        C = min(_size(rng, 1, 1024), max(1, int(6e9 / (m * n * d))))
        return dict(kind=kind, m=m, n=n, density=d, C=C, act=rng.choice((0, 1, 2, 3)), bias=bias, rows="iid")
    if kind == "spmv":
        m, n, d = _size(rng, 1024, 65536), _size(rng, 1024, 65536), _density(rng, 0.01, 0.2)
        return dict(kind=kind, m=m, n=n, density=min(d, round(2e8 / (m * n), 4) if m * n * d > 2e8 else d), bias=bias)
    if kind == "matmul":
        return dict(kind=kind, m=_size(rng, 256, 4096), n=_size(rng, 256, 4096), density=_density(rng, 0.02, 0.3),
                    C=_size(rng, 1, 512), bias=bias)
    if kind == "matvec":
        return dict(kind=kind, m=_size(rng, 256, 8192), n=_size(rng, 256, 8192), density=_density(rng, 0.02, 0.3), bias=bias)
    if kind == "mlp":
        return dict(kind=kind, width=_size(rng, 256, 4096), depth=rng.randint(2, 5), out=rng.choice((10, 100, 1000)),
                    density=_density(rng, 0.05, 0.2), batch=_size(rng, 1, 256), host=rng.random() < 0.5)
    if kind == "codec":
        return dict(kind=kind, m=_size(rng, 256, 8192), n=_size(rng, 256, 8192), density=_density(rng, 0.02, 0.3))
    k = rng.choice((1, 3, 3, 3, 5))
    c = dict(kind=kind, Cin=rng.choice((3, _size(rng, 16, 512), _size(rng, 16, 512))), Cout=_size(rng, 16, 512), k=k,
             stride=rng.choice((1, 1, 2)), pad=k // 2, H=_size(rng, 7, 112), W=0, B=rng.choice((1, rng.randint(1, 32), 32)),
             density=_density(rng, 0.05, 0.5), layout=rng.choice(("chwb", "chwb", "nchw", "fmajor")), act=rng.choice((0, 1)), bias=bias)
    c["W"] = c["H"] if rng.random() < 0.7 else _size(rng, 7, 112)
    while work(c)["flops"] > 2.2e10:        # no more than the listed convolution
        c["B"], c["Cout"] = max(1, c["B"] // 2), max(16, c["Cout"] * 2 // 3)
    return c


# ---- inputs --------------------------------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _uniform(g, *shape, lo=-1.0, hi=1.0):
    return torch.empty(shape, device="cuda").uniform_(lo, hi, generator=g)


def _dense(g, m, n, density, sigma=1.0):
    """Dense m x n matrix with iid kept entries, drawn in row blocks so that the mask stays small."""
    W = torch.empty((m, n), device="cuda")
    step = max(1, (1 << 28) // max(1, n))
    for r in range(0, m, step):
        w = W[r:r + step]
        w.normal_(0.0, sigma, generator=g)
        w.masked_fill_(torch.rand(w.shape, device="cuda", generator=g) >= density, 0.0)
    return W


def _power_csr(g, m, n):
    """Rows of power-law length (workloads.powerlaw_pmf), sorted distinct uniform columns, N(0, 1) values."""
    kmax = min(_KMAX, n)
    cdf = torch.from_numpy(np.cumsum(workloads.powerlaw_pmf(kmax, min(_MEAN, kmax / 2)))).cuda()
    k = torch.searchsorted(cdf, torch.rand(m, device="cuda", dtype=torch.float64, generator=g)).clamp_(max=kmax - 1) + 1
    k[0] = kmax
    rows = torch.repeat_interleave(torch.arange(m, device="cuda"), k)
    key = torch.unique(rows * n + torch.randint(0, n, rows.shape, device="cuda", generator=g))
    rows = torch.div(key, n, rounding_mode="floor")
    rowptr = torch.zeros(m + 1, dtype=torch.int64, device="cuda")
    rowptr[1:] = torch.cumsum(torch.bincount(rows, minlength=m), 0)
    val = torch.empty(key.shape, device="cuda").normal_(generator=g)
    return (rowptr.cpu().numpy().astype(np.uint64), (key - rows * n).to(torch.int32).cpu().numpy().view(np.uint32), val.cpu().numpy())


def prepare(case, seed):
    g, kind, lib = _gen(seed), case["kind"], _spx()
    s = {"case": case, "stream": torch.cuda.current_stream().cuda_stream}
    if kind in ("matvec", "matmul"):
        s["E"] = sb.convert_to_ellpack(_dense(g, case["m"], case["n"], case["density"]).cpu().numpy())
        X = _uniform(g, case["n"]) if kind == "matvec" else _uniform(g, case["n"], case["C"])
        s["X"] = X.cpu().numpy()
        s["bias"] = torch.randn(case["m"], device="cuda", generator=g).cpu().numpy() if case["bias"] else None
    elif kind in ("spmv", "spmm"):
        m, n = case["m"], case["n"]
        if case.get("rows") == "power":
            s["E"] = lib.ell_create_csr(m, n, *_power_csr(g, m, n))
        else:
            W = _dense(g, m, n, case["density"], 1.0 / math.sqrt(max(1.0, case["density"] * n)) if kind == "spmv" else 1.0)
            s["E"] = lib.ell_encode_device(W.data_ptr(), m, n, s["stream"])
            del W
        shape = (n,) if kind == "spmv" else (n, case["C"])
        s["X"] = _uniform(g, *shape)
        s["Y"] = torch.empty((m,) + shape[1:], device="cuda")
        s["bias"] = torch.randn(m, device="cuda", generator=g) if case["bias"] else None
    elif kind == "conv":
        c = case
        geom = sx.conv_geom(c["Cin"], c["Cout"], c["k"], c["k"], c["H"], c["W"], c["stride"], c["stride"], c["pad"], c["pad"])
        K = c["Cin"] * c["k"] * c["k"]
        W = _dense(g, c["Cout"], K, c["density"], math.sqrt(2.0 / K))
        s["E"], s["geom"] = lib.ell_encode_device(W.data_ptr(), c["Cout"], K, s["stream"]), geom
        shape = {"chwb": lambda ch, h, w, b: (ch, h, w, b), "nchw": lambda ch, h, w, b: (b, ch, h, w),
                 "fmajor": lambda ch, h, w, b: (w, h, ch, b)}[c["layout"]]
        s["X"] = torch.randn(shape(c["Cin"], c["H"], c["W"], c["B"]), device="cuda", generator=g)
        s["Y"] = torch.empty(shape(c["Cout"], geom.Ho, geom.Wo, c["B"]), device="cuda")
        s["bias"] = torch.randn(c["Cout"], device="cuda", generator=g) if c["bias"] else None
    elif kind == "mlp":
        dims = [case["width"]] * case["depth"] + [case["out"]]
        ws = [_dense(g, dims[i + 1], dims[i], case["density"], math.sqrt(2.0 / (dims[i] * case["density"]))).cpu().numpy()
              for i in range(case["depth"])]
        bs = [(0.1 * torch.randn(d, device="cuda", generator=g)).cpu().numpy() for d in dims[1:]]
        acts = ["Relu"] * (case["depth"] - 1) + ["Sigmoid"]
        with tempfile.NamedTemporaryFile(suffix=".onnx") as f:
            f.write(onnx_wire.mlp_model(ws, bs, acts, case["batch"]))
            f.flush()
            s["model"] = sb.SparseOnnxModel(f.name)
        s["model"].resize_buffers(case["batch"])
        x = _uniform(g, dims[0], case["batch"], lo=0.0)          # feature-major, batch fastest
        if case["host"]:
            s["X"] = x.cpu().numpy().reshape(case["batch"], dims[0])
        else:
            s["X"], s["Y"] = x, torch.empty((dims[-1], case["batch"]), device="cuda")
    else:
        s["W"] = _dense(g, case["m"], case["n"], case["density"])
        s["Y"] = torch.empty_like(s["W"])
    torch.cuda.synchronize()
    return s


def run(s):
    case, kind = s["case"], s["case"]["kind"]
    if kind == "matvec":
        return sb.ellpack_matvec(s["E"], s["X"], s["bias"])
    if kind == "matmul":
        return sb.ellpack_matmul(s["E"], s["X"], s["bias"])
    if kind == "mlp" and case["host"]:
        return s["model"].run(s["X"])
    if kind == "mlp":
        s["model"].run_device(s["X"].data_ptr(), case["batch"], s["Y"].data_ptr(), s["stream"])
        return s["Y"]
    if kind == "codec":
        lib, e = _spx(), _spx().ell_encode_device(s["W"].data_ptr(), case["m"], case["n"], s["stream"])
        lib.spx_ell_decode_device(e.h, s["Y"].data_ptr(), s["stream"])
        count = e.nnz_total
        e.close()
        return s["Y"], count
    bias = s["bias"].data_ptr() if s["bias"] is not None else None
    if kind == "spmv":
        s["E"].spmv(s["X"].data_ptr(), bias, s["Y"].data_ptr(), s["stream"])
    elif kind == "spmm":
        C = case["C"]
        s["E"].spmm(s["X"].data_ptr(), C, C, bias, _ACTS[case["act"]], s["Y"].data_ptr(), C, s["stream"])
    else:
        s["E"].conv2d(s["geom"], _LAYOUTS[case["layout"]], s["X"].data_ptr(), case["B"], bias, _ACTS[case["act"]],
                      s["Y"].data_ptr(), s["stream"])
    return s["Y"]


def work(case):
    """8 bytes per stored entry (value and column id), the row counts, bias, operands and results once."""
    kind = case["kind"]
    if kind == "mlp":
        dims = [case["width"]] * case["depth"] + [case["out"]]
        nnz = sum(case["density"] * a * b for a, b in zip(dims, dims[1:]))
        return {"bytes": 8 * nnz + 8 * sum(dims[1:]) + 4 * case["batch"] * (dims[0] + dims[-1]), "flops": 2 * nnz * case["batch"]}
    if kind == "conv":
        c = case
        Ho, Wo = ((x + 2 * c["pad"] - c["k"]) // c["stride"] + 1 for x in (c["H"], c["W"]))
        nnz = c["density"] * c["Cout"] * c["Cin"] * c["k"] ** 2
        return {"bytes": 8 * nnz + 8 * c["Cout"] + 4 * c["B"] * (c["Cin"] * c["H"] * c["W"] + c["Cout"] * Ho * Wo),
                "flops": 2 * nnz * Ho * Wo * c["B"]}
    m, n = case["m"], case["n"]
    nnz = case["density"] * m * n
    if kind == "codec":
        return {"bytes": 8 * m * n + 16 * nnz + 8 * m, "flops": 0}
    C = case.get("C", 1)
    return {"bytes": 8 * nnz + 4 * m * (2 if case["bias"] else 1) + 4 * C * (n + m), "flops": 2 * nnz * C}


def tolerance(case):
    """float32 sums of at most a few thousand terms, in any order; the codec moves values unchanged."""
    return "exact" if case["kind"] == "codec" else {"rel": 1e-5}
