"""Workloads whose speed this repository tracks.

Each case is one call (or one replayed batch) of the public Python binding on
device-resident operands: dot, mtv / vtm, mtm in its precision choices, the
grouped batch and the transpose, over the sizes the library is used at - from
a 4096-element dot, which is all launch latency, to an 8192^3 matrix product.

  listed()              the fixed cases
  draw(rng)             one more case of the same ranges
  prepare(case, seed)   operands (and a batch's handle) on the GPU
  run(state)            one call; returns its outputs
  work(case)            bytes and flops the call cannot do without
  exact(case, seed)     the outputs in 64-bit arithmetic by plain torch
"""
import math
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "openmp-blas_gb300"))
import gbblas  # noqa: E402

ROW, COL = gbblas.LAST_ORDER, gbblas.FIRST_ORDER
ACCURACY = {
    "fp32": gbblas.ACCURACY_FP32,
    "auto": gbblas.ACCURACY_AUTO,
    "fp16x3": gbblas.ACCURACY_FP16X3,
    "bf16x3": gbblas.ACCURACY_BF16X3,
    "bf16x6": gbblas.ACCURACY_BF16X6,
    "fp8": gbblas.ACCURACY_FP8,
    "default": gbblas.ACCURACY_FP32,  # double: gbblas_dgemm, the drop-in mtm<double>
}
DTYPE = {"f32": torch.float32, "f64": torch.float64}


def listed():
    return [
        # a short inner product inside an iterative method: launch latency
        {"name": "dot_f32_4096", "kind": "dot", "dtype": "f32", "n": 4096},
        # the double half of the bandwidth configuration's dots
        {"name": "dot_f64_2e28", "kind": "dot", "dtype": "f64", "n": 1 << 28},
        # the bandwidth configuration's matrix-vector product
        {"name": "mtv_f32_row_16384", "kind": "mv", "op": "mtv", "dtype": "f32", "layout": "row", "M": 16384, "N": 16384},
        # double, column-major (uBLAS's default layout), odd extents: y += A x
        {"name": "mtv_f64_col_ragged", "kind": "mv", "op": "mtv", "dtype": "f64", "layout": "col", "M": 8191, "N": 6001},
        # a small product of the reference's size sweep: latency and launch geometry
        {"name": "mtm_f32_small", "kind": "mtm", "dtype": "f32", "acc": "fp32", "M": 211, "N": 190, "K": 173, "la": "row",
         "lb": "row", "lc": "row", "values": "uniform"},
        # the plain single-precision configuration on the FMA pipe
        {"name": "mtm_f32_1024", "kind": "mtm", "dtype": "f32", "acc": "fp32", "M": 1024, "N": 1024, "K": 1024,
         "la": "row", "lb": "row", "lc": "row", "values": "uniform"},
        # the precision configuration, FP32-accurate on the tensor cores
        {"name": "mtm_auto_8192", "kind": "mtm", "dtype": "f32", "acc": "auto", "M": 8192, "N": 8192, "K": 8192,
         "la": "row", "lb": "row", "lc": "row", "values": "uniform"},
        # a served request's size: dimensions as they come, multiples of nothing
        {"name": "mtm_auto_ragged", "kind": "mtm", "dtype": "f32", "acc": "auto", "M": 3970, "N": 3475, "K": 4050,
         "la": "row", "lb": "row", "lc": "row", "values": "uniform"},
        # the precision configuration's low-accuracy path on its wide-range inputs
        {"name": "mtm_fp8_8192", "kind": "mtm", "dtype": "f32", "acc": "fp8", "M": 8192, "N": 8192, "K": 8192,
         "la": "row", "lb": "row", "lc": "row", "values": "wide"},
        # a served double-precision request, column-major as uBLAS lays it out
        {"name": "mtm_f64_ragged", "kind": "mtm", "dtype": "f64", "acc": "default", "M": 1531, "N": 1400, "K": 1601,
         "la": "col", "lb": "col", "lc": "col", "values": "uniform"},
        # the batching configuration's 512 products beside matrix-vector
        # products of its range, one replayed graph
        {"name": "batch_512", "kind": "batch", "acc": "bf16x3", "gemms": 512, "gemvs": 32, "shapes": 3},
        # a transpose between row-major matrices whose rows are not 16-byte aligned
        {"name": "transpose_f32_ragged", "kind": "transpose", "dtype": "f32", "M": 9001, "N": 7003, "la": "row", "lc": "row"},
    ]


def _size(rng, lo, hi):
    """A size of [lo, hi], even over its logarithm; odd ones, multiples of 8
    and powers of two all occur."""
    v = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    how = rng.random()
    if how < 0.3:
        v = max(8, v // 8 * 8)
    elif how < 0.4:
        v = 1 << max(0, round(math.log2(v)))
    return min(hi, max(lo, v))


def draw(rng):
    kind = rng.choice(["dot", "mv", "mv", "mtm", "mtm", "mtm", "mtm", "batch", "transpose"])
    dtype = "f64" if rng.random() < 0.3 else "f32"
    layout = lambda: rng.choice(["row", "col"])  # noqa: E731
    if kind == "dot":
        return {"kind": kind, "dtype": dtype, "n": _size(rng, 1024, 1 << 28)}
    if kind == "mv":
        while True:
            c = {"kind": kind, "op": rng.choice(["mtv", "vtm"]), "dtype": dtype, "layout": layout(),
                 "M": _size(rng, 64, 32768), "N": _size(rng, 64, 32768)}
            if c["M"] * c["N"] <= 1 << 28:
                return c
    if kind == "transpose":
        return {"kind": kind, "dtype": dtype, "M": _size(rng, 64, 16384), "N": _size(rng, 64, 16384), "la": layout(),
                "lc": layout()}
    if kind == "batch":
        return {"kind": kind, "acc": rng.choice(["bf16x3", "bf16x6"]), "gemms": _size(rng, 16, 512),
                "gemvs": _size(rng, 8, 32), "shapes": rng.randrange(1, 1 << 20)}
    acc = "default" if dtype == "f64" else rng.choice(["fp32", "fp32", "auto", "auto", "auto", "fp16x3", "bf16x3", "bf16x6", "fp8"])
    # no dearer than the dearest listed case: the FMA pipe and the double
    # path run tens of TFLOP/s, the tensor-core splits hundreds
    most = {"default": 6e10, "fp32": 1e11, "bf16x6": 5e11}.get(acc, 1.1e12)
    while True:
        c = {"kind": kind, "dtype": dtype, "acc": acc, "M": _size(rng, 32, 8192), "N": _size(rng, 32, 8192),
             "K": _size(rng, 32, 8192), "la": layout(), "lb": layout(), "lc": layout(),
             "values": "wide" if rng.random() < 0.25 else "uniform"}
        if 2.0 * c["M"] * c["N"] * c["K"] <= most:
            return c


# ------------------------------------------------------------------ operands

def _values(gen, n, dtype, values="uniform"):
    """n values: uniform [-1, 1), or wide: random sign, mantissa in [1, 2),
    exponent uniform in [-10, 10]."""
    u = torch.rand(n, generator=gen, device="cuda", dtype=DTYPE[dtype]) * 2 - 1
    if values == "wide":
        e = torch.randint(-10, 11, (n,), generator=gen, device="cuda")
        u = torch.ldexp(torch.where(u < 0, u - 1, u + 1), e)
    return u


def _matrix(gen, rows, cols, dtype, layout, values="uniform"):
    """A dense rows x cols matrix in `layout`, as a strided view."""
    flat = _values(gen, rows * cols, dtype, values)
    return flat.view(rows, cols) if layout == "row" else flat.view(cols, rows).t()


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _batch_shapes(case):
    """GEMM dimensions log-uniform in [32, 2048] (multiples of 8), GEMV
    dimensions log-uniform in [256, 16384]."""
    r = random.Random(case["shapes"])
    logu = lambda lo, hi: int(round(math.exp(r.uniform(math.log(lo), math.log(hi)))))  # noqa: E731
    mm = [tuple(max(32, logu(32, 2048) // 8 * 8) for _ in range(3)) for _ in range(case["gemms"])]
    mv = [(logu(256, 16384), logu(256, 16384)) for _ in range(case["gemvs"])]
    return mm, mv


def _batch_operands(case, seed):
    mm, mv = _batch_shapes(case)
    gen = _gen(seed)
    at = lambda sizes: np.concatenate([[0], np.cumsum(sizes)]).tolist()  # noqa: E731
    # every operand starts on a 16-byte boundary
    pad = lambda n: (n + 3) // 4 * 4  # noqa: E731
    oa, ob, oc = (at([pad(f(s)) for s in mm]) for f in (lambda s: s[0] * s[2], lambda s: s[2] * s[1], lambda s: s[0] * s[1]))
    ov, ox, oy = (at([pad(f(s)) for s in mv]) for f in (lambda s: s[0] * s[1], lambda s: s[1], lambda s: s[0]))
    A, B, C, V, X = (_values(gen, n, "f32") for n in (oa[-1], ob[-1], oc[-1], ov[-1], ox[-1]))
    Y = torch.zeros(oy[-1], device="cuda")
    part = lambda flat, o, i, shape: flat[o[i]:o[i] + math.prod(shape)].view(shape)  # noqa: E731
    gemms = [(part(A, oa, i, (m, k)), part(B, ob, i, (k, n)), part(C, oc, i, (m, n))) for i, (m, n, k) in enumerate(mm)]
    gemvs = [(part(V, ov, i, (m, n)), part(X, ox, i, (n,)), part(Y, oy, i, (m,))) for i, (m, n) in enumerate(mv)]
    return gemms, gemvs, C, Y


def _operands(case, seed):
    kind, gen = case["kind"], _gen(seed)
    if kind == "dot":
        return _values(gen, case["n"], case["dtype"]), _values(gen, case["n"], case["dtype"])
    if kind == "mv":
        M, N = case["M"], case["N"]
        A = _matrix(gen, M, N, case["dtype"], case["layout"])
        n_in, n_out = (N, M) if case["op"] == "mtv" else (M, N)
        return A, _values(gen, n_in, case["dtype"]), _values(gen, n_out, case["dtype"])
    if kind == "transpose":
        A = _matrix(gen, case["M"], case["N"], case["dtype"], case["la"])
        flat = torch.zeros(case["M"] * case["N"], device="cuda", dtype=DTYPE[case["dtype"]])
        T = flat.view(case["N"], case["M"]) if case["lc"] == "row" else flat.view(case["M"], case["N"]).t()
        return A, T
    M, N, K, d, v = case["M"], case["N"], case["K"], case["dtype"], case["values"]
    return (_matrix(gen, M, K, d, case["la"], v), _matrix(gen, K, N, d, case["lb"], v), _matrix(gen, M, N, d, case["lc"]))


# ---------------------------------------------------------------- the calls

def prepare(case, seed):
    state = dict(case)
    if case["kind"] == "batch":
        gemms, gemvs, C, Y = _batch_operands(case, seed)
        # a program that replays a batch keeps its handle, like its operands
        state["batch"] = gbblas.Batch([gbblas.gemm_desc(*g) for g in gemms],
                                      [gbblas.gemv_desc(ROW, False, a.shape[0], a.shape[1], a, x, y) for a, x, y in gemvs],
                                      accuracy=ACCURACY[case["acc"]])
        state["held"], state["C"], state["Y"] = (gemms, gemvs), C, Y
        return state
    state["ops"] = _operands(case, seed)
    if case["kind"] == "dot":
        state["out"] = torch.zeros(1, device="cuda", dtype=DTYPE[case["dtype"]])
    return state


def run(s):
    kind = s["kind"]
    if kind == "dot":
        a, b = s["ops"]
        return gbblas.dot(a, b, s["out"])
    if kind == "mv":
        A, x, y = s["ops"]
        call = gbblas.mtv if s["op"] == "mtv" else gbblas.vtm
        return call(ROW if s["layout"] == "row" else COL, s["M"], s["N"], A, x, y)
    if kind == "mtm":
        A, B, C = s["ops"]
        return gbblas.gemm(A, B, C, accuracy=ACCURACY[s["acc"]])
    if kind == "transpose":
        A, T = s["ops"]
        gbblas.call("gbblas_stranspose" if s["dtype"] == "f32" else "gbblas_dtranspose", s["M"], s["N"], A.data_ptr(),
                    A.stride(0), A.stride(1), T.data_ptr(), T.stride(0), T.stride(1), None)
        return T
    s["batch"].run()
    return s["C"], s["Y"]


def work(case):
    kind = case["kind"]
    size = 8 if case.get("dtype") == "f64" else 4
    if kind == "dot":
        return {"bytes": 2 * case["n"] * size, "flops": 2 * case["n"]}
    if kind == "mv":
        M, N = case["M"], case["N"]
        return {"bytes": (M * N + M + N) * size, "flops": 2 * M * N}
    if kind == "transpose":
        return {"bytes": 2 * case["M"] * case["N"] * size, "flops": 0}
    if kind == "mtm":
        M, N, K = case["M"], case["N"], case["K"]
        return {"bytes": (M * K + K * N + 2 * M * N) * size, "flops": 2 * M * N * K}
    mm, mv = _batch_shapes(case)
    return {"bytes": 4 * (sum(m * k + k * n + 2 * m * n for m, n, k in mm) + sum(m * n + m + n for m, n in mv)),
            "flops": 2 * (sum(m * n * k for m, n, k in mm) + sum(m * n for m, n in mv))}


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        gemms, gemvs, C, Y = _batch_operands(case, seed)
        C64, Y64 = C.double(), Y.double()
        for a, b, c in gemms:
            o = c.storage_offset()
            C64[o:o + c.numel()] += (a.double() @ b.double()).reshape(-1)
        for a, x, y in gemvs:
            o = y.storage_offset()
            Y64[o:o + y.numel()] = a.double() @ x.double()
        return C64, Y64
    ops = [t.double() for t in _operands(case, seed)]
    if kind == "dot":
        return torch.dot(*ops).reshape(1)
    if kind == "mv":
        A, x, y = ops
        r = A @ x if case["op"] == "mtv" else A.t() @ x
        # column-major operands accumulate into y, row-major ones overwrite
        # it; a vector times a matrix is the product with the transpose
        accumulates = (case["layout"] == "col") == (case["op"] == "mtv")
        return y + r if accumulates else r
    if kind == "transpose":
        return ops[0].t()
    A, B, C = ops
    return C + A @ B
