"""Performance cases of the skinny SGEMM/SGEMV path and its k-means consumer.

Each case is one call (or one launch of a plan) that a program using this
library makes, through the package's public entry points: SGEMM and SGEMV on
CUDA tensors, the reference's host-array ``hmlSgemm``, a batch of uneven
SGEMMs behind a plan, and the k-means assignment step.  Operands are dense, as
programs allocate them, so an odd size means rows that are not 16-byte
aligned.  FP32 is the only data type of the path.

kinds
  gemm      C = A @ B on CUDA tensors; a / b: "row" or "col" major storage
            ("col" of a row-major program is a transposed view); C is
            column-major, the library's default
  host      hmlSgemm on numpy arrays (row-major, C updated in place)
  gemv      y = A x
  residual  r = b - A x  (alpha = -1, beta = 1 on a copy of b)
  batch     one graph launch of a plan of many uneven SGEMMs
  kmeans    nearest-centroid index of every point
"""
import random

import numpy as np
import torch

import hiperml_b200 as hml


def listed():
    return [
        # one small product, as a program's inner step makes thousands of:
        # launch latency and host overhead
        {"name": "gemm_small_512x16x256", "kind": "gemm", "m": 512, "n": 16, "k": 256,
         "a": "row", "b": "row"},
        # the reference's plain skinny SGEMM, column-major
        {"name": "gemm_4096x16x4096", "kind": "gemm", "m": 4096, "n": 16, "k": 4096,
         "a": "col", "b": "col"},
        # two widths of the precision sweep, tall A read once
        {"name": "gemm_65536x32x4096", "kind": "gemm", "m": 65536, "n": 32, "k": 4096,
         "a": "col", "b": "col"},
        {"name": "gemm_65536x128x4096_row", "kind": "gemm", "m": 65536, "n": 128, "k": 4096,
         "a": "row", "b": "row"},
        # a data matrix of odd sizes times a narrow factor, row-major and dense
        {"name": "gemm_ragged_20011x45x1501", "kind": "gemm", "m": 20011, "n": 45, "k": 1501,
         "a": "row", "b": "row"},
        # the square product of the sweep
        {"name": "gemm_8192x8192x8192", "kind": "gemm", "m": 8192, "n": 8192, "k": 8192,
         "a": "col", "b": "col"},
        # the reference's own interface: host arrays in, host array out
        {"name": "host_16384x32x1024", "kind": "host", "m": 16384, "n": 32, "k": 1024},
        # the reference's SGEMV, column-major
        {"name": "gemv_32768x4096", "kind": "gemv", "m": 32768, "n": 4096, "a": "col"},
        # the residual of an overdetermined system of odd sizes, row-major
        {"name": "residual_10007x3001", "kind": "residual", "m": 10007, "n": 3001, "a": "row"},
        # many uneven problems behind one plan, transposes at random
        {"name": "batch_60", "kind": "batch", "count": 60, "sizes_seed": 3, "max_m": 16384,
         "max_n": 128, "max_k": 4096},
        # one k-means iteration's assignment: a million short points
        {"name": "kmeans_1048576x32x64", "kind": "kmeans", "points": 1048576, "dims": 32,
         "clusters": 64},
        # the same on wider points, odd sizes
        {"name": "kmeans_300007x100x50", "kind": "kmeans", "points": 300007, "dims": 100,
         "clusters": 50},
    ]


def _log_int(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def _size(rng, lo, hi):
    """Log-uniform; half of them rounded to a multiple of 16 (where that
    stays in range), the others left as they fall, odd ones among them."""
    v = _log_int(rng, lo, hi)
    return max(16, v // 16 * 16) if v >= 16 and rng.random() < 0.5 else v


def draw(rng):
    kind = rng.choice(["gemm", "gemm", "gemm", "gemv", "residual", "batch", "kmeans", "kmeans",
                       "host"])
    side = lambda: rng.choice(["row", "col"])
    if kind == "gemm":
        return {"kind": kind, "m": _size(rng, 512, 65536), "n": _size(rng, 2, 128),
                "k": _size(rng, 64, 4096), "a": side(), "b": side()}
    if kind == "host":
        return {"kind": kind, "m": _size(rng, 512, 16384), "n": _size(rng, 2, 128),
                "k": _size(rng, 64, 1024)}
    if kind in ("gemv", "residual"):
        return {"kind": kind, "m": _size(rng, 256, 65536), "n": _size(rng, 64, 4096), "a": side()}
    if kind == "batch":
        return {"kind": kind, "count": _log_int(rng, 8, 60), "sizes_seed": rng.randrange(1000),
                "max_m": 16384, "max_n": 128, "max_k": 4096}
    return {"kind": kind, "points": _log_int(rng, 20000, 1000000), "dims": _size(rng, 2, 256),
            "clusters": _size(rng, 2, 256)}


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _uniform(g, *shape):
    return torch.empty(*shape, device="cuda").uniform_(-1.0, 1.0, generator=g)


def _matrix(g, rows, cols, layout):
    return _uniform(g, rows, cols) if layout == "row" else _uniform(g, cols, rows).t()


def _batch_sizes(case):
    """(transA, transB, M, N, K) of every problem of a batch."""
    r = random.Random(case["sizes_seed"])
    return [(r.randrange(2), r.randrange(2), _log_int(r, 256, case["max_m"]),
             r.randint(1, case["max_n"]), _log_int(r, 64, case["max_k"]))
            for _ in range(case["count"])]


def _padded(g, rows, cols):
    """Column-major rows x cols, leading dimension rounded up to 16 bytes."""
    ld = (rows + 3) // 4 * 4
    return torch.randn(cols, ld, device="cuda", generator=g), ld


def _batch_operands(case, seed):
    g = _generator(seed)
    out = []
    for ta, tb, m, n, k in _batch_sizes(case):
        a, lda = _padded(g, k if ta else m, m if ta else k)
        b, ldb = _padded(g, n if tb else k, k if tb else n)
        out.append((ta, tb, m, n, k, a, lda, b, ldb))
    return out


def _host_operands(case, seed):
    r = np.random.default_rng(seed)
    m, n, k = case["m"], case["n"], case["k"]
    a = r.random((m, k), dtype=np.float32) * np.float32(2) - np.float32(1)
    b = r.random((k, n), dtype=np.float32) * np.float32(2) - np.float32(1)
    return a, b


def _inputs(case, seed):
    """The numeric inputs of a case, a tuple."""
    kind = case["kind"]
    if kind == "host":
        return _host_operands(case, seed)
    if kind == "batch":
        return _batch_operands(case, seed)
    g = _generator(seed)
    if kind == "gemm":
        return (_matrix(g, case["m"], case["k"], case["a"]),
                _matrix(g, case["k"], case["n"], case["b"]))
    if kind in ("gemv", "residual"):
        a = _matrix(g, case["m"], case["n"], case["a"])
        x = torch.randn(case["n"], device="cuda", generator=g)
        b = torch.randn(case["m"], device="cuda", generator=g)
        return a, x, b
    # points around cluster centres; the centroids a few iterations in, close
    # to the centres but not on them
    n, d, k = case["points"], case["dims"], case["clusters"]
    centres = torch.randn(k, d, device="cuda", generator=g)
    which = torch.randint(k, (n,), device="cuda", generator=g)
    points = centres[which] + torch.randn(n, d, device="cuda", generator=g)
    centroids = centres + 0.1 * torch.randn(k, d, device="cuda", generator=g)
    return points, centroids


def prepare(case, seed):
    kind = case["kind"]
    state = {"kind": kind, "in": _inputs(case, seed)}
    if kind == "host":
        state["c"] = np.zeros((case["m"], case["n"]), dtype=np.float32)
    elif kind == "batch":
        problems, outs = [], []
        for ta, tb, m, n, k, a, lda, b, ldb in state["in"]:
            ldc = (m + 3) // 4 * 4
            c = torch.empty(n, ldc, device="cuda")
            outs.append(c[:, :m].t())
            problems.append((ta, tb, m, n, k, 1.0, a, lda, b, ldb, 0.0, c, ldc))
        state["plan"] = hml.BatchPlan(hml.COL_MAJOR, problems)
        state["out"] = outs
    return state


def _sgemv(a, x, y, alpha, beta):
    m, n = a.shape
    if a.stride(1) == 1:
        hml.sgemv_ex(hml.ROW_MAJOR, hml.OP_N, m, n, alpha, a, n, x, beta, y)
    else:
        hml.sgemv_ex(hml.COL_MAJOR, hml.OP_N, m, n, alpha, a, m, x, beta, y)
    return y


def run(state):
    kind = state["kind"]
    if kind == "gemm":
        a, b = state["in"]
        return hml.sgemm(a, b)
    if kind == "host":
        a, b = state["in"]
        c = state["c"]
        hml.hmlSgemm(c, a, b, a.shape[0], b.shape[1], a.shape[1], 1.0, 0.0)
        return c
    if kind == "gemv":
        a, x, _ = state["in"]
        return _sgemv(a, x, torch.empty(a.shape[0], device="cuda"), 1.0, 0.0)
    if kind == "residual":
        a, x, b = state["in"]
        return _sgemv(a, x, b.clone(), -1.0, 1.0)
    if kind == "batch":
        state["plan"].graph_launch()
        return state["out"]
    points, centroids = state["in"]
    return hml.kmeans_assign(points, centroids)


def work(case):
    kind = case["kind"]
    if kind in ("gemm", "host"):
        m, n, k = case["m"], case["n"], case["k"]
        return {"bytes": 4 * (m * k + k * n + m * n), "flops": 2 * m * n * k}
    if kind in ("gemv", "residual"):
        m, n = case["m"], case["n"]
        return {"bytes": 4 * (m * n + n + m * (2 if kind == "residual" else 1)),
                "flops": 2 * m * n}
    if kind == "batch":
        s = _batch_sizes(case)
        return {"bytes": sum(4 * (m * k + k * n + m * n) for _, _, m, n, k in s),
                "flops": sum(2 * m * n * k for _, _, m, n, k in s)}
    n, d, k = case["points"], case["dims"], case["clusters"]
    return {"bytes": 4 * (n * d + k * d + n), "flops": 2 * n * k * d}


def exact(case, seed):
    """The same outputs in 64 bits.  The k-means indices are whole numbers
    defined by the reference's own FP32 sums (a tie there is no tie here), so
    they have none."""
    kind = case["kind"]
    if kind == "kmeans":
        return None
    ins = _inputs(case, seed)
    if kind == "gemm":
        a, b = ins
        return a.double() @ b.double()
    if kind == "host":
        a, b = ins
        return a.astype(np.float64) @ b.astype(np.float64)
    if kind == "batch":
        out = []
        for ta, tb, m, n, k, a, lda, b, ldb in ins:
            sa = a[:, :k].double() if ta else a[:, :m].t().double()
            sb = b[:, :n].double() if tb else b[:, :k].t().double()
            out.append(sa @ sb)
        return out
    a, x, b = ins
    y = a.double() @ x.double()
    return b.double() - y if kind == "residual" else y
