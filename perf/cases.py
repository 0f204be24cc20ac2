"""The workloads whose time this framework is judged by, on one GPU.

Each case is one call (or one short sequence of calls) that a program makes
through the public Python entry points: the sparse products of a solver, a
graph iteration, a training step, a batch of small matrices, and the harness
front end that turns COO triplets into a product.  Matrices and vectors are
drawn on the GPU from a seed, with the structure and the value distributions
of the repository's benchmark configurations:

* ``laplace2d``  5-point Laplacian of an nx x ny grid, values 4 / -1;
* ``stencil27``  27-point stencil of an nx x ny x nz grid, N(0,1) values and a
  dominant diagonal;
* ``zipf``       row lengths from a Zipf(1.8) law capped at 200,000 entries,
  10% empty rows, sorted columns spread uniformly, N(0,1) values;
* ``rmat``       R-MAT graphs (0.57, 0.19, 0.19, 0.05) of n nodes and n * deg
  distinct edges, N(0,1) values (1/outdegree for PageRank).

``listed`` names the fixed cases, ``draw`` gives further ones from the same
ranges, ``prepare`` builds what a program holds before the call, ``run`` makes
the call, ``work`` counts the bytes and operations it cannot do without, and
``exact`` is the same result in 64-bit arithmetic from plain torch.
"""
import functools
import math

import numpy as np
import torch

import merbit_b200 as mb
from merbit_b200.autograd import SparseMatrix

DEV = "cuda"
VALS = {"f64": torch.float64, "f32": torch.float32, "bf16": torch.bfloat16}
VBYTES = {"f64": 8, "f32": 4, "bf16": 2}
ZIPF_S, ZIPF_CAP, ZIPF_EMPTY = 1.8, 200_000, 0.1
RMAT = (0.57, 0.19, 0.19, 0.05)


def _xy(dtype):
    return torch.float64 if dtype == "f64" else torch.float32


def _gen(seed, stream):
    g = torch.Generator(device=DEV)
    g.manual_seed(1_000_003 * int(seed) + stream)
    return g


def _uniform(g, *shape, dtype):
    return torch.rand(*shape, generator=g, device=DEV, dtype=dtype).mul_(2).sub_(1)


# --------------------------------------------------------------------------
# Structure: (row_ptr int32, col int32) on the GPU
# --------------------------------------------------------------------------

@functools.lru_cache(maxsize=8)
def _zipf_lengths(n, ncol):
    """Row lengths of the Zipf law at n evenly spaced quantiles (so the number
    of nonzeros depends on n alone), empty rows first; prepare shuffles them."""
    cap = min(ZIPF_CAP, ncol)
    cdf = np.cumsum(np.arange(1, cap + 1, dtype=np.float64) ** -ZIPF_S)
    cdf /= cdf[-1]
    full = n - int(ZIPF_EMPTY * n)
    q = (np.arange(full, dtype=np.float64) + 0.5) / full
    length = np.searchsorted(cdf, q) + 1
    return np.concatenate([np.zeros(n - full, np.int64), np.minimum(length, cap)])


def _row_ptr(lengths):
    rp = torch.zeros(lengths.numel() + 1, dtype=torch.int64, device=DEV)
    torch.cumsum(lengths, 0, out=rp[1:])
    return rp


def _zipf(n, seed):
    g = _gen(seed, 1)
    lengths = torch.from_numpy(_zipf_lengths(n, n)).to(DEV)
    lengths = lengths[torch.randperm(n, generator=g, device=DEV)]
    rp = _row_ptr(lengths)
    nnz = int(rp[-1])
    # entry j of a row of L lies in the j-th of L equal column intervals
    j = torch.arange(nnz, device=DEV) - torch.repeat_interleave(rp[:-1], lengths)
    width = torch.repeat_interleave(float(n) / lengths.clamp(min=1).double(), lengths)
    col = ((j + torch.rand(nnz, generator=g, device=DEV, dtype=torch.float64)) * width).long()
    return rp.int(), col.clamp_(max=n - 1).int()


def _grid(dims, offsets):
    """Neighbours inside the grid, by rising linear index."""
    nx, ny, nz = dims
    n = nx * ny * nz
    i = torch.arange(n, device=DEV, dtype=torch.int32)
    ix, iy, iz = i % nx, (i // nx) % ny, i // (nx * ny)
    cols, keep = [], []
    for dz, dy, dx in offsets:
        jx, jy, jz = ix + dx, iy + dy, iz + dz
        keep.append((jx >= 0) & (jx < nx) & (jy >= 0) & (jy < ny) & (jz >= 0) & (jz < nz))
        cols.append((jz * ny + jy) * nx + jx)
    keep = torch.stack(keep, 1)
    col = torch.stack(cols, 1)[keep]
    return _row_ptr(keep.sum(1)).int(), col.contiguous()


def _laplace2d(nx, ny):
    return _grid((nx, ny, 1), [(0, -1, 0), (0, 0, -1), (0, 0, 0), (0, 0, 1), (0, 1, 0)])


def _stencil27(nx, ny, nz):
    r = (-1, 0, 1)
    return _grid((nx, ny, nz), [(dz, dy, dx) for dz in r for dy in r for dx in r])


def _rmat_edges(n, edges, seed, stream=2):
    """`edges` distinct (row, col) pairs as sorted keys row * n + col."""
    g = _gen(seed, stream)
    levels = max(1, math.ceil(math.log2(n)))
    a, b, c, _ = RMAT
    keys = torch.empty(0, dtype=torch.int64, device=DEV)
    while keys.numel() < edges:
        m = int(1.3 * (edges - keys.numel())) + 64
        row = torch.zeros(m, dtype=torch.int64, device=DEV)
        col = torch.zeros(m, dtype=torch.int64, device=DEV)
        for _ in range(levels):
            u = torch.rand(m, generator=g, device=DEV)
            row = 2 * row + (u >= a + b)
            col = 2 * col + (((u >= a) & (u < a + b)) | (u >= a + b + c))
        row, col = (row * n) >> levels, (col * n) >> levels
        keys = torch.unique(torch.cat([keys, row * n + col]))
    drop = torch.randperm(keys.numel(), generator=g, device=DEV)[:edges]
    return keys[drop.sort().values]


def _rmat(n, deg, seed, stream=2):
    keys = _rmat_edges(n, n * deg, seed, stream)
    lengths = torch.bincount(keys // n, minlength=n)
    return _row_ptr(lengths).int(), (keys % n).int()


def _structure(case, seed):
    kind = case["matrix"]
    if kind == "laplace2d":
        return _laplace2d(case["nx"], case["ny"])
    if kind == "stencil27":
        return _stencil27(case["nx"], case["ny"], case["nz"])
    if kind == "zipf":
        return _zipf(case["n"], seed)
    return _rmat(case["n"], case["deg"], seed)


def _size(case):
    """(rows, nonzeros) of a case's matrix."""
    kind = case["matrix"]
    if kind == "laplace2d":
        nx, ny = case["nx"], case["ny"]
        return nx * ny, 5 * nx * ny - 2 * nx - 2 * ny
    if kind == "stencil27":
        d = (case["nx"], case["ny"], case["nz"])
        return d[0] * d[1] * d[2], math.prod(3 * v - 2 for v in d)
    if kind == "zipf":
        return case["n"], int(_zipf_lengths(case["n"], case["n"]).sum())
    return case["n"], case["n"] * case["deg"]


def _rows_of(rp):
    return torch.repeat_interleave(torch.arange(rp.numel() - 1, device=DEV), (rp[1:] - rp[:-1]).long())


def _values(case, rp, col, seed):
    g = _gen(seed, 3)
    v = torch.randn(col.numel(), generator=g, device=DEV, dtype=torch.float32).double()
    if case["matrix"] == "laplace2d":
        v = torch.where(_rows_of(rp) == col, 4.0, -1.0).double()
    elif case["matrix"] == "stencil27":
        v[_rows_of(rp) == col] += 32.0  # diagonally dominant
    return v.to(VALS[case["dtype"]])


# --------------------------------------------------------------------------
# Cases
# --------------------------------------------------------------------------

def listed():
    return [
        # The smallest product a solver makes: a 5-point Laplacian that stays in
        # L2, one call per iteration; launch and host time weigh most here.
        {"name": "spmv laplace2d 256 f64", "kind": "spmv", "matrix": "laplace2d", "nx": 256, "ny": 256,
         "dtype": "f64", "tune": True, "residual": False},
        # The headline configuration: a power-law matrix in plain FP64, tuned
        # once and multiplied many times.
        {"name": "spmv zipf 2M f64", "kind": "spmv", "matrix": "zipf", "n": 2_000_000,
         "dtype": "f64", "tune": True, "residual": False},
        # The same law at another size in the BF16-value precision form, on a
        # plan used as it was created.
        {"name": "spmv zipf 1.1M bf16", "kind": "spmv", "matrix": "zipf", "n": 1_100_003,
         "dtype": "bf16", "tune": False, "residual": False},
        # The precision form's benchmark: a 3-D 27-point stencil, FP32 values.
        {"name": "spmv stencil 160 f32", "kind": "spmv", "matrix": "stencil27", "nx": 160, "ny": 160, "nz": 160,
         "dtype": "f32", "tune": True, "residual": False},
        # The residual r = b - A x of an iterative solver on an odd-sized grid,
        # with a plan used as it was created (alpha = -1, beta = 1).
        {"name": "residual stencil 113 f64", "kind": "spmv", "matrix": "stencil27", "nx": 113, "ny": 97, "nz": 61,
         "dtype": "f64", "tune": False, "residual": True},
        # PageRank on a web-like graph: 20 fused steps, the residual read by the
        # host every second one.
        {"name": "pagerank rmat 400k f64", "kind": "pagerank", "matrix": "rmat", "n": 400_003, "deg": 16,
         "dtype": "f64", "tune": True},
        # A block of 8 vectors in FP64 (block Krylov methods).
        {"name": "spmm zipf 500k f64 k8", "kind": "spmm", "matrix": "zipf", "n": 500_009, "dtype": "f64", "k": 8,
         "pad": 0},
        # Node features through a graph, a width that is no power of two.
        {"name": "spmm rmat 300k f32 k20", "kind": "spmm", "matrix": "rmat", "n": 300_007, "deg": 24,
         "dtype": "f32", "k": 20, "pad": 0},
        # The differentiation benchmark: a training step's forward and backward
        # with gradients for the values and for X.
        {"name": "grad zipf 1M f32 k16", "kind": "grad", "matrix": "zipf", "n": 1_000_000, "dtype": "f32", "k": 16},
        # The batched benchmark at k = 1: many uneven graphs in one launch.
        {"name": "batch rmat 64 f32 k1", "kind": "batch", "matrix": "rmat", "count": 64, "nmin": 4_000,
         "nmax": 300_000, "dtype": "f32", "k": 1},
        # The batched benchmark at its widest, k = 32.
        {"name": "batch rmat 32 f32 k32", "kind": "batch", "matrix": "rmat", "count": 32, "nmin": 4_000,
         "nmax": 300_000, "dtype": "f32", "k": 32},
        # The harness from end to end: unsorted COO triplets, sorted, turned
        # into CSR, planned and multiplied once.
        {"name": "coo rmat 250k f64", "kind": "coo", "matrix": "rmat", "n": 250_007, "deg": 16, "dtype": "f64"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_matrix(rng, nnz_lo, nnz_hi, kinds):
    """A matrix of one of `kinds` with about a log-uniform number of nonzeros."""
    nnz, kind = _log_int(rng, nnz_lo, nnz_hi), rng.choice(kinds)
    if kind == "laplace2d":
        n = max(64, nnz // 5)
        nx = max(8, int(math.sqrt(n) * rng.uniform(0.5, 2.0)))
        return {"matrix": kind, "nx": nx, "ny": max(8, n // nx)}
    if kind == "stencil27":
        side = max(6.0, (nnz / 27.0) ** (1.0 / 3.0))
        nx, ny = (max(5, int(side * rng.uniform(0.6, 1.6))) for _ in range(2))
        return {"matrix": kind, "nx": nx, "ny": ny, "nz": max(5, int(side ** 3 / (nx * ny)))}
    if kind == "zipf":
        return {"matrix": kind, "n": max(500, nnz // 22)}
    deg = rng.randint(8, 48)
    return {"matrix": kind, "n": max(2_000, nnz // deg), "deg": deg}


def draw(rng):
    kind = rng.choice(["spmv", "spmv", "spmv", "pagerank", "spmm", "spmm", "grad", "batch", "batch", "coo"])
    every = ["laplace2d", "stencil27", "zipf", "rmat"]
    if kind == "spmv":
        return {"kind": kind, **_draw_matrix(rng, 40_000, 40_000_000, every), "dtype": rng.choice(list(VALS)),
                "tune": rng.random() < 0.5, "residual": rng.random() < 0.3}
    if kind == "pagerank":
        return {"kind": kind, **_draw_matrix(rng, 100_000, 8_000_000, ["rmat"]), "dtype": rng.choice(["f64", "f32"]),
                "tune": True}
    if kind == "spmm":
        return {"kind": kind, **_draw_matrix(rng, 100_000, 12_000_000, every), "dtype": rng.choice(list(VALS)),
                "k": rng.choice([rng.randint(2, 40), rng.choice([2, 4, 8, 16, 32])]), "pad": rng.choice([0, 0, 4])}
    if kind == "grad":
        return {"kind": kind, **_draw_matrix(rng, 100_000, 12_000_000, ["zipf", "rmat"]),
                "dtype": rng.choice(["f64", "f32"]), "k": rng.choice([1, 4, 8, 16, 32])}
    if kind == "batch":
        return {"kind": kind, "matrix": "rmat", "count": rng.randint(4, 48), "nmin": 2_000,
                "nmax": _log_int(rng, 10_000, 200_000), "dtype": rng.choice(["f32", "f32", "bf16", "f64"]),
                "k": rng.choice([1, 2, 4, 8, 16, 32])}
    return {"kind": kind, **_draw_matrix(rng, 100_000, 8_000_000, ["rmat"]), "dtype": rng.choice(["f64", "f32"])}


# --------------------------------------------------------------------------
# State
# --------------------------------------------------------------------------

def _batch_sizes(case):
    """(rows, average degree) of each member, evenly spread over the range of
    sizes (in the logarithm) and of degrees (8 to 48, in mixed order)."""
    m = case["count"]
    ratio = case["nmax"] / case["nmin"]
    return [(int(case["nmin"] * ratio ** ((i + 0.5) / m)), 8 + (i * 17) % 41) for i in range(m)]


def _inputs(case, seed):
    """The tensors a case starts from (no plan)."""
    kind = case["kind"]
    xy, vt = _xy(case["dtype"]), VALS[case["dtype"]]
    if kind == "batch":
        mats = []
        for i, (n, deg) in enumerate(_batch_sizes(case)):
            rp, col = _rmat(n, deg, seed, 16 + i)
            g = _gen(seed, 1000 + i)
            mats.append((rp, col, torch.randn(col.numel(), generator=g, device=DEV).to(vt),
                         _uniform(g, n, case["k"], dtype=xy)))
        return {"mats": mats}
    if kind == "coo":
        n = case["n"]
        g = _gen(seed, 4)
        keys = _rmat_edges(n, n * case["deg"], seed)
        keys = keys[torch.randperm(keys.numel(), generator=g, device=DEV)]
        vals = torch.randn(keys.numel(), generator=g, device=DEV, dtype=xy)
        return {"rows": (keys // n).int(), "cols": (keys % n).int(), "vals": vals, "n": n,
                "x": _uniform(g, n, dtype=xy)}
    rp, col = _structure(case, seed)
    n = rp.numel() - 1
    g = _gen(seed, 5)
    if kind == "pagerank":
        out = torch.bincount(col, minlength=n).clamp(min=1).double()
        return {"rp": rp, "col": col, "vals": (1.0 / out[col.long()]).to(vt), "n": n}
    vals = _values(case, rp, col, seed)
    if kind == "spmv":
        return {"rp": rp, "col": col, "vals": vals, "n": n, "x": _uniform(g, n, dtype=xy),
                "b": _uniform(g, n, dtype=xy) if case["residual"] else None}
    k, pad = case["k"], case.get("pad", 0)
    x = _uniform(g, n, k + pad, dtype=xy)[:, :k]
    s = {"rp": rp, "col": col, "vals": vals, "n": n, "x": x}
    if kind == "grad":
        s["g"] = torch.randn(n, k, generator=g, device=DEV, dtype=xy)
    return s


def prepare(case, seed):
    s = _inputs(case, seed)
    kind, xy = case["kind"], _xy(case["dtype"])
    s["kind"] = kind
    if kind == "batch":
        offs, rows = [], 0
        for rp, *_ in s["mats"]:
            offs.append(rows)
            rows += -(-(rp.numel() - 1) // 64) * 64
        s["y"] = torch.zeros(rows, case["k"], dtype=xy, device=DEV)
        s["plans"] = [mb.Plan(rp, col, v) for rp, col, v, _ in s["mats"]]
        s["batch"] = mb.Batch(s["plans"], [m[3] for m in s["mats"]],
                              [s["y"][o:o + p.nrow] for o, p in zip(offs, s["plans"])])
    elif kind == "grad":
        s["vals"].requires_grad_()
        s["x"].requires_grad_()
        s["A"] = SparseMatrix(s["rp"], s["col"], s["vals"])
    elif kind != "coo":
        s["plan"] = mb.Plan(s["rp"], s["col"], s["vals"])
        if case.get("tune"):
            s["plan"].tune()
        if kind == "spmv":
            s["y"] = torch.empty(s["n"], dtype=xy, device=DEV)
        elif kind == "spmm":
            s["Y"] = torch.empty(s["n"], case["k"], dtype=xy, device=DEV)
    return s


def run(s):
    kind = s["kind"]
    if kind == "spmv":
        if s["b"] is None:
            return s["plan"].spmv(s["x"], s["y"])
        return s["plan"].spmv(s["x"], s["b"].clone(), alpha=-1.0, beta=1.0)
    if kind == "pagerank":
        x, steps, history = mb.pagerank(s["plan"], damp=0.85, tol=0.0, maxiter=10, perrnd=2)
        return {"x": x, "steps": steps, "residual": history}
    if kind == "spmm":
        return s["plan"].spmm(s["x"], s["Y"])
    if kind == "grad":
        s["vals"].grad = s["x"].grad = None
        y = s["A"].matmul(s["x"])
        y.backward(s["g"])
        return {"y": y.detach(), "dx": s["x"].grad, "dvals": s["vals"].grad}
    if kind == "batch":
        s["batch"].run()
        return s["y"]
    rows, cols, vals = s["rows"].clone(), s["cols"].clone(), s["vals"].clone()
    mb.coo_sort(rows, cols, vals)
    rp = mb.coo_to_csr(rows, s["n"])
    plan = mb.Plan(rp, cols, vals)
    y = plan.spmv(s["x"])
    return {"row_ptr": rp, "cols": cols, "vals": vals, "y": y}


# --------------------------------------------------------------------------
# What a call cannot do without
# --------------------------------------------------------------------------

def _product(n, nnz, dtype, k):
    """(bytes, flops) of Y = A X: matrix, X and Y once each."""
    xb = 8 if dtype == "f64" else 4
    return 4 * (n + 1) + nnz * (4 + VBYTES[dtype]) + 2 * k * n * xb, 2 * nnz * k


def work(case):
    kind, dtype = case["kind"], case["dtype"]
    xb = 8 if dtype == "f64" else 4
    if kind == "batch":
        parts = [_product(n, n * deg, dtype, case["k"]) for n, deg in _batch_sizes(case)]
        return {"bytes": sum(p[0] for p in parts), "flops": sum(p[1] for p in parts)}
    n, nnz = _size(case)
    if kind == "spmv":
        b, f = _product(n, nnz, dtype, 1)
        return {"bytes": b + (n * xb if case["residual"] else 0), "flops": f}
    if kind == "pagerank":  # 20 steps, each also reading the teleport vector
        b, f = _product(n, nnz, dtype, 1)
        return {"bytes": 20 * (b + n * xb), "flops": 20 * (f + 4 * n)}
    if kind == "spmm":
        b, f = _product(n, nnz, dtype, case["k"])
        return {"bytes": b, "flops": f}
    if kind == "grad":
        b, f = _product(n, nnz, dtype, case["k"])
        # backward: the matrix, G and X read, dX and dvals written
        back = 4 * (n + 1) + nnz * (4 + VBYTES[dtype]) + 3 * case["k"] * n * xb + nnz * VBYTES[dtype]
        return {"bytes": b + back, "flops": 3 * f}
    # coo: triplets read, the sorted CSR written, then read for the product
    csr = 4 * (n + 1) + nnz * (4 + xb)
    return {"bytes": nnz * (8 + xb) + 2 * csr + 2 * n * xb, "flops": 2 * nnz}


# --------------------------------------------------------------------------
# The same results in 64 bits
# --------------------------------------------------------------------------

def _mm64(rp, col, vals, x, ncol=None):
    """A x in FP64 for a matrix or vector x, a few columns at a time."""
    n = rp.numel() - 1
    rows = _rows_of(rp)
    x2 = (x if x.dim() == 2 else x.unsqueeze(1)).detach().double()
    v, c = vals.detach().double(), col.long()
    y = torch.zeros(n, x2.shape[1], dtype=torch.float64, device=DEV)
    for j in range(x2.shape[1]):
        y[:, j].index_add_(0, rows, v * x2[c, j])
    return y if x.dim() == 2 else y[:, 0]


def exact(case, seed):
    s = _inputs(case, seed)
    kind = case["kind"]
    if kind == "batch":
        out = []
        for rp, col, v, x in s["mats"]:
            n = rp.numel() - 1
            y = torch.zeros(-(-n // 64) * 64, case["k"], dtype=torch.float64, device=DEV)
            y[:n] = _mm64(rp, col, v, x)
            out.append(y)
        return torch.cat(out)
    if kind == "coo":
        n = s["n"]
        order = (s["rows"].long() * n + s["cols"].long()).argsort()
        rows, cols, vals = s["rows"][order], s["cols"][order], s["vals"][order]
        rp = _row_ptr(torch.bincount(rows, minlength=n)).int()
        return {"row_ptr": rp, "cols": cols, "vals": vals.double(), "y": _mm64(rp, cols, vals, s["x"])}
    if kind == "pagerank":
        n, history = s["n"], []
        t = torch.full((n,), 1.0 / n, dtype=_xy(case["dtype"]), device=DEV).double()
        x = t.clone()
        for step in range(20):
            y = 0.85 * _mm64(s["rp"], s["col"], s["vals"], x) + (1.0 - 0.85) * t
            if step % 2:
                history.append(float((y - x).abs().sum()))
            x = y
        return {"x": x, "steps": None, "residual": history}
    y = _mm64(s["rp"], s["col"], s["vals"], s["x"])
    if kind == "spmv":
        return y if s["b"] is None else s["b"].double() - y
    if kind == "spmm":
        return y
    rows, col = _rows_of(s["rp"]), s["col"].long()
    g, x, v = s["g"].double(), s["x"].detach().double(), s["vals"].detach().double()
    dx, dv = torch.zeros_like(x), torch.zeros(col.numel(), dtype=torch.float64, device=DEV)
    for j in range(case["k"]):
        gj = g[rows, j]
        dx[:, j].index_add_(0, col, v * gj)
        dv += gj * x[col, j]
    return {"y": y, "dx": dx, "dvals": dv}
