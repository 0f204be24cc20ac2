"""The SpMM walk at the places where its branches change: rows that end at,
just before and just after the ends of lane-group segments and tiles, runs of
empty rows, rows over several tiles (look-backs, more of them per warp than its
queue holds), vector and scalar stores of Y, and alpha / beta on all of them.

Tolerances as for every SpMM test (component-wise against the
extended-precision oracle): 1e-13 for f64, 1e-6 for f32 / bf16 values."""
import numpy as np
import pytest
import torch

import merbit_b200 as mb
from merbit_b200 import synth
from merbit_b200.autograd import SparseMatrix
from oracle import oracle as O
from tests.helpers import csr_from_lengths, stored_values, to_cuda

TOL = {"f64": 1e-13, "f32": 1e-6, "bf16": 1e-6}
# merge items of a lane group's segment and of a tile (vector width 4)
SEG = {4: 15, 8: 31, 16: 63, 32: 127}
TILE = {4: 480, 8: 496, 16: 504, 32: 508}
# and at vector width 2 (FP64, and widths that are no multiple of 4)
SEG2 = {4: 31, 8: 63, 16: 127, 32: 255}
TILE2 = {4: 496, 8: 504, 16: 508, 32: 510}


def _lengths(k, seg=SEG, tile=TILE):
    s, t = seg[k], tile[k]
    rng = np.random.default_rng(k)
    return np.concatenate([
        np.arange(s - 3, s + 3).repeat(9),           # row ends drift over segment ends
        [s - 1] * 40,                                # every segment one whole row
        np.arange(t - 2, t + 3).repeat(3),           # ... and over tile ends
        [t - 1] * 4, [0] * (2 * t + 1), [1] * (t + 5),
        [0, 3 * t, 0, 0, 2 * t - 1, 2 * t, 1, 2 * t + 1, 0],   # rows over three tiles
        rng.integers(0, 3, 3 * t), [2] * t, [5 * t + 7], [0] * 40,
    ]).astype(np.int64)


def _matrix(k, seed=0, width2=False):
    L = _lengths(k, SEG2, TILE2) if width2 else _lengths(k)
    return csr_from_lengths(L, ncol=4000, seed=seed)


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", ["f64", "f32", "bf16"])
@pytest.mark.parametrize("k", [4, 8, 16, 32])
@pytest.mark.parametrize("alpha,beta,pad", [(1.0, 0.0, 0), (1.0, 0.0, 1), (-0.5, 2.0, 4)])
def test_rows_at_segment_and_tile_ends(dtype, k, alpha, beta, pad):
    A = _matrix(k)
    xy = np.float64 if dtype == "f64" else np.float32
    X = synth.uniform(5, A.ncol * k).reshape(A.ncol, k).astype(xy)
    Y0 = synth.uniform(6, A.nrow * (k + pad)).reshape(A.nrow, k + pad).astype(xy)
    if beta == 0.0:
        Y0[:, :k] = np.nan  # never read
    plan = mb.Plan(*to_cuda(A, dtype), ncol=A.ncol)
    xd = torch.from_numpy(X).cuda()
    yo, ya = O.spmm(A.row_ptr, A.col, stored_values(A, dtype), X, k=k, alpha=alpha)
    want = yo + (beta * Y0[:, :k].astype(np.float64) if beta else 0.0)
    scale = ya + abs(beta) * (np.abs(Y0[:, :k]) if beta else 0.0)
    bits = None
    for _ in range(3):  # launches of either slot parity give the same bits
        Yd = torch.from_numpy(Y0).cuda()
        plan.spmm(xd, Yd[:, :k], alpha=alpha, beta=beta)
        got = Yd.cpu().numpy()
        assert (np.abs(got[:, :k] - want) <= TOL[dtype] * np.maximum(scale, 1e-300)).all()
        assert np.array_equal(got[:, k:], Y0[:, k:])  # columns beyond k untouched
        assert bits is None or np.array_equal(got, bits, equal_nan=True)
        bits = got
    plan.check()


@pytest.mark.gpu
@pytest.mark.parametrize("k", [1, 2, 3, 5, 6, 7, 9, 12, 15, 17, 18, 20, 24, 28, 31, 33, 44])
@pytest.mark.parametrize("dtype,pad", [("f32", 0), ("f32", 4), ("f64", 2), ("bf16", 1)])
def test_columns_that_are_no_power_of_two(dtype, pad, k):
    """A launch whose last lanes have no column: every vector width that k and
    the leading dimension give, rows over several tiles among them, and the
    columns of X and Y beyond k neither read into the result nor written."""
    A = _matrix(16, seed=2)
    xy = np.float64 if dtype == "f64" else np.float32
    X = synth.uniform(11, A.ncol * (k + pad)).reshape(A.ncol, k + pad).astype(xy)
    X[:, k:] = np.nan
    Y0 = synth.uniform(12, A.nrow * (k + pad)).reshape(A.nrow, k + pad).astype(xy)
    plan = mb.Plan(*to_cuda(A, dtype), ncol=A.ncol)
    yo, ya = O.spmm(A.row_ptr, A.col, stored_values(A, dtype), X[:, :k].copy(), k=k)
    yo, ya = yo.reshape(-1, k), ya.reshape(-1, k)
    for alpha, beta in ((1.0, 0.0), (2.0, 0.5)):
        Yd = torch.from_numpy(Y0).cuda()
        plan.spmm(torch.from_numpy(X).cuda()[:, :k], Yd[:, :k], alpha=alpha, beta=beta)
        got = Yd.cpu().numpy()
        want = alpha * yo + beta * Y0[:, :k].astype(np.float64)
        scale = abs(alpha) * ya + abs(beta) * np.abs(Y0[:, :k])
        assert (np.abs(got[:, :k] - want) <= TOL[dtype] * np.maximum(scale, 1e-300)).all()
        assert np.array_equal(got[:, k:], Y0[:, k:])
    plan.check()


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", ["f64", "f32", "bf16"])
@pytest.mark.parametrize("kk", [4, 8, 16, 32])
@pytest.mark.parametrize("alpha,beta", [(1.0, 0.0), (-0.5, 2.0)])
def test_vector_width_two_at_segment_and_tile_ends(dtype, kk, alpha, beta):
    """k = kk - 2 (and kk in FP64): tiles of an odd length per group of kk/2 lanes."""
    A = _matrix(kk, seed=4, width2=True)
    xy = np.float64 if dtype == "f64" else np.float32
    for k in ([kk - 2, kk] if dtype == "f64" else [kk - 2]):
        if k < 3:
            continue
        X = synth.uniform(15, A.ncol * k).reshape(A.ncol, k).astype(xy)
        Y0 = synth.uniform(16, A.nrow * k).reshape(A.nrow, k).astype(xy)
        plan = mb.Plan(*to_cuda(A, dtype), ncol=A.ncol)
        yo, ya = O.spmm(A.row_ptr, A.col, stored_values(A, dtype), X, k=k)
        want = alpha * yo + beta * Y0.astype(np.float64)
        scale = abs(alpha) * ya + abs(beta) * np.abs(Y0)
        for _ in range(2):  # either slot parity
            Yd = torch.from_numpy(Y0).cuda()
            plan.spmm(torch.from_numpy(X).cuda(), Yd, alpha=alpha, beta=beta)
            got = Yd.cpu().numpy()
            assert (np.abs(got - want) <= TOL[dtype] * np.maximum(scale, 1e-300)).all()
        plan.check()


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", ["f64", "f32"])
@pytest.mark.parametrize("k", [4, 8, 16, 32])
def test_tiles_of_small_and_large_matrices_agree_with_the_oracle(dtype, k):
    """Matrices on both sides of one round of the smaller tile, long rows in
    them: whichever tile the size picks gives the oracle's product."""
    xy = np.float64 if dtype == "f64" else np.float32
    rng = np.random.default_rng(k)
    for rows in (300, 18_000, 24_000, 40_000):
        L = rng.integers(0, 60, rows)
        L[rows // 2] = 3000
        rp = np.zeros(rows + 1, np.int32)
        np.cumsum(L, out=rp[1:])
        nnz = int(rp[-1])
        A = synth.CSR(rp, rng.integers(0, 5000, nnz, dtype=np.int32), rng.standard_normal(nnz), 5000)
        X = synth.uniform(17, A.ncol * k).reshape(A.ncol, k).astype(xy)
        plan = mb.Plan(*to_cuda(A, dtype), ncol=A.ncol)
        yo, ya = O.spmm(A.row_ptr, A.col, stored_values(A, dtype), X, k=k)
        xd = torch.from_numpy(X).cuda()
        for _ in range(2):
            Y = plan.spmm(xd).cpu().numpy()
            assert (np.abs(Y - yo) <= TOL[dtype] * np.maximum(ya, 1e-300)).all()
        plan.check()


@pytest.mark.gpu
def test_captured_product_with_the_slots_of_narrower_ones():
    """A product of 20 columns captured after products of 16 and 4 (whose
    carry slots the plan then holds), as when each power of two had its own."""
    A = _matrix(16, seed=3)
    k = 20
    X = synth.uniform(13, A.ncol * k).reshape(A.ncol, k).astype(np.float32)
    plan = mb.Plan(*to_cuda(A, "f32"), ncol=A.ncol)
    xd = torch.from_numpy(X).cuda()
    Yd = torch.zeros(A.nrow, k, dtype=torch.float32, device="cuda")
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        plan.spmm(xd[:, :16], Yd[:, :16])
        plan.spmm(xd[:, 16:], Yd[:, 16:])
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        plan.spmm(xd, Yd, stream=s)
    yo, ya = O.spmm(A.row_ptr, A.col, A.vals.astype(np.float32), X, k=k)
    for _ in range(3):
        Yd.fill_(float("nan"))
        g.replay()
        torch.cuda.synchronize()
        assert (np.abs(Yd.cpu().numpy() - yo) <= 1e-6 * np.maximum(ya, 1e-300)).all()


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", ["f64", "f32"])
@pytest.mark.parametrize("k", [1, 2, 4, 8, 16, 32])
def test_fused_backward_at_segment_and_tile_ends(dtype, k):
    """The same rows as the columns of A (rows of the transpose plan)."""
    B = _matrix(max(k, 4), seed=1)
    rows = np.repeat(np.arange(B.nrow), np.diff(B.row_ptr))
    order = np.lexsort((rows, B.col))
    rp = np.zeros(B.ncol + 1, np.int32)
    np.cumsum(np.bincount(B.col, minlength=B.ncol), out=rp[1:])
    A = synth.CSR(rp, rows[order].astype(np.int32), B.vals[order], B.nrow)  # A = B^T
    xy = np.float64 if dtype == "f64" else np.float32
    G = synth.uniform(7, A.nrow * k).reshape(A.nrow, k).astype(xy)
    X = synth.uniform(8, A.ncol * k).reshape(A.ncol, k).astype(xy)
    M = SparseMatrix(*to_cuda(A, dtype), ncol=A.ncol)
    dX, dv = M.backward_fused(torch.from_numpy(G).cuda(), torch.from_numpy(X).cuda())
    v = stored_values(A, dtype)
    do = O.spmm_t(A.row_ptr, A.col, v, G, A.ncol)
    da = O.spmm_t(A.row_ptr, A.col, np.abs(v), np.abs(G), A.ncol)
    assert (np.abs(dX.cpu().numpy() - do) <= TOL[dtype] * np.maximum(da, 1e-300)).all()
    ar = np.repeat(np.arange(A.nrow), np.diff(A.row_ptr))
    g64, x64 = G.astype(np.longdouble)[ar], X.astype(np.longdouble)[A.col]
    want, scale = (g64 * x64).sum(1), np.abs(g64 * x64).sum(1)
    # at most 32 products and their sums, each within one unit of the partial sums
    eps = np.finfo(xy).eps
    assert (np.abs(dv.cpu().numpy() - want) <= (k + 1) * eps * np.maximum(scale, 1e-300)).all()


@pytest.mark.gpu
def test_more_look_backs_than_a_warp_queues():
    """Rows of 700 nonzeros (three tiles of 256 items at k = 1): every warp
    completes more split rows than its queue of 8 holds."""
    nrow, length, ncol = 44_000, 700, 5_000
    rng = np.random.default_rng(4)
    rp = (np.arange(nrow + 1) * length).astype(np.int32)
    col = rng.integers(0, ncol, nrow * length, dtype=np.int32)
    vals = rng.standard_normal(nrow * length).astype(np.float32)
    A = synth.CSR(rp, col, vals.astype(np.float64), ncol)
    X = synth.uniform(9, ncol).reshape(ncol, 1).astype(np.float32)
    plan = mb.Plan(*to_cuda(A, "f32"), ncol=ncol)
    Y = plan.spmm(torch.from_numpy(X).cuda())
    yo, ya = O.spmm(A.row_ptr, A.col, vals, X, k=1)
    assert (np.abs(Y.cpu().numpy() - yo.reshape(-1, 1)) <= 1e-6 * ya.reshape(-1, 1)).all()
    plan.check()
