"""Which tiles a product takes, read off the partition that its first call adds
to the plan's metadata (8 bytes a tile boundary), and that every choice is right.

Tolerances as for every SpMM test: 1e-13 for f64, 1e-6 for f32 values."""
import numpy as np
import pytest
import torch

import merbit_b200 as mb
from merbit_b200 import synth
from merbit_b200.autograd import SparseMatrix
from oracle import oracle as O
from tests.helpers import stored_values, to_cuda

TOL = {"f64": 1e-13, "f32": 1e-6, "bf16": 1e-6}


def _warps(ctas):
    return 4 * ctas * torch.cuda.get_device_properties(0).multi_processor_count


def _added_tiles(plan, call):
    before = plan.info().metadata_bytes
    out = call()
    torch.cuda.synchronize()
    return (plan.info().metadata_bytes - before) // 8 - 1, out


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", ["f64", "f32"])
def test_rounds_are_as_wide_as_the_fused_backward(dtype):
    """Between one round of 16 warps an SM and one of 20 in 272-item tiles: FP64
    with the fused dval holds 16 and keeps the larger tile, FP32 takes the smaller."""
    k = 8
    A = synth.stencil27(30, 30, 30, seed=4)
    n = A.nrow
    items = A.nrow + A.nnz
    assert 272 * _warps(4) < items < 272 * _warps(5)
    xy = np.float64 if dtype == "f64" else np.float32
    G = synth.uniform(5, n * k).reshape(n, k).astype(xy)
    X = synth.uniform(6, n * k).reshape(n, k).astype(xy)
    M = SparseMatrix(*to_cuda(A, dtype), ncol=A.ncol)
    T = M.transpose_plan()
    Gd, Xd = torch.from_numpy(G).cuda(), torch.from_numpy(X).cuda()
    tiles, (dX, _) = _added_tiles(T, lambda: M.backward_fused(Gd, Xd))
    assert tiles == -(-items // (496 if dtype == "f64" else 272))
    v = stored_values(A, dtype)
    do = O.spmm_t(A.row_ptr, A.col, v, G, A.ncol)
    da = O.spmm_t(A.row_ptr, A.col, np.abs(v), np.abs(G), A.ncol)
    assert (np.abs(dX.cpu().numpy() - do) <= TOL[dtype] * np.maximum(da, 1e-300)).all()


def _ends_at(tile, seg, items, seed):
    """At least `items` merge items in rows that end at, before and after the ends
    of segments and tiles; empty rows, rows over several tiles."""
    L = np.array([seg - 1, seg, seg - 2, 0, 0, tile - 1, tile, tile - 2, 1, 2, 2 * tile - 1, 0, 3 * tile,
                  5 * tile + 7, 1, 1, 0, 4 * seg])
    L = np.tile(L, -(-items // int(L.sum() + L.size)))
    rng = np.random.default_rng(seed)
    rp = np.concatenate([[0], np.cumsum(L)]).astype(np.int32)
    nnz, ncol = int(rp[-1]), 3000
    return synth.CSR(rp, rng.integers(0, ncol, nnz, dtype=np.int32), rng.standard_normal(nnz), ncol, "ends")


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", ["f64", "f32", "bf16"])
@pytest.mark.parametrize("k, tile", [(1, 480), (2, None), (1, 256)])
def test_one_and_two_columns_at_tile_ends(dtype, k, tile):
    tile = tile or (224 if dtype == "f64" else 352)
    few = tile == 256  # one round of 256-item tiles
    A = _ends_at(tile, tile // 32, 400_000 if few else 256 * _warps(6) + 50_000, seed=k)
    xy = np.float64 if dtype == "f64" else np.float32
    X = synth.uniform(7, A.ncol * k).reshape(A.ncol, k).astype(xy)
    plan = mb.Plan(*to_cuda(A, dtype), ncol=A.ncol)
    Xd = torch.from_numpy(X).cuda()
    tiles, Y = _added_tiles(plan, lambda: plan.spmm(Xd))
    # (-1: the SpMV has tiles of these items too, 480 untuned, and may have built them)
    assert tiles == -(-(A.nrow + A.nnz) // tile) or (tiles == -1 and tile in (224, 352, 480))
    yo, ya = O.spmm(A.row_ptr, A.col, stored_values(A, dtype), X, k=k)
    for _ in range(3):  # both parities
        Y = plan.spmm(Xd, alpha=-0.5, beta=0.0)
        e = np.abs(Y.cpu().numpy().reshape(A.nrow, k) + 0.5 * yo.reshape(A.nrow, k))
        assert (e <= TOL[dtype] * np.maximum(ya.reshape(A.nrow, k), 1e-300)).all()


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", ["f64", "f32"])
def test_one_column_fused_backward_at_tile_ends(dtype):
    """More than one round of 256-item tiles on the transpose plan."""
    B = _ends_at(256, 8, 256 * _warps(7) + 50_000, seed=3)
    rows = np.repeat(np.arange(B.nrow, dtype=np.int32), np.diff(B.row_ptr))
    order = np.lexsort((rows, B.col))
    rp = np.concatenate([[0], np.cumsum(np.bincount(B.col, minlength=B.ncol))]).astype(np.int32)
    A = synth.CSR(rp, rows[order], B.vals[order], B.nrow, "ends transposed")
    xy = np.float64 if dtype == "f64" else np.float32
    G = synth.uniform(8, A.nrow).reshape(-1, 1).astype(xy)
    X = synth.uniform(9, A.ncol).reshape(-1, 1).astype(xy)
    M = SparseMatrix(*to_cuda(A, dtype), ncol=A.ncol)
    dX, dv = M.backward_fused(torch.from_numpy(G).cuda(), torch.from_numpy(X).cuda())
    v = stored_values(A, dtype)
    do = O.spmm_t(A.row_ptr, A.col, v, G, A.ncol)
    da = O.spmm_t(A.row_ptr, A.col, np.abs(v), np.abs(G), A.ncol)
    assert (np.abs(dX.cpu().numpy() - do) <= TOL[dtype] * np.maximum(da, 1e-300)).all()
    ar = np.repeat(np.arange(A.nrow), np.diff(A.row_ptr))
    want = (G.astype(np.float64)[ar] * X.astype(np.float64)[A.col])[:, 0]
    # one product, rounded once
    assert (np.abs(dv.cpu().numpy() - want) <= np.finfo(xy).eps * np.abs(want)).all()


def _launches(call):
    """Kernels that a call captures."""
    rt = pytest.importorskip("cuda.bindings.runtime")
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    g = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(g, stream=s):
        call(s)
    err, _, n = rt.cudaGraphGetNodes(rt.cudaGraph_t(g.raw_cuda_graph()), 0)
    assert int(err) == 0
    return n


@pytest.mark.gpu
@pytest.mark.parametrize("dtype, k, ld, launches", [
    ("f32", 17, 20, 2), ("f32", 17, 17, 2), ("f32", 9, 12, 2), ("f32", 9, 10, 2), ("f32", 9, 9, 1),
    ("f32", 21, 24, 2), ("f32", 21, 22, 1), ("f32", 49, 52, 3), ("f32", 5, 8, 1), ("f32", 20, 20, 1),
    ("bf16", 9, 9, 2), ("bf16", 13, 16, 2), ("bf16", 17, 18, 2), ("bf16", 25, 25, 1),
    ("f64", 17, 18, 2), ("f64", 17, 17, 1), ("f64", 21, 24, 1), ("f64", 9, 10, 1),
])
def test_a_last_column_of_its_own(dtype, k, ld, launches):
    """A column more than a multiple of 4: apart where the others then take whole
    vectors; columns beyond k are neither read nor written."""
    A = _ends_at(504, 63, 2_050_000, seed=9)
    xy = np.float64 if dtype == "f64" else np.float32
    X = synth.uniform(10, A.ncol * k).reshape(A.ncol, k).astype(xy)
    Xd = torch.full((A.ncol, ld), float("nan"), dtype=torch.from_numpy(X).dtype, device="cuda")
    Xd[:, :k] = torch.from_numpy(X)
    Yd = torch.full((A.nrow, ld), -7.0, dtype=Xd.dtype, device="cuda")
    plan = mb.Plan(*to_cuda(A, dtype), ncol=A.ncol)
    yo, ya = O.spmm(A.row_ptr, A.col, stored_values(A, dtype), X, k=k)
    for _ in range(3):
        Yd[:, :k] = float("nan")
        plan.spmm(Xd[:, :k], Yd[:, :k])
        torch.cuda.synchronize()
        e = np.abs(Yd[:, :k].cpu().numpy() - yo)
        assert (e <= TOL[dtype] * np.maximum(ya, 1e-300)).all()
        assert bool((Yd[:, k:] == -7.0).all())
    assert _launches(lambda s: plan.spmm(Xd[:, :k], Yd[:, :k], stream=s)) == launches
