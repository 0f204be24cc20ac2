"""The untuned SpMV choice (merbit_plan_create): row groups for matrices whose
longest row is short, tiles with a full row_ptr window where the default's tiles
end too many rows, the merge path otherwise -- at the edges of each rule, on
every form of call the plan takes, against the merge-path kernels and the oracle."""
import numpy as np
import pytest
import torch

import merbit_b200 as mb
from merbit_b200 import synth
from oracle import oracle as O
from tests.helpers import csr_from_lengths, stored_values, to_cuda

TOL = {"f64": 1e-13, "f32": 1e-6, "bf16": 1e-6}


def _mixed(lo, hi, n, longest, seed):
    rng = np.random.default_rng(seed)
    L = rng.integers(lo, hi + 1, n)
    L[rng.integers(0, n)] = longest
    return csr_from_lengths(L, ncol=3000, seed=seed)


# matrix, whether row groups serve it, and their lanes per row
CASES = [
    ("mean_above_2.5", csr_from_lengths([2, 3, 3] * 500, ncol=900, seed=1), True, 1),
    ("mean_at_2.5", csr_from_lengths([2, 3] * 700, ncol=900, seed=2), True, 1),
    ("mean_below_2.5", csr_from_lengths([2, 2, 3] * 500, ncol=900, seed=3), False, 0),
    ("mean_below_14", _mixed(13, 13, 1111, 13, 4), True, 1),
    ("mean_14", csr_from_lengths([14] * 777, ncol=900, seed=5), True, 4),
    ("longest_32", _mixed(3, 6, 1501, 32, 6), True, 1),
    ("longest_33", _mixed(3, 6, 1501, 33, 7), True, 4),
    ("mean_39", csr_from_lengths([39] * 300, ncol=900, seed=8), True, 4),
    ("mean_40", csr_from_lengths([40] * 300, ncol=900, seed=9), True, 8),
    ("longest_128", _mixed(0, 60, 900, 128, 10), True, 4),
    ("longest_129", _mixed(0, 60, 900, 129, 11), False, 0),
    ("one_row", csr_from_lengths([7], ncol=50, seed=12), True, 1),
    ("empty_rows_between", csr_from_lengths([0, 9, 0, 0, 11] * 321 + [0], ncol=900, seed=13), True, 1),
]


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", ["f64", "f32", "bf16"])
@pytest.mark.parametrize("name,A,groups,lanes", CASES, ids=[c[0] for c in CASES])
def test_short_row_matrices_start_from_row_groups(name, A, groups, lanes, dtype):
    xy = np.float64 if dtype == "f64" else np.float32
    rp, col, v = to_cuda(A, dtype)
    off = [torch.cat([t[:1], t])[1:] for t in (rp, col, v)]  # not 16-byte aligned
    x = synth.uniform(3, A.ncol).astype(xy)
    y0 = synth.uniform(4, A.nrow).astype(xy)
    yo, ya = O.spmm(A.row_ptr, A.col, stored_values(A, dtype), x)
    xd = torch.from_numpy(x).cuda()
    for arrays, validate in (((rp, col, v), True), ((rp, col, v), False), (off, True)):
        plan = mb.Plan(*arrays, ncol=A.ncol, validate=validate)
        info = plan.info()
        assert (info.kind == 3) == groups, info
        if groups:
            assert info.items_per_thread == lanes
        for alpha, beta in ((1.0, 0.0), (-1.0, 1.0), (0.5, -2.0)):
            y = plan.spmv(xd, torch.from_numpy(y0).cuda(), alpha=alpha, beta=beta).cpu().numpy()
            want = alpha * yo + beta * y0.astype(np.float64)
            scale = abs(alpha) * ya + abs(beta) * np.abs(y0)
            assert (np.abs(y - want) <= TOL[dtype] * np.maximum(scale, 1e-300)).all(), (alpha, beta)
        plan.check()
        # replacing the values keeps a usable choice
        plan.set_values(arrays[2].clone())
        y = plan.spmv(xd).cpu().numpy()
        assert (np.abs(y - yo) <= TOL[dtype] * np.maximum(ya, 1e-300)).all()
        # the SpMM and the merge-path kernels of the same plan
        merge = [c for c in plan.configs() if c[1] != 3]
        plan.set_config(merge[0][0])
        y = plan.spmv(xd).cpu().numpy()
        assert (np.abs(y - yo) <= TOL[dtype] * np.maximum(ya, 1e-300)).all()


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", ["f64", "f32", "bf16"])
def test_tiles_of_empty_rows_start_from_a_full_window(dtype):
    A = csr_from_lengths([300] + [0] * 4000 + [1, 0] * 900 + [2000], ncol=3000, seed=5)
    plan = mb.Plan(*to_cuda(A, dtype), ncol=A.ncol)
    assert plan.info().kind == 1 and plan.info().tile_items == 352
    x = synth.uniform(3, A.ncol).astype(np.float64 if dtype == "f64" else np.float32)
    yo, ya = O.spmm(A.row_ptr, A.col, stored_values(A, dtype), x)
    y = plan.spmv(torch.from_numpy(x).cuda()).cpu().numpy()
    assert (np.abs(y - yo) <= TOL[dtype] * np.maximum(ya, 1e-300)).all()
    # unaligned arrays take CTA tiles, as before
    off = [torch.cat([t[:1], t])[1:] for t in to_cuda(A, dtype)]
    p2 = mb.Plan(*off, ncol=A.ncol)
    assert p2.info().kind == 0
    y = p2.spmv(torch.from_numpy(x).cuda()).cpu().numpy()
    assert (np.abs(y - yo) <= TOL[dtype] * np.maximum(ya, 1e-300)).all()


@pytest.mark.gpu
def test_residual_and_capture_on_the_untuned_choice():
    """PageRank residual and CUDA-graph replay on a plan that starts from row
    groups, without a warm-up product."""
    A = synth.workload("laplace2d_small")
    rp, col, v = to_cuda(A, "f64")
    plan = mb.Plan(rp, col, v)
    assert plan.info().kind == 3
    x = synth.uniform(1, A.ncol)
    t = synth.uniform(2, A.nrow)
    xd, td = torch.from_numpy(x).cuda(), torch.from_numpy(t).cuda()
    res = torch.zeros(1, dtype=torch.float64, device="cuda")
    y = plan.pagerank_step(xd, td, 0.85, residual=res).cpu().numpy()
    yo, ya = O.spmm(A.row_ptr, A.col, A.vals, x)
    want = 0.85 * yo + (1.0 - 0.85) * t
    assert np.abs(y - want).max() <= 1e-13 * (ya.max() + 1)
    assert abs(res.item() - np.abs(y - x).sum()) <= 1e-12 * np.abs(y - x).sum()
    plan2 = mb.Plan(rp, col, v)
    yd = torch.empty(A.nrow, dtype=torch.float64, device="cuda")
    s = torch.cuda.Stream()
    g = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(g, stream=s):
        plan2.spmv(xd, yd, stream=s)
    for rep in range(2):
        xr = synth.uniform(20 + rep, A.ncol)
        xd.copy_(torch.from_numpy(xr))
        g.replay()
        torch.cuda.synchronize()
        yo, ya = O.spmm(A.row_ptr, A.col, A.vals, xr)
        assert (np.abs(yd.cpu().numpy() - yo) <= 1e-13 * ya).all()
