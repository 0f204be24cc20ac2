"""A captured SpMV stays valid when later calls make its plan grow: SpMM
partitions of smaller tiles leave the SpMV's carry words alone, and a
configuration of more tiles takes a block of its own.

Tolerances as for every product (component-wise against the
extended-precision oracle): 1e-13 for f64, 1e-6 for f32 values."""
import numpy as np
import pytest
import torch

import merbit_b200 as mb
from merbit_b200 import synth
from oracle import oracle as O
from tests.helpers import stored_values, to_cuda

TOL = {"f64": 1e-13, "f32": 1e-6}


def _captured_spmv(plan, x, y):
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        plan.spmv(x, y)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        plan.spmv(x, y, stream=s)
    return g


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", ["f64", "f32"])
@pytest.mark.parametrize("matrix", ["zipf", "rmat"])
def test_captured_spmv_after_the_first_spmm(dtype, matrix):
    A = synth.zipf(20000, 1.8, 20000, 0.1, seed=5) if matrix == "zipf" else synth.rmat(12000, 24.0, seed=6)
    xy = np.float64 if dtype == "f64" else np.float32
    plan = mb.Plan(*to_cuda(A, dtype), ncol=A.ncol)
    assert plan.info().kind != 3
    bytes_before = plan.info().metadata_bytes
    xh = synth.uniform(2, A.ncol).astype(xy)
    yo, ya = O.spmm(A.row_ptr, A.col, stored_values(A, dtype), xh)
    x = torch.from_numpy(xh).cuda()
    y = torch.empty(A.nrow, dtype=x.dtype, device="cuda")
    g = _captured_spmv(plan, x, y)

    def replay_is_right():
        y.fill_(float("nan"))
        g.replay()
        torch.cuda.synchronize()
        assert (np.abs(y.cpu().numpy() - yo) <= TOL[dtype] * np.maximum(ya, 1e-300)).all()

    others = []
    for i, k in enumerate((1, 4, 16, 32)):
        Xh = synth.uniform(3 + k, A.ncol * k).reshape(A.ncol, k).astype(xy)
        Yo, Ya = O.spmm(A.row_ptr, A.col, stored_values(A, dtype), Xh, k=k)
        X = torch.from_numpy(Xh).cuda()
        Y = plan.spmm(X)
        # another plan takes whatever the pool has free, and fills it
        others.append(mb.Plan(*to_cuda(A, dtype), ncol=A.ncol))
        others[-1].spmm(X)
        replay_is_right()
        for _ in range(i % 2 + 1):  # eager products in between, an odd and an even number
            plan.spmv(x)
        replay_is_right()
        replay_is_right()
        Y2 = plan.spmm(X)
        torch.cuda.synchronize()
        for got in (Y, Y2):
            e = np.abs(got.cpu().numpy().reshape(A.nrow, k) - Yo.reshape(A.nrow, k))
            assert (e <= TOL[dtype] * np.maximum(Ya.reshape(A.nrow, k), 1e-300)).all()
    plan.check()
    # the partitions of the SpMM tiles (8 bytes a tile boundary) and no words beside them
    tiles = [-(-(A.nrow + A.nnz) // t) + 1 for t in (256, 260)]
    assert plan.info().metadata_bytes - bytes_before <= 8 * 5 * max(tiles)


@pytest.mark.gpu
@pytest.mark.parametrize("eager", [0, 1, 2, 3])
def test_captured_spmv_after_a_configuration_of_more_tiles(eager):
    """Launches on the later block do not turn the captured one's parity."""
    A = synth.zipf(20000, 1.8, 20000, 0.1, seed=5)
    plan = mb.Plan(*to_cuda(A, "f64"), ncol=A.ncol)
    x = torch.from_numpy(synth.uniform(2, A.ncol)).cuda()
    y = torch.empty_like(x)
    items = plan.info().tile_items
    g = _captured_spmv(plan, x, y)
    ref = y.clone()
    smaller = [c for c in plan.configs() if c[1] == 1 and 32 * c[3] < items]
    assert smaller
    mem = []
    for idx, *_ in smaller:
        plan.set_config(idx)
        mem.append(mb.Plan(*to_cuda(A, "f64"), ncol=A.ncol))
        mem[-1].spmv(x)
        z = [plan.spmv(x) for _ in range(eager)]
        for _ in range(2):
            y.fill_(float("nan"))
            g.replay()
            torch.cuda.synchronize()
            assert torch.equal(y, ref)
        assert all(torch.equal(z[0], v) for v in z)
    plan.check()


@pytest.mark.gpu
def test_captured_residual_after_more_partials():
    """More CTAs than the captured step had: its partial sums keep their place.  On
    CTA tiles, where one tile finishes each row and the residual repeats bit for bit
    (warp tiles that share a row leave its term to the later one)."""
    A = synth.laplace2d(1100, 1000)
    plan = mb.Plan(*to_cuda(A, "f64"), ncol=A.ncol)
    plan.set_config(next(c for c in plan.configs() if c[1] == 0 and c[2] * c[3] == 1792)[0])
    n = A.nrow
    x = torch.from_numpy(synth.uniform(2, n)).cuda()
    t = torch.full((n,), 1.0 / n, dtype=torch.float64, device="cuda")
    y, res = torch.empty_like(x), torch.zeros(1, dtype=torch.float64, device="cuda")
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        plan.pagerank_step(x, t, y=y, residual=res)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        plan.pagerank_step(x, t, y=y, residual=res, stream=s)
    ref, yref = float(res), y.clone()
    cta = next(c for c in plan.configs() if c[1] == 0 and c[2] * c[3] == 1152)
    assert (A.nrow + A.nnz) // 1152 > 32 * torch.cuda.get_device_properties(0).multi_processor_count
    plan.set_config(cta[0])
    plan.pagerank_step(x, t, residual=res)
    fill = [mb.Plan(*to_cuda(A, "f64"), ncol=A.ncol) for _ in range(2)]
    for p in fill:
        p.pagerank_step(x, t, residual=torch.zeros_like(res))
    res.zero_()
    g.replay()
    torch.cuda.synchronize()
    assert float(res) == ref and torch.equal(y, yref)


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", ["f64", "f32"])
def test_partitions_of_other_launches_are_checked_for_the_spmv(dtype):
    """A batch and an SpMM leave coordinates alone; an SpMV configuration on the
    same tiles still finds out whether its row_ptr window holds them."""
    L = [300] + [0] * 4000 + [1, 0] * 900 + [2000] + [40] * 700
    rp = np.concatenate([[0], np.cumsum(L)]).astype(np.int32)
    rng = np.random.default_rng(3)
    nnz = int(rp[-1])
    A = synth.CSR(rp, rng.integers(0, 3000, nnz, dtype=np.int32), rng.standard_normal(nnz), 3000, "runs")
    xy = np.float64 if dtype == "f64" else np.float32
    xh = synth.uniform(4, A.ncol).astype(xy)
    yo, ya = O.spmm(A.row_ptr, A.col, stored_values(A, dtype), xh)
    x = torch.from_numpy(xh).cuda()
    fresh = mb.Plan(*to_cuda(A, dtype), ncol=A.ncol)
    plan = mb.Plan(*to_cuda(A, dtype), ncol=A.ncol)
    y = torch.empty(A.nrow, 1, dtype=x.dtype, device="cuda")
    b = mb.Batch([plan], [x.view(-1, 1)], [y])
    for variant, ipts in ((0, (7, 11, 15)), (3, (15, 19, 23))):
        b.set_kernel(1, variant)
        for ipt in ipts:
            b.set_matrix_config(0, ipt)
    b.run()
    plan.spmm(x.view(-1, 1).expand(-1, 2).contiguous())
    usable = plan.configs()
    assert usable == fresh.configs()
    assert len(usable) < mb.lib().merbit_num_configs(plan.dtype)
    for idx, *_ in usable:
        plan.set_config(idx)
        got = plan.spmv(x).cpu().numpy()
        assert (np.abs(got - yo) <= TOL[dtype] * np.maximum(ya, 1e-300)).all(), idx
    plan.check()
