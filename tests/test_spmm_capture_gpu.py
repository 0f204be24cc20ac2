"""SpMM while its stream is being captured: what a plan holds decides what runs,
and nothing but the products' kernels enters the caller's graph.

Tolerances as for every SpMM test (component-wise against the
extended-precision oracle): 1e-13 for f64, 1e-6 for f32 values."""
import numpy as np
import pytest
import torch

import merbit_b200 as mb
from merbit_b200 import synth
from merbit_b200.autograd import SparseMatrix
from oracle import oracle as O
from tests.helpers import stored_values, to_cuda

TOL = {"f64": 1e-13, "f32": 1e-6}
XY = {"f64": np.float64, "f32": np.float32}


def _operands(A, k, dtype, ld=None, seed=3):
    X = synth.uniform(seed + k, A.ncol * k).reshape(A.ncol, k).astype(XY[dtype])
    buf = torch.full((A.ncol, ld or k), float("nan"), dtype=torch.from_numpy(X).dtype, device="cuda")
    buf[:, :k] = torch.from_numpy(X)
    return X, buf[:, :k], torch.zeros(A.nrow, k, dtype=buf.dtype, device="cuda")


def _check(A, dtype, X, Y):
    k = X.shape[1]
    yo, ya = O.spmm(A.row_ptr, A.col, stored_values(A, dtype), X, k=k)
    e = np.abs(Y.cpu().numpy().reshape(A.nrow, k) - yo.reshape(A.nrow, k))
    assert (e <= TOL[dtype] * np.maximum(ya.reshape(A.nrow, k), 1e-300)).all()


def _side_stream():
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    return s


@pytest.mark.gpu
@pytest.mark.parametrize("warm, k", [((16, 4), 20), ((8, 4, 1), 13), ((20,), 20)])
def test_graph_holds_kernels_alone(warm, k):
    rt = pytest.importorskip("cuda.bindings.runtime")
    A = synth.zipf(4000, 1.8, 4000, 0.1, seed=3)
    plan = mb.Plan(*to_cuda(A, "f32"), ncol=A.ncol)
    X, xd, Yd = _operands(A, k, "f32")
    s = _side_stream()
    with torch.cuda.stream(s):
        j = 0
        for w in warm:
            plan.spmm(xd[:, j:j + w], Yd[:, j:j + w])
            j += w
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(g, stream=s):
        plan.spmm(xd, Yd, stream=s)
    raw = rt.cudaGraph_t(g.raw_cuda_graph())
    err, _, n = rt.cudaGraphGetNodes(raw, 0)
    assert int(err) == 0 and n >= 1
    err, nodes, n = rt.cudaGraphGetNodes(raw, n)
    kinds = [rt.cudaGraphNodeGetType(v)[1] for v in nodes]
    assert all(t == rt.cudaGraphNodeType.cudaGraphNodeTypeKernel for t in kinds), kinds
    for _ in range(3):
        Yd.fill_(float("nan"))
        g.replay()
        torch.cuda.synchronize()
        _check(A, "f32", X, Yd)


@pytest.mark.gpu
def test_capture_without_slots_is_refused():
    A = synth.zipf(4000, 1.8, 4000, 0.1, seed=3)
    plan = mb.Plan(*to_cuda(A, "f64"), ncol=A.ncol)
    X, xd, Yd = _operands(A, 8, "f64")
    s = _side_stream()
    g = torch.cuda.CUDAGraph()
    with pytest.raises(mb.MerbitError) as e:
        with torch.cuda.graph(g, stream=s):
            plan.spmm(xd, Yd, stream=s)
    assert e.value.status == 1
    plan.spmm(xd, Yd)
    torch.cuda.synchronize()
    _check(A, "f64", X, Yd)


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", ["f64", "f32"])
@pytest.mark.parametrize("warm, captured", [
    ((12, 12), (8, 8)), ((12, 12), (4, 4)), ((20, 20), (16, 16)), ((40, 40), (8, 8)), ((3, 3), (2, 2)),
    ((17, 20), (1, 1)), ((31, 31), (1, 2)), ((6, 6), (4, 5)), ((6, 6), (2, 3)), ((10, 10), (8, 9)),
    ((8, 10), (8, 9)), ((18, 18), (16, 17)), ((2, 2), (2, 3)), ((32, 34), (32, 33)),
])
def test_capture_of_another_width_with_the_slots_there_are(dtype, warm, captured):
    """A part of what was run before, by other leading dimensions: captured as
    when every power of two of a call had slots of its own.  (k, ld) pairs."""
    A = synth.zipf(4000, 1.8, 4000, 0.1, seed=3)
    plan = mb.Plan(*to_cuda(A, dtype), ncol=A.ncol)
    Xw, xw, Yw = _operands(A, warm[0], dtype, warm[1])
    X, xd, Yd = _operands(A, captured[0], dtype, captured[1])
    s = _side_stream()
    with torch.cuda.stream(s):
        plan.spmm(xw, Yw)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        plan.spmm(xd, Yd, stream=s)
    for _ in range(3):
        Yd.fill_(float("nan"))
        g.replay()
        torch.cuda.synchronize()
        _check(A, dtype, X, Yd)
        plan.spmm(xw, Yw)  # the warm shape in between, on slots it may share
        torch.cuda.synchronize()
        _check(A, dtype, Xw, Yw)


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", ["f64", "f32"])
@pytest.mark.parametrize("k, pad", [(1, 0), (2, 0), (2, 1), (8, 0), (8, 2), (8, 1), (16, 0), (32, 2)])
def test_backward_captured_with_the_slots_of_a_product(dtype, k, pad):
    """The transpose product warms up the fused backward, and the other way round."""
    A = synth.zipf(4000, 1.8, 4000, 0.1, seed=7)
    M = SparseMatrix(*to_cuda(A, dtype), ncol=A.ncol)
    T = M.transpose_plan()
    G, gd, dXd = _operands(A, k, dtype, k + pad, seed=11)
    X, xd, _ = _operands(A, k, dtype, k + pad, seed=12)
    want = O.spmm_t(A.row_ptr, A.col, stored_values(A, dtype), G, A.ncol)
    scale = O.spmm_t(A.row_ptr, A.col, np.abs(stored_values(A, dtype)), np.abs(G), A.ncol)
    s = _side_stream()
    with torch.cuda.stream(s):
        T.spmm(gd, dXd)
        dval_eager = M.dval(gd, xd)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        dX, dval = M.backward_fused(gd, xd)
    for _ in range(3):
        g.replay()
        torch.cuda.synchronize()
        assert (np.abs(dX.cpu().numpy() - want) <= TOL[dtype] * np.maximum(scale, 1e-300)).all()
    rows = np.repeat(np.arange(A.nrow), np.diff(A.row_ptr))
    bound = (k + 2) * np.finfo(XY[dtype]).eps * (np.abs(G.astype(np.float64))[rows] * np.abs(X.astype(np.float64))[A.col]).sum(1)
    assert (np.abs(dval.cpu().numpy().astype(np.float64) - dval_eager.cpu().numpy()) <= bound).all()
    # a fresh matrix: the backward first, the product captured
    M2 = SparseMatrix(*to_cuda(A, dtype), ncol=A.ncol)
    with torch.cuda.stream(s):
        M2.backward_fused(gd, xd)
    torch.cuda.synchronize()
    g2 = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g2, stream=s):
        M2.transpose_plan().spmm(gd, dXd, stream=s)
    for _ in range(3):
        dXd.fill_(float("nan"))
        g2.replay()
        torch.cuda.synchronize()
        assert (np.abs(dXd.cpu().numpy() - want) <= TOL[dtype] * np.maximum(scale, 1e-300)).all()
