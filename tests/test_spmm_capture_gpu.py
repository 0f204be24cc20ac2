"""SpMM while its stream is being captured: what a plan holds decides what runs,
and nothing but the products' kernels enters the caller's graph.

Tolerances as for every SpMM test (component-wise against the
extended-precision oracle): 1e-13 for f64, 1e-6 for f32 values."""
import numpy as np
import pytest
import torch

import merbit_b200 as mb
from merbit_b200 import synth
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
