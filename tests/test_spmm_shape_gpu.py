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
