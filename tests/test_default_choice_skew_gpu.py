"""The untuned SpMV choice on short but uneven rows: row groups wait for the longest
row of a warp, so skew (longest / mean) times rows decides, per type of x."""
import numpy as np
import pytest
import torch

import merbit_b200 as mb
from merbit_b200 import synth
from oracle import oracle as O
from tests.helpers import stored_values, to_cuda

TOL = {"f64": 1e-13, "f32": 1e-6, "bf16": 1e-6}


def _rows(n, length, longest, ncol=5000):
    """n rows of `length` entries, one of them (in the middle) of `longest`."""
    L = np.full(n, length)
    L[n // 2] = longest
    rp = np.concatenate([[0], np.cumsum(L)]).astype(np.int32)
    rng = np.random.default_rng(n)
    nnz = int(rp[-1])
    return synth.CSR(rp, rng.integers(0, ncol, nnz, dtype=np.int32), rng.standard_normal(nnz), ncol, "rows")


# rows, length, longest; whether FP64 and 4-byte x take row groups
CASES = [
    (90_000, 3, 128, True, True),     # skew x rows 3.8 million
    (120_000, 3, 128, False, False),  # 5.1 million, rows that do not fill 4 lanes
    (150_000, 4, 128, False, True),   # 4.8 million
    (300_000, 4, 128, False, False),  # 9.6 million
    (300_000, 3, 32, True, True),     # a lane per row at any skew
]


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", ["f64", "f32", "bf16"])
@pytest.mark.parametrize("n, length, longest, f64, f32", CASES)
def test_skew_decides(n, length, longest, f64, f32, dtype):
    A = _rows(n, length, longest)
    rp, col, v = to_cuda(A, dtype)
    plan = mb.Plan(rp, col, v, ncol=A.ncol)
    assert (plan.info().kind == 3) == (f64 if dtype == "f64" else f32)
    off = [torch.cat([t[:1], t])[1:] for t in (rp, col, v)]  # not 16-byte aligned
    p2 = mb.Plan(*off, ncol=A.ncol)
    assert p2.info().kind == 3
    x = synth.uniform(3, A.ncol).astype(np.float64 if dtype == "f64" else np.float32)
    yo, ya = O.spmm(A.row_ptr, A.col, stored_values(A, dtype), x)
    for p in (plan, p2):
        y = p.spmv(torch.from_numpy(x).cuda()).cpu().numpy()
        assert (np.abs(y - yo) <= TOL[dtype] * np.maximum(ya, 1e-300)).all()


@pytest.mark.gpu
def test_even_rows_take_row_groups_at_any_size():
    n = 1_900_000
    L = torch.full((n,), 14, dtype=torch.int64, device="cuda")
    L[n // 2] = 34  # skew 2.43
    rp = torch.zeros(n + 1, dtype=torch.int32, device="cuda")
    rp[1:] = torch.cumsum(L, 0)
    nnz = int(rp[-1])
    plan = mb.Plan(rp, torch.zeros(nnz, dtype=torch.int32, device="cuda"),
                   torch.ones(nnz, dtype=torch.float64, device="cuda"))
    assert plan.info().kind == 3
