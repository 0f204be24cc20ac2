"""merbit_coo_sort: indices of few bits (one packed word per triplet) and of so
many that words do not hold them (separate keys), equal keys in their original
order, negative indices ordered as unsigned ones."""
import numpy as np
import pytest
import torch

import merbit_b200 as mb


def _bounds():
    return [(1, 1), (1, 700), (700, 1), (250_007, 250_007), (3, 2**31 - 1), (2**31 - 1, 5),
            (2**31 - 1, 2**31 - 1), (-5, 40), (40, -5)]


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 2, 3, 1000, 65_537])
@pytest.mark.parametrize("hi_major,hi_minor", _bounds())
@pytest.mark.parametrize("dtype", [None, torch.float64, torch.float32, torch.bfloat16])
def test_coo_sort_is_the_stable_order_of_unsigned_indices(n, hi_major, hi_minor, dtype):
    rng = np.random.default_rng(n)

    def draw(hi):
        lo, hi = (hi, -hi) if hi < 0 else (0, hi)
        return rng.integers(lo, hi, n, dtype=np.int64).astype(np.int32)

    major, minor = draw(hi_major), draw(hi_minor)
    if n > 2:  # both ends of the range, and equal triplets
        major[0] = hi_major - 1 if hi_major > 0 else hi_major
        minor[-1] = hi_minor - 1 if hi_minor > 0 else hi_minor
        major[1], minor[1] = major[-1], minor[-1]
    order = np.lexsort((minor.view(np.uint32), major.view(np.uint32)))
    vals = torch.arange(n, device="cuda").to(dtype) if dtype is not None else None
    dM, dm = torch.from_numpy(major).cuda(), torch.from_numpy(minor).cuda()
    want = None if vals is None else vals[torch.from_numpy(order).cuda()].clone()
    mb.coo_sort(dM, dm, vals)
    assert np.array_equal(dM.cpu().numpy(), major[order])
    assert np.array_equal(dm.cpu().numpy(), minor[order])
    if vals is not None:
        assert torch.equal(vals, want)
