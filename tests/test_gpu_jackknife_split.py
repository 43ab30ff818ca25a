"""The jackknife splits an item's blocks over the warps of a CTA: sums of compensated partial
sums against the oracle, at the edges of the split (1 to a few rounds of blocks per warp, one
item to a ragged last CTA). Every sum is compensated, so both sides are within a few
roundings of each result: 1e-13 relative on the estimate; the variance squares differences of
leave-one-out values around 1e-3 of the value, so it keeps 1e-10."""
from __future__ import annotations

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,nb", [(1, 2), (31, 15), (33, 16), (32, 17), (5, 511), (70, 513), (3, 1025)])
def test_jackknife_split(ctx, m, nb):
    rng = np.random.default_rng(m * 10007 + nb)
    x = rng.normal(0.1, 0.01, (nb, m))
    bs = rng.integers(50, 4000, nb).astype(np.int32)
    est, var = ctx.jackknife(x.reshape(-1), bs, m, nb)
    we, wv = oracle.block_jackknife(x.reshape(-1), bs, m, nb)
    np.testing.assert_allclose(est, we, rtol=1e-13)
    np.testing.assert_allclose(var, wv, rtol=1e-10)
