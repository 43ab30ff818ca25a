"""Both forms of the jackknife (a warp per 32 items, or 16 that share their blocks) on each side
of the rule between them (12 blocks; 250 items per block), with ragged last warps and CTAs,
against the oracle within a few roundings (the tolerances of test_gpu_jackknife_split.py), and
with values that are not finite in one item only."""
from __future__ import annotations

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def _values(m, nb):
    rng = np.random.default_rng(m * 10007 + nb)
    return rng.normal(0.1, 0.01, (nb, m)), rng.integers(50, 4000, nb).astype(np.int32)


@pytest.mark.parametrize("m,nb", [(1, 3), (31, 12), (129, 12), (129, 13), (3249, 13), (3250, 13), (8065, 33), (8250, 33),
                                  (20_000, 80), (20_001, 81), (99_999, 401), (100_000, 401)])
def test_forms_match_oracle(ctx, m, nb):
    x, bs = _values(m, nb)
    est, var = ctx.jackknife(x.reshape(-1), bs, m, nb)
    we, wv = oracle.block_jackknife(x.reshape(-1), bs, m, nb)
    np.testing.assert_allclose(est, we, rtol=1e-13)
    np.testing.assert_allclose(var, wv, rtol=1e-10)


@pytest.mark.parametrize("m,nb", [(200, 5), (200, 40)])
@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
def test_values_that_are_not_finite_stay_in_their_item(ctx, m, nb, bad):
    x, bs = _values(m, nb)
    want = ctx.jackknife(x.reshape(-1), bs, m, nb)
    x[nb // 2, 133] = bad
    got = ctx.jackknife(x.reshape(-1), bs, m, nb)
    keep = np.arange(m) != 133
    for g, w in zip(got, want):
        assert np.array_equal(g[keep], w[keep]) and np.isnan(g[133])
