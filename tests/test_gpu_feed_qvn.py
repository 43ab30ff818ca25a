"""The fixed-point feeder of dense frequencies (64 populations x 32 SNPs per CTA, values
crossing shared memory) against the oracle: populations around a CTA's 64 and a row tile's
128 (stacked and general images), blocks around a column tile, an empty block, populations
without a call whose Q and N hold anything."""
from __future__ import annotations

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu

SIZES = [1, 31, 32, 0, 33, 64, 65, 130]


@pytest.mark.parametrize("P", [1, 8, 63, 64, 65, 127, 128, 131])
def test_feed_matches_oracle(ctx, P):
    import torch

    rng = np.random.default_rng(P)
    M, nb = sum(SIZES), len(SIZES)
    bid = np.repeat(np.arange(nb, dtype=np.int32), SIZES)
    N = rng.integers(1, 40, (M, P)).astype(float)
    Q = rng.integers(0, 2 ** 31, (M, P)) % (N + 1) / N
    V = (rng.random((M, P)) < 0.8).astype(float)
    want_q, want_n = np.where(V > 0, Q, 0.0), np.where(V > 0, N, 0.0)
    f2, vp, _ = oracle.compute_f2_blocks(want_q.reshape(-1), V.reshape(-1), want_n.reshape(-1), P, bid, nb)
    Q[V == 0] = np.nan  # never used
    got = ctx.f2_from_qvn(Q.reshape(-1), V.reshape(-1), N.reshape(-1), P, bid, nb, precision="fixed_i8")
    assert np.array_equal(got.vpair, vp)
    assert np.all(np.abs(got.f2 - f2) <= 1e-6 * np.abs(f2) + 1e-9)  # the fixed point's bound (test_gpu_parity.py)
    d = [torch.as_tensor(x.reshape(-1)).cuda() for x in (Q, V, N)]
    out = tuple(torch.full((P * P * nb,), 3.0, dtype=torch.float64, device="cuda") for _ in range(2))
    ctx.f2_from_qvn(*d, P, bid, nb, precision="fixed_i8", out=out)
    assert np.array_equal(out[0].cpu().numpy(), got.f2) and np.array_equal(out[1].cpu().numpy(), vp)
