"""Split-precision tile pairs with few rows or columns: valid 8-row groups copied alone, MMA
columns rounded up to 16, epilogue warps without populations skipped; against the oracle
within each form's bound, counts exactly, alone and in a batch whose requests leave the
shared-memory slots in other shapes."""
from __future__ import annotations

import numpy as np
import pytest

import oracle
from steppecu_b200 import synth

pytestmark = pytest.mark.gpu

SIZES = [1, 0, 31, 32, 33, 63, 64, 65, 200]
# A block mean's worst error, which a one-SNP block can reach. With the unit roundoff u of the
# 16-bit type, a term split into hi + lo keeps u^2 of itself: T = 2 (A_i + A_j - x_i x_j) with
# |A| <= 1/2 and |x| <= 1 loses 2 u^2 (1/2 + 1/2 + 2) to the splits and 2 u^2 to the lo * lo
# product left out: 8 u^2. The FP32 sums add one rounding of 2^-23 of the partial sum per MMA,
# 28 MMAs per 64-SNP chunk.
ROUNDOFF = {"split_f16": 2.0**-12, "split_f16_fine": 2.0**-12, "split_bf16": 2.0**-9}
BOUND = {mode: 8 * u * u + 28 * 2.0**-23 for mode, u in ROUNDOFF.items()}


@pytest.mark.parametrize("mode", list(BOUND))
@pytest.mark.parametrize("P", [1, 8, 9, 31, 33, 64, 65, 72, 97, 120, 121, 128, 129, 150, 192, 233, 300])
def test_split_tiles_match_oracle(ctx, mode, P):
    p = synth.generate("c4", seed=40 + P, n_snp=sum(SIZES), n_pop=P)
    sel, po = p.selection()
    rec = p.records_numpy()
    bid = np.repeat(np.arange(len(SIZES), dtype=np.int32), SIZES)
    f2, vp, _ = oracle.f2_from_panel(rec, sel, po, bid, len(SIZES), oracle.detect_ploidy_pa(rec, sel), threads=8)
    got = ctx.extract_blocks(rec, p.n_ind, sel, po, bid, len(SIZES), precision=mode)
    assert np.array_equal(got.vpair, vp)
    assert np.abs(got.f2 - f2).max() <= BOUND[mode]


def test_batch_equals_single_requests(ctx):
    p = synth.generate("c4", seed=8, n_snp=5_000, n_pop=300)
    rng = np.random.default_rng(2)
    reqs = []
    for k in (300, 3, 140, 64, 17, 129):
        sel, po = p.selection(np.sort(rng.choice(300, k, replace=False)).tolist())
        reqs.append({"sel_rows": sel, "pop_offsets": po, "block_id": p.block_id, "n_block": p.n_block})
    rec = p.records_numpy()
    for g, q in zip(ctx.extract_batch(rec, p.n_ind, reqs, precision="split_f16"), reqs):
        w = ctx.extract_blocks(rec, p.n_ind, q["sel_rows"], q["pop_offsets"], q["block_id"], q["n_block"], precision="split_f16")
        assert np.array_equal(g.f2, w.f2) and np.array_equal(g.vpair, w.vpair)
