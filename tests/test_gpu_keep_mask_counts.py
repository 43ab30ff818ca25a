"""The keep mask's pooled sums from packed counts (eight populations per step, the quotient
from a reciprocal) against the oracle, bit for bit: population counts around the step, a
population far above the table of small counts, SNPs around a CTA."""
from __future__ import annotations

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("P,n_snp,big", [(1, 255, 0), (7, 256, 0), (8, 257, 3000), (9, 300, 0), (17, 40, 16383)])
def test_pooled_sums_bitexact(ctx, P, n_snp, big):
    rng = np.random.default_rng(P * 1000 + n_snp)
    sizes = rng.integers(1, 14, P)
    if big:
        sizes[P // 2] = big
    N = int(sizes.sum())
    rec = rng.integers(0, 256, (n_snp, max(48, (N + 3) // 4)), dtype=np.uint8)
    sel = rng.permutation(N).astype(np.int64)
    po = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64)
    pl = oracle.detect_ploidy_pa(rec, sel)
    q, _, nd = oracle.counts_to_qvn(*oracle.decode_counts_pa(rec, sel, po, pl))
    ref, alt = np.full(n_snp, ord("A"), np.uint8), np.full(n_snp, ord("C"), np.uint8)
    chrom = np.ones(n_snp, np.int32)
    keep, summ = ctx.snp_keep_mask(rec, N, sel, po, ref, alt, chrom, maf_min=0.3, summary=True)
    want, wsum = oracle.keep_mask(q, nd, P, ref, alt, chrom, maf_min=0.3, total_indiv=float(N))
    assert np.array_equal(summ, wsum)
    assert np.array_equal(keep, want.astype(bool))
