"""The keep mask's terms from the shared table (populations of up to 15 samples, enough of them
for the table's size) and on the fly (either side of both lines): the same sums as the oracle, bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("P,largest", [(7, 15), (8, 1), (8, 15), (8, 16), (41, 15), (200, 3),
                                       (17, 15), (18, 15), (9, 10), (10, 10), (4, 5), (5, 5), (2, 1), (3, 1)])
@pytest.mark.parametrize("n_snp", [1, 257, 1000])
def test_pooled_sums_bitexact(ctx, P, largest, n_snp):
    rng = np.random.default_rng(P * 100 + largest + n_snp)
    sizes = rng.integers(1, largest + 1, P)
    sizes[P // 2] = largest
    N = int(sizes.sum())
    rec = rng.integers(0, 256, (n_snp, max(48, (N + 3) // 4)), dtype=np.uint8)
    rec[n_snp // 2] = 0xFF  # nothing called
    sel = rng.permutation(N).astype(np.int64)
    po = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64)
    pl = oracle.detect_ploidy_pa(rec, sel)
    q, _, nd = oracle.counts_to_qvn(*oracle.decode_counts_pa(rec, sel, po, pl))
    ref, alt = np.full(n_snp, ord("A"), np.uint8), np.full(n_snp, ord("C"), np.uint8)
    chrom = np.ones(n_snp, np.int32)
    keep, summ = ctx.snp_keep_mask(rec, N, sel, po, ref, alt, chrom, maf_min=0.3, maxmiss=0.5, summary=True)
    want, wsum = oracle.keep_mask(q, nd, P, ref, alt, chrom, maf_min=0.3, maxmiss=0.5, total_indiv=float(N))
    assert np.array_equal(summ, wsum)
    assert np.array_equal(keep, want.astype(bool))
