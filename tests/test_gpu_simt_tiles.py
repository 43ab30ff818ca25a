"""The FP32 contraction's tiles: the smaller side as rows (swapped or not), warps without
populations skipped, integer counts, odd block sizes; against the oracle within the form's
tolerance (test_gpu_parity.py: FP32 sums of 16 SNPs, FP64 across)."""
from __future__ import annotations

import numpy as np
import pytest

import oracle
from steppecu_b200 import synth

pytestmark = pytest.mark.gpu

SIZES = [1, 0, 15, 16, 17, 63, 64, 65, 200]


@pytest.mark.parametrize("P", [1, 8, 9, 63, 64, 65, 72, 100, 127, 129])
def test_simt_matches_oracle(ctx, P):
    p = synth.generate("c4", seed=60 + P, n_snp=sum(SIZES), n_pop=P)
    sel, po = p.selection()
    rec = p.records_numpy()
    bid = np.repeat(np.arange(len(SIZES), dtype=np.int32), SIZES)
    f2, vp, _ = oracle.f2_from_panel(rec, sel, po, bid, len(SIZES), oracle.detect_ploidy_pa(rec, sel), threads=8)
    got = ctx.extract_blocks(rec, p.n_ind, sel, po, bid, len(SIZES), precision="fp32")
    assert np.array_equal(got.vpair, vp)
    assert np.all(np.abs(got.f2 - f2) <= 5e-6 * np.abs(f2) + 5e-8)
