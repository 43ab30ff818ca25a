"""The stacked kernel's items around one per SM: a CTA's first item is its own number, the
others come from the counter, and the counter is left for the next launch."""
from __future__ import annotations

import numpy as np
import pytest

import oracle
from steppecu_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_block", [1, 2, 147, 148, 149, 296, 700])
def test_every_block_once(ctx, n_block):
    rng = np.random.default_rng(n_block)
    sizes = rng.integers(0, 70, n_block)
    sizes[-1] = 200
    p = synth.generate("c4", seed=n_block, n_snp=int(sizes.sum()), n_pop=9)
    sel, po = p.selection()
    rec = p.records_numpy()
    bid = np.repeat(np.arange(n_block, dtype=np.int32), sizes)
    f2, vp, _ = oracle.f2_from_panel(rec, sel, po, bid, n_block, oracle.detect_ploidy_pa(rec, sel), threads=8)
    for _ in range(2):
        got = ctx.extract_blocks(rec, p.n_ind, sel, po, bid, n_block)
        assert np.array_equal(got.vpair, vp)
        assert np.all(np.abs(got.f2 - f2) <= 1e-6 * np.abs(f2) + 1e-9)
