"""Parts of a fixed-point tile pair that hold nothing to store (past the last population, below
the diagonal) are passed over: every entry of f2 and vpair is written all the same, over blocks
of one and several segments, on buffers that held something else, in a batch as alone."""
from __future__ import annotations

import numpy as np
import pytest

import oracle
from steppecu_b200 import synth

pytestmark = pytest.mark.gpu

SIZES = [1, 0, 31, 33, 16_385, 64, 200]


@pytest.mark.parametrize("P", [65, 72, 73, 97, 128, 129, 136, 161, 257])
def test_every_entry_matches_oracle(ctx, P):
    p = synth.generate("c4", seed=60 + P, n_snp=sum(SIZES), n_pop=P)
    sel, po = p.selection()
    rec = p.records_numpy()
    bid = np.repeat(np.arange(len(SIZES), dtype=np.int32), SIZES)
    f2, vp, _ = oracle.f2_from_panel(rec, sel, po, bid, len(SIZES), oracle.detect_ploidy_pa(rec, sel), threads=16)
    got = ctx.extract_blocks(rec, p.n_ind, sel, po, bid, len(SIZES))
    assert np.array_equal(got.vpair, vp)
    assert np.all(np.abs(got.f2 - f2) <= 1e-6 * np.abs(f2) + 1e-9)
    slabs = got.f2.reshape(len(SIZES), P, P)
    assert np.array_equal(slabs, slabs.transpose(0, 2, 1))


def test_batch_equals_single_requests(ctx):
    p = synth.generate("c4", seed=9, n_snp=30_000, n_pop=300)
    rng = np.random.default_rng(3)
    reqs = []
    for k in (300, 3, 140, 64, 97, 129):
        sel, po = p.selection(np.sort(rng.choice(300, k, replace=False)).tolist())
        reqs.append({"sel_rows": sel, "pop_offsets": po, "block_id": p.block_id, "n_block": p.n_block})
    rec = p.records_numpy()
    for g, q in zip(ctx.extract_batch(rec, p.n_ind, reqs), reqs):
        w = ctx.extract_blocks(rec, p.n_ind, q["sel_rows"], q["pop_offsets"], q["block_id"], q["n_block"])
        assert np.array_equal(g.f2, w.f2) and np.array_equal(g.vpair, w.vpair)
