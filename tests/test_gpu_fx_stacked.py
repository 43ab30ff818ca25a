"""The stacked fixed-point contraction (up to 64 populations, f2_fxs.cu) against the general
kernels, bit for bit, and against the oracle.

Both form the same integers from the same digits, so f2 and vpair agree exactly while a
block is one accumulation in each (16,384 SNPs in the general kernel). Longer blocks are
summed in FP64 per segment by the general one only: there the oracle is the reference,
within the fixed point's bound (relative 1e-6 with a floor of 1e-9, see test_gpu_parity.py).
The general kernels run as a plan's per-block comparison form."""
from __future__ import annotations

import dataclasses

import numpy as np
import pytest

import oracle
from steppecu_b200 import synth

pytestmark = pytest.mark.gpu

# SNPs per block: an empty block, the edges of a chunk of 32, of a copy of 128 / R chunks.
SIZES = [1, 0, 31, 32, 33, 64, 65, 511, 512, 513, 1500, 2]


def _plan_out(ctx, plan, rec, n):
    import torch

    out = [torch.full((n,), 3.0, dtype=torch.float64, device="cuda") for _ in range(2)]
    plan.run(rec, *out)
    torch.cuda.synchronize()
    return out


@pytest.mark.parametrize("P", [1, 2, 7, 8, 9, 16, 17, 24, 31, 32, 33, 40, 41, 56, 63, 64])
def test_stacked_equals_general(ctx, P):
    import torch

    p = synth.generate("c4", seed=900 + P, n_snp=sum(SIZES), n_pop=P)
    sel, po = p.selection()
    bid = np.repeat(np.arange(len(SIZES), dtype=np.int32), SIZES)
    rec = p.records.cuda()
    plan = ctx.plan(rec, p.n_ind, sel, po, bid, len(SIZES), precision="fixed_i8")
    n = P * P * len(SIZES)
    a = _plan_out(ctx, plan, rec, n)
    plan.set_per_block_launch(True)
    b = _plan_out(ctx, plan, rec, n)
    plan.set_per_block_launch(False)
    c = _plan_out(ctx, plan, rec, n)
    plan.close()
    for k in range(2):
        assert torch.equal(a[k], b[k]) and torch.equal(a[k], c[k])


@pytest.mark.parametrize("P", [5, 40])
def test_blocks_of_several_segments(ctx, P):
    """One SNP past two accumulator segments (131,040 SNPs each), then a short block."""
    wl = dataclasses.replace(synth.WORKLOADS["c2"], ind_per_pop=2)
    M = 262_081 + 40
    p = synth.generate(wl, seed=77 + P, n_snp=M, n_pop=P)
    sel, po = p.selection()
    rec = p.records_numpy()
    bid = (np.arange(M) >= 262_081).astype(np.int32)
    pl = oracle.detect_ploidy_pa(rec, sel)
    f2, vp, _ = oracle.f2_from_panel(rec, sel, po, bid, 2, pl, threads=8)
    got = ctx.extract_blocks(rec, p.n_ind, sel, po, bid, 2, precision="fixed_i8")
    assert np.array_equal(got.vpair, vp)
    assert np.all(np.abs(got.f2 - f2) <= 1e-6 * np.abs(f2) + 1e-9)


def test_mixed_batch_equals_single_requests(ctx):
    """A batch whose requests lie on both sides of the 64 populations, and on both sides of
    the 32 up to which two accumulators alternate."""
    p = synth.generate("c4", seed=41, n_snp=9_000, n_pop=140)
    rng = np.random.default_rng(5)
    reqs = []
    for k in (3, 130, 64, 65, 20, 33, 32, 2):
        sel, po = p.selection(np.sort(rng.choice(140, k, replace=False)).tolist())
        reqs.append({"sel_rows": sel, "pop_offsets": po, "block_id": p.block_id, "n_block": p.n_block})
    rec = p.records_numpy()
    got = ctx.extract_batch(rec, p.n_ind, reqs, precision="fixed_i8")
    for g, q in zip(got, reqs):
        w = ctx.extract_blocks(rec, p.n_ind, q["sel_rows"], q["pop_offsets"], q["block_id"], q["n_block"], precision="fixed_i8")
        assert np.array_equal(g.f2, w.f2) and np.array_equal(g.vpair, w.vpair)
