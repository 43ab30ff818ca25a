"""The general fixed-point kernels (more than 64 populations) where tests of few populations
reach the stacked one: a wait that runs out in the f2 kernel, a block whose counts take two
accumulations of the vpair kernel, and the tile classes of a last tile of few populations."""
from __future__ import annotations

import dataclasses

import numpy as np
import pytest

import oracle
from steppecu_b200 import Context, StpError, synth

pytestmark = pytest.mark.gpu

RTOL, ATOL = 1e-6, 1e-9  # the fixed point's bound, as in test_gpu_fx.py


@pytest.mark.parametrize("P,stage", [(65, 0), (130, 2), (300, 30)])
def test_wait_timeout_reports_and_context_recovers(P, stage):
    """The feed of every CTA stops before its stage of this index (the first, one with two stages
    of copies and MMAs before it, one deep in a block): the call ends with STP_DEVICE_TIMEOUT, the
    kernel gives its tensor memory back, and the same context then extracts correctly."""
    p = synth.generate("c1", seed=11 + P, n_snp=3000 if stage < 30 else 60_000, n_pop=P)
    sel, po = p.selection()
    rec = p.records_numpy()
    with Context(0) as c:
        want = c.extract_blocks(rec, p.n_ind, sel, po, p.block_id, p.n_block)
        for _ in range(2):
            c.set_wait_bounds(timeout_ns=50_000_000, withhold_stage=stage)
            with pytest.raises(StpError, match="device_timeout"):
                c.extract_blocks(rec, p.n_ind, sel, po, p.block_id, p.n_block)
            c.set_wait_bounds()
            got = c.extract_blocks(rec, p.n_ind, sel, po, p.block_id, p.n_block)
            assert np.array_equal(got.f2, want.f2) and np.array_equal(got.vpair, want.vpair)


def _f2_fp64(rec, sel, po, bid, nb):
    """f2 and vpair of whole blocks as FP64 matrix products of the oracle's q, v, n (f2_estimator.hpp:38-46):
    sums of 530,000 terms of order 1, so within 1e-10 of the exact ones."""
    pl = oracle.detect_ploidy_pa(rec, sel)
    P, M = len(po) - 1, rec.shape[0]
    q, v, n = (a.reshape(M, P) for a in oracle.counts_to_qvn(*oracle.decode_counts_pa(rec, sel, po, pl)))
    a = (q * q - q * (1.0 - q) / np.maximum(n - 1.0, 1.0)) * v
    p = q * v
    f2, vp = np.zeros((nb, P, P)), np.zeros((nb, P, P))
    for b in range(nb):
        k = bid == b
        av = a[k].T @ v[k]
        vp[b] = v[k].T @ v[k]
        f2[b] = np.divide(av + av.T - 2.0 * (p[k].T @ p[k]), vp[b], out=np.zeros((P, P)), where=vp[b] > 0)
    return f2.reshape(-1), vp.reshape(-1)


@pytest.mark.parametrize("P", [65, 130, 257])
def test_block_longer_than_one_count_accumulation(ctx, P):
    """530,000 SNPs: the vpair kernel's accumulator holds 524,032, so the counts are added to the
    first part's, in single units, in both halves of paired ones and where parts of a tile
    hold nothing; a short block follows."""
    wl = dataclasses.replace(synth.WORKLOADS["c2"], ind_per_pop=1)
    p = synth.generate(wl, seed=21 + P, n_snp=531_000, n_pop=P)
    sel, po = p.selection()
    rec = p.records_numpy()
    for row in (sel[0], sel[P // 2], sel[P - 1]):  # called everywhere: pairs past one accumulation
        rec[:, row // 4] &= np.uint8(0xFF ^ (1 << (6 - 2 * (row % 4))))
    bid = (np.arange(p.n_snp) >= 530_000).astype(np.int32)
    f2, vp = _f2_fp64(rec, sel, po, bid, 2)
    assert vp.max() > 524_032
    got = ctx.extract_blocks(rec, p.n_ind, sel, po, bid, 2)
    assert np.array_equal(got.vpair, vp)
    assert np.all(np.abs(got.f2 - f2) <= ATOL + RTOL * np.abs(f2))


@pytest.mark.parametrize("P", [66, 169, 297])
def test_tile_classes_do_not_change_results(ctx, P):
    """Last tiles of 66, 41 and 41 populations: copied whole or by their valid rows, the same
    f2 and vpair, bit for bit."""
    p = synth.generate("c4", seed=300 + P, n_snp=20_000, n_pop=P)
    sel, po = p.selection()
    rec = p.records_numpy()
    outs = []
    with Context(0) as c:
        for mask in (0, 0xFFFF, 0x5555, 0xAAAA):
            c.set_tile_classes(mask)
            outs.append(c.extract_blocks(rec, p.n_ind, sel, po, p.block_id, p.n_block))
    for t in outs[1:]:
        assert np.array_equal(t.f2, outs[0].f2) and np.array_equal(t.vpair, outs[0].vpair)
