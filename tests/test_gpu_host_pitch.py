"""Host records at pitches on both sides of the rule that uploads them in one piece or row by
row (128 bytes between rows, 512 in all, whole words): every entry point that takes them gives
what the tight records give, and rows far apart take no room for the gaps on the device."""
from __future__ import annotations

import subprocess
import sys

import numpy as np
import pytest

from steppecu_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def panel():
    out = []
    for k, n_pop in enumerate((30, 80)):
        p = synth.generate("c4", seed=23 + k, n_snp=6_000, n_pop=n_pop)
        sel, po = p.selection()
        out.append((p, sel, po, np.ascontiguousarray(p.records_numpy()[:, :max(48, (p.n_ind + 3) // 4)])))
    return out


def _all(ctx, p, sel, po, rec):
    a = np.full(p.n_snp, ord("A"), np.uint8)
    req = {"sel_rows": sel, "pop_offsets": po, "block_id": p.block_id, "n_block": p.n_block}
    f2 = np.full(p.n_pop * p.n_pop * p.n_block, np.nan)
    k = p.n_pop * p.n_pop

    def sink(b0, b1, x, v):
        f2[b0 * k:b1 * k] = x

    t = ctx.extract_blocks(rec, p.n_ind, sel, po, p.block_id, p.n_block)
    s = ctx.extract_blocks(rec, p.n_ind, sel, po, p.block_id, p.n_block, precision="fp32")
    b = ctx.extract_batch(rec, p.n_ind, [req, req])[1]
    ctx.extract_streamed(rec, p.n_ind, sel, po, p.block_id, p.n_block, sink)
    return [t.f2, t.vpair, s.f2, b.f2, b.vpair, f2, *ctx.decode_counts(rec, p.n_ind, sel, po),
            ctx.snp_keep_mask(rec, p.n_ind, sel, po, a, a + 2, p.chrom, maf_min=0.1)]


@pytest.mark.parametrize("which,gap", [(0, 1), (0, 400), (0, 499), (1, 127), (1, 129), (1, 131), (1, 400), (1, 1001)])
def test_same_results(ctx, panel, which, gap):
    p, sel, po, rec = panel[which]
    wide = np.full((p.n_snp, rec.shape[1] + gap), 0xA5, np.uint8)
    wide[:, :rec.shape[1]] = rec
    assert all(np.array_equal(x, y) for x, y in zip(_all(ctx, p, sel, po, wide), _all(ctx, p, sel, po, rec)))


def test_gaps_take_no_device_memory():
    code = """
import torch, numpy as np
from steppecu_b200 import Context
M, N = 20_000, 300
rec = np.zeros((M, 100_001), np.uint8)  # 2 GB, of which 75 bytes per row are records
c = Context(0)
sel, po, bid = np.arange(N, dtype=np.int64), np.arange(0, N + 1, 10, dtype=np.int64), np.arange(M, dtype=np.int32) // 500
before = torch.cuda.mem_get_info()[0]
t = c.extract_blocks(rec, N, sel, po, bid, 40)
assert before - torch.cuda.mem_get_info()[0] < 1 << 30
assert t.vpair.min() == 500
print('ok')
"""
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=600)
    assert r.returncode == 0 and r.stdout.strip().endswith("ok"), r.stdout + r.stderr
