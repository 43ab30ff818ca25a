"""Device records are read where they lie on every call: a request repeated with records one
byte further on takes the plan of the first call, a plan runs on records of any base, and the
streamed extraction takes device records of an odd pitch and base, all bit for bit what host
records give."""
from __future__ import annotations

import numpy as np
import pytest

from steppecu_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def panel():
    p = synth.generate("c4", seed=19, n_snp=9_000, n_pop=70)
    sel, po = p.selection()
    return p, sel, po, np.ascontiguousarray(p.records_numpy()[:, :(p.n_ind + 3) // 4])


def _device(rec, base, pad=0):
    """The records with `pad` bytes after each row, `base` bytes off an aligned address."""
    import torch

    m, w = rec.shape
    flat = torch.full((base + m * (w + pad),), 0xA5, dtype=torch.uint8, device="cuda")
    v = flat[base:].view(m, w + pad)
    v[:, :w] = torch.as_tensor(rec).cuda()
    assert v.data_ptr() % 16 == base % 16
    return v


@pytest.mark.parametrize("mode", ["fixed_i8", "split_f16", "fp32"])
def test_equal_requests_at_other_bases(ctx, panel, mode):
    p, sel, po, rec = panel
    pad = -rec.shape[1] % 4  # whole words, so that only the base is off
    want = ctx.extract_blocks(rec, p.n_ind, sel, po, p.block_id, p.n_block, precision=mode)
    for base in (0, 1, 0, 4, 3):
        got = ctx.extract_blocks(_device(rec, base, pad), p.n_ind, sel, po, p.block_id, p.n_block, precision=mode)
        assert np.array_equal(got.f2, want.f2) and np.array_equal(got.vpair, want.vpair)


def test_plan_runs_on_any_base(ctx, panel):
    import torch

    p, sel, po, rec = panel
    pad = -rec.shape[1] % 4
    n = p.n_pop * p.n_pop * p.n_block
    recs = [_device(rec, base, pad) for base in (0, 1, 6)]
    outs = []
    plan = ctx.plan(recs[0], p.n_ind, sel, po, p.block_id, p.n_block)
    for r in recs:
        for run in (plan.run, plan.run_graph):
            out = [torch.full((n,), -7.0, dtype=torch.float64, device="cuda") for _ in range(2)]
            torch.cuda.synchronize()
            run(r, *out)
            torch.cuda.synchronize()
            outs.append(out)
    plan.close()
    assert all(torch.equal(a, b) for o in outs[1:] for a, b in zip(o, outs[0]))


@pytest.mark.parametrize("base,pad", [(0, 1), (1, 0), (3, 2)])
def test_streamed_device_records(ctx, panel, base, pad):
    p, sel, po, rec = panel
    want = ctx.extract_blocks(rec, p.n_ind, sel, po, p.block_id, p.n_block)
    f2, vp = np.full_like(want.f2, np.nan), np.full_like(want.vpair, np.nan)
    k = p.n_pop * p.n_pop

    def sink(b0, b1, a, v):
        f2[b0 * k:b1 * k], vp[b0 * k:b1 * k] = a, v

    ctx.extract_streamed(_device(rec, base, pad), p.n_ind, sel, po, p.block_id, p.n_block, sink)
    assert np.array_equal(f2, want.f2) and np.array_equal(vp, want.vpair)
