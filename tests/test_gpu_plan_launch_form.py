"""A plan whose launch form cannot be switched stays as it was: the general form's operands of
this one (three million blocks of one SNP, padded to 64 columns each) are 221 GB, more than the
device has, so the switch is refused, and the plan runs and replays as before."""
from __future__ import annotations

import numpy as np
import pytest

from steppecu_b200 import StpError, _lib

pytestmark = pytest.mark.gpu


def test_refused_switch_leaves_the_plan(ctx):
    import torch

    M = 3_000_000
    rec = torch.randint(0, 256, (M, 48), dtype=torch.uint8, device="cuda")
    sel, po = np.arange(2, dtype=np.int64), np.arange(3, dtype=np.int64)
    plan = ctx.plan(rec, 2, sel, po, np.arange(M, dtype=np.int32), M)
    launches = plan.launches

    def outputs(run):
        out = [torch.full((4 * M,), -7.0, dtype=torch.float64, device="cuda") for _ in range(2)]
        torch.cuda.synchronize()
        run(rec, *out)
        torch.cuda.synchronize()
        return out

    want = outputs(plan.run)
    replay = [torch.zeros(4 * M, dtype=torch.float64, device="cuda") for _ in range(2)]
    plan.run_graph(rec, *replay)
    for _ in range(2):
        with pytest.raises(StpError) as e:
            plan.set_per_block_launch(True)
        assert e.value.status == _lib.STP_DEVICE_OOM
        assert plan.launches == launches
        assert all(torch.equal(a, b) for a, b in zip(outputs(plan.run), want))
        for t in replay:
            t.fill_(-7.0)
        torch.cuda.synchronize()
        plan.run_graph(rec, *replay)
        torch.cuda.synchronize()
        assert all(torch.equal(a, b) for a, b in zip(replay, want))
    plan.set_per_block_launch(False)  # what the plan already is
    assert all(torch.equal(a, b) for a, b in zip(outputs(plan.run), want))
    plan.close()
