"""The allocation-free decode keeps nothing per SNP but its column map: a request of 2,000,000
SNPs, 24 MB of scratch, fits its 32 MiB, and one past the limit is refused."""
from __future__ import annotations

import numpy as np
import pytest

import oracle
from steppecu_b200 import StpError

pytestmark = pytest.mark.gpu


def test_two_million_snps_fit(ctx):
    import torch

    M = 2_000_000
    rec = np.random.default_rng(4).integers(0, 256, (M, 16), dtype=np.uint8)
    d_rec = torch.as_tensor(np.pad(rec, ((0, 0), (0, 32)))).cuda()
    sel, po = np.arange(3, 31, dtype=np.int64), np.array([0, 5, 28], dtype=np.int64)
    ac2, n = (torch.full((2 * M,), -7, dtype=torch.int32, device="cuda") for _ in range(2))
    ctx.decode_counts_noalloc(d_rec, 64, sel, po, ac2, n)
    wa, wn = oracle.decode_counts_pa(rec, sel, po, oracle.detect_ploidy_pa(rec, sel))
    assert np.array_equal(ac2.cpu().numpy(), np.asarray(wa).reshape(-1))
    assert np.array_equal(n.cpu().numpy(), np.asarray(wn).reshape(-1))
    ac2.fill_(-7)
    with pytest.raises(StpError, match="scratch"):
        ctx.decode_counts_noalloc(d_rec, 64, np.arange(56, dtype=np.int64), np.array([0, 20, 56], dtype=np.int64), ac2, n)
    assert bool((ac2 == -7).all())
