"""Kernels that start before the one ahead of them has ended (the transpose over the ploidy
pass, the contraction over the decode, f2 over vpair) and work counters that kernels reset
themselves: passes back to back, of plans of several sizes taking turns on one stream, as
launches and as graphs, equal a pass that is waited for; a pass right after records change
reads the new ploidy and genotypes."""
from __future__ import annotations

import numpy as np
import pytest

from steppecu_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("graph", [False, True])
def test_back_to_back_passes(ctx, graph):
    import torch

    jobs = []
    for k, (n_pop, n_snp) in enumerate([(20, 9_000), (150, 7_000), (64, 3_000), (2, 500)]):
        p = synth.generate("c2", seed=500 + k, n_snp=n_snp, n_pop=n_pop)
        q = synth.generate("c2", seed=900 + k, n_snp=n_snp, n_pop=n_pop)  # other genotypes and ploidy
        sel, po = p.selection()
        buf = p.records.cuda().clone()
        plan = ctx.plan(buf, p.n_ind, sel, po, p.block_id, p.n_block)
        n = n_pop * n_pop * p.n_block
        out = [[torch.zeros(n, dtype=torch.float64, device="cuda") for _ in range(2)] for _ in range(4)]
        jobs.append((plan, buf, p.records.cuda(), q.records.cuda(), out))
    s = torch.cuda.Stream()
    torch.cuda.synchronize()

    def run(job, o):
        (job[0].run_graph if graph else job[0].run)(job[1], *o, stream=s.cuda_stream)

    with torch.cuda.stream(s):
        for job in jobs:  # waited for, one by one
            for which, o in ((2, job[4][0]), (3, job[4][1])):
                job[1].copy_(job[which])
                s.synchronize()
                run(job, o)
                s.synchronize()
        for r in range(6):  # nothing waits
            for job in jobs:
                job[1].copy_(job[2])
                run(job, job[4][2])
                job[1].copy_(job[3])
                run(job, job[4][3])
    torch.cuda.synchronize()
    for job in jobs:
        for a, b in ((0, 2), (1, 3)):
            assert all(torch.equal(x, y) for x, y in zip(job[4][a], job[4][b]))
        assert not torch.equal(job[4][0][0], job[4][1][0])
        job[0].close()
