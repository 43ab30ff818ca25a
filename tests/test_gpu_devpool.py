"""Released device blocks are kept per device and handed out again: calls of several sizes in
several threads (a context each) give what a single thread gives, and the last context
returns every block to the device."""
from __future__ import annotations

import subprocess
import sys
import threading

import numpy as np
import pytest

from steppecu_b200 import Context, synth

pytestmark = pytest.mark.gpu


def _panels():
    out = []
    for k, (n_pop, n_snp) in enumerate([(5, 4_000), (40, 9_000), (17, 2_000)]):
        p = synth.generate("c1", seed=70 + k, n_snp=n_snp, n_pop=n_pop)
        out.append((p, *p.selection(), p.records_numpy()))
    return out


def _call(c, p, sel, po, rec):
    a = np.full(p.n_snp, ord("A"), np.uint8)
    keep = c.snp_keep_mask(rec, p.n_ind, sel, po, a, np.full_like(a, ord("C")), p.chrom, maf_min=0.1)
    t = c.extract_blocks(rec, p.n_ind, sel, po, p.block_id, p.n_block)
    return keep, t.f2, t.vpair


def test_threads_share_the_store(ctx):
    panels = _panels()
    want = [_call(ctx, *x) for x in panels]
    bad = []

    def work(k):
        with Context(0) as c:
            for r in range(12):
                i = (k + r) % len(panels)
                if not all(np.array_equal(g, w) for g, w in zip(_call(c, *panels[i]), want[i])):
                    bad.append((k, r))

    th = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in th:
        t.start()
    for t in th:
        t.join()
    assert not bad


def test_the_last_context_returns_the_memory():
    code = """
import torch, numpy as np
from steppecu_b200 import Context, synth
Context(0).close()  # the library's own module memory
torch.cuda.synchronize()
before = torch.cuda.mem_get_info()[0]
p = synth.generate("c1", seed=3, n_snp=30000, n_pop=40)
sel, po = p.selection()
c = Context(0)
for n in (40, 20, 40):
    c.decode_counts(p.records_numpy(), p.n_ind, sel[:po[n]], po[:n + 1])
c.close()
after = torch.cuda.mem_get_info()[0]
assert before - after < (64 << 20), (before, after)
"""
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
