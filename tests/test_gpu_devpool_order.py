"""The device block store keeps what was released last: calls of other sizes that came before
make room, and the memory held stays bounded."""
from __future__ import annotations

import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu


def test_old_blocks_make_room():
    code = """
import torch, numpy as np
from steppecu_b200 import Context
Context(0).close()
torch.cuda.synchronize()
before = torch.cuda.mem_get_info()[0]
c = Context(0)
P, held = 300, []
sel, po = np.arange(P, dtype=np.int64), np.arange(P + 1, dtype=np.int64)
# Counts of 1.8, 1.3 and 1.0 GB, no block fit for another: more than the store holds.
for M in (1_500_000, 1_100_000, 850_000, 850_000):
    a = np.full(M, ord('A'), np.uint8)
    keep = c.snp_keep_mask(np.zeros((M, 75), np.uint8), P, sel, po, a, a + 2, np.ones(M, np.int32), maf_min=0.1)
    assert keep.shape == (M,) and not keep.any()
    held.append(before - torch.cuda.mem_get_info()[0])
assert max(held) < 4.6e9, held
assert held[2] < held[1], held   # the first call's counts made room for the third's
assert abs(held[3] - held[2]) < 64 << 20, held  # which the fourth call took again
c.close()
assert before - torch.cuda.mem_get_info()[0] < 64 << 20
print('ok')
"""
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=600)
    assert r.returncode == 0 and r.stdout.strip().endswith("ok"), r.stdout + r.stderr
