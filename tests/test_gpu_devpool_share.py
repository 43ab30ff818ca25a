"""The device block store leaves a device with little free memory to others: after calls whose
buffers are a good part of it, at most a sixteenth of it stays with the library, an allocation
of the rest by another allocator succeeds, and the calls work all the same."""
from __future__ import annotations

import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu


def test_a_small_share_stays():
    code = """
import torch, numpy as np
from steppecu_b200 import Context
Context(0).close()
torch.cuda.synchronize()
left = 6 << 30
fill = torch.empty(torch.cuda.mem_get_info()[0] - left, dtype=torch.uint8, device='cuda')
before = torch.cuda.mem_get_info()[0]
assert before < left + (64 << 20)
c = Context(0)
P = 300
sel, po = np.arange(P, dtype=np.int64), np.arange(P + 1, dtype=np.int64)
# Counts of 1.0, 1.8 and 0.4 GB.
for M in (850_000, 1_500_000, 350_000, 1_500_000):
    a = np.full(M, ord('A'), np.uint8)
    keep = c.snp_keep_mask(np.zeros((M, 75), np.uint8), P, sel, po, a, a + 2, np.ones(M, np.int32), maf_min=0.1)
    assert keep.shape == (M,) and not keep.any()
    kept = before - torch.cuda.mem_get_info()[0]
    assert kept < before // 16 + (64 << 20), kept
rest = torch.empty(before - before // 16 - (128 << 20), dtype=torch.uint8, device='cuda')
c.close()
print('ok')
"""
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=600)
    assert r.returncode == 0 and r.stdout.strip().endswith("ok"), r.stdout + r.stderr
