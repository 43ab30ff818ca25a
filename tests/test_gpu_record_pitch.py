"""The decode reads genotype records of any pitch and base alignment in place (16-byte
granules, with one PRMT per word where rows start off a word): counts and detected ploidy
against the oracle, bit for bit, at the edges of a record slice (1,024 samples) and of a
column quad (128 SNPs), with bytes that no record owns around the buffer."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

import oracle
from steppecu_b200 import _lib as L
from steppecu_b200.api import _i64

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_ind,n_snp,pad,base", [
    (190, 129, 0, 0),     # 48-byte records: 16-byte aligned rows
    (190, 257, 4, 0),     # 52: word aligned
    (209, 128, 0, 0),     # 53: byte aligned
    (1024, 300, 0, 4),    # one whole slice, base 4 bytes off
    (1027, 300, 1, 1),    # 258: a second slice of three samples, base 1 byte off
    (1021, 1100, 2, 3),   # 258: past the ploidy window
    (2050, 140, 0, 15),   # 513
    (4, 40, 0, 7),        # one-byte rows: sixteen share a granule
])
def test_counts_of_any_pitch_and_base(ctx, n_ind, n_snp, pad, base):
    import torch

    rng = np.random.default_rng(n_ind + n_snp + base)
    bpr = (n_ind + 3) // 4
    pitch = bpr + pad
    flat = rng.integers(0, 256, base + pitch * n_snp, dtype=np.uint8)
    rec = np.ascontiguousarray(flat[base:].reshape(n_snp, pitch))
    d = torch.as_tensor(flat).cuda()
    k = max(1, min(n_ind, 700))
    sel = np.sort(rng.choice(n_ind, k, replace=False))
    rng.shuffle(sel)
    P = min(k, 9)
    po = np.concatenate([[0], np.sort(rng.choice(np.arange(1, k), P - 1, replace=False)), [k]]) if P > 1 else np.array([0, k])
    sel, po = _i64(sel), _i64(po)
    v = L.GenoView(int(d.data_ptr()) + base, bpr, pitch, n_snp, n_ind, 1)
    ac2, n = np.zeros(P * n_snp, np.int32), np.zeros(P * n_snp, np.int32)
    L.check(L.lib().stp_decode_counts(ctx._h, C.byref(v), L.ptr(sel), L.ptr(po), P, None, L.PLOIDY_AUTO, L.ptr(ac2), L.ptr(n)))
    pl = oracle.detect_ploidy_pa(rec, sel)
    wa, wn = oracle.decode_counts_pa(rec, sel, po, pl)
    assert np.array_equal(ac2, np.asarray(wa).reshape(-1)) and np.array_equal(n, np.asarray(wn).reshape(-1))
