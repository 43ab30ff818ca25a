"""Records whose pitch is below bytes_per_record (48 for a small panel): refused by every entry
point that takes a genotype view when the rows do not hold all samples in whole words, and read
right where plans, counts and the keep mask take them, from host and device."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

import oracle
from steppecu_b200 import _lib as L
from steppecu_b200 import StpError

pytestmark = pytest.mark.gpu

N, M, BPR = 100, 700, 48  # 25 bytes of codes
SEL, PO = np.arange(N, dtype=np.int64), np.array([0, 40, 73, 100], dtype=np.int64)
BID = (np.arange(M) // 50).astype(np.int32)
NB = int(BID[-1]) + 1


def _view(pitch, on_device):
    import torch

    rng = np.random.default_rng(pitch)
    # A host view may end right after its last row's pitch bytes.
    rec = rng.integers(0, 256, (M, pitch), dtype=np.uint8)
    keep = torch.as_tensor(rec).cuda() if on_device else rec
    return rec, L.GenoView(int(keep.data_ptr()) if on_device else keep.ctypes.data, BPR, pitch, M, N, int(on_device)), keep


def _counts(ctx, v):
    ac2, n = np.zeros(3 * M, np.int32), np.zeros(3 * M, np.int32)
    L.check(L.lib().stp_decode_counts(ctx._h, C.byref(v), L.ptr(SEL), L.ptr(PO), 3, None, L.PLOIDY_AUTO, L.ptr(ac2), L.ptr(n)))
    return ac2, n


def _keep(ctx, v):
    a, chrom = np.full(M, 65, np.uint8), np.ones(M, np.int32)
    c, k, nk, summ = a + 2, np.zeros(M, np.uint8), C.c_int64(0), np.zeros(4 * M)
    f = L.SnpFilter(0.05, 0.5, 0, 0, 0, L.STRAND_KEEP)
    L.check(L.lib().stp_snp_keep_mask(ctx._h, C.byref(v), L.ptr(SEL), L.ptr(PO), 3, None, L.PLOIDY_AUTO, L.ptr(a),
                                      L.ptr(c), L.ptr(chrom), C.byref(f), L.ptr(k), C.byref(nk), L.ptr(summ)))
    return k, summ


def _plan(ctx, v):
    st = C.c_int(0)
    r = L.F2Request(v, L.ptr(SEL), L.ptr(PO), 3, None, L.PLOIDY_AUTO, L.ptr(BID), NB, L.PREC_FIXED_I8, None, 0)
    h = L.lib().stp_plan_create(ctx._h, C.byref(r), C.byref(st))
    L.check(st.value)
    return h


@pytest.mark.parametrize("pitch", [4, 20, 24, 25, 26, 27, 30])
def test_refused(ctx, pitch):
    for on_device in (False, True):
        _, v, keep = _view(pitch, on_device)
        calls = [_counts, _keep] + ([_plan] if on_device else [])
        for f in calls:
            with pytest.raises(StpError, match="pitch < bytes_per_record") as e:
                f(ctx, v)
            assert e.value.status == L.STP_INVALID_ARGUMENT


@pytest.mark.parametrize("pitch", [28, 44, 48, 49])
def test_read_right(ctx, pitch):
    import torch

    outs = []
    for on_device in (False, True):
        rec, v, keep = _view(pitch, on_device)
        pl = oracle.detect_ploidy_pa(rec, SEL)
        wa, wn = oracle.decode_counts_pa(rec, SEL, PO, pl)
        ac2, n = _counts(ctx, v)
        assert np.array_equal(ac2, np.asarray(wa).reshape(-1)) and np.array_equal(n, np.asarray(wn).reshape(-1))
        outs.append(_keep(ctx, v))
    assert all(np.array_equal(a, b) for a, b in zip(*outs))
    h = _plan(ctx, v)
    f2, vp = (torch.zeros(9 * NB, dtype=torch.float64, device="cuda") for _ in range(2))
    L.check(L.lib().stp_plan_run(h, int(keep.data_ptr()), int(f2.data_ptr()), int(vp.data_ptr()), None))
    torch.cuda.synchronize()
    L.lib().stp_plan_destroy(h)
    wf, wv, _ = oracle.f2_from_panel(rec, SEL, PO, BID, NB, pl)
    assert np.array_equal(vp.cpu().numpy(), wv)
    assert np.all(np.abs(f2.cpu().numpy() - wf) <= 1e-6 * np.abs(wf) + 1e-9)  # the fixed point's bound, test_gpu_fx.py
