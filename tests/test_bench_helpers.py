"""The bench line's arithmetic, on CPU: the metric's units, the issued tensor work of the
split contraction counted from its MMA schedule, and the bytes the host-output extraction
downloads (upper tiles: f2 in FP64, vpair as packed counts)."""
from __future__ import annotations

import importlib.util
from pathlib import Path

import numpy as np
import pytest

ROOT = Path(__file__).resolve().parents[1]
_spec = importlib.util.spec_from_file_location("bench_module", ROOT / "bench.py")
bench = importlib.util.module_from_spec(_spec)
_spec.loader.exec_module(bench)


def test_units_count_unordered_pairs():
    assert bench.units(1000, 1_150_000) == 1_150_000 * 1000 * 999 / 2
    assert bench.units(1, 10) == 0


@pytest.mark.parametrize("P", [100, 128, 129, 1000])
def test_issued_work_matches_mma_count(P):
    sizes = np.array([1, 31, 32, 33, 1600, 0, 6000])
    bid = np.repeat(np.arange(sizes.size), sizes)
    w = bench.issued_tensor_work(P, bid, sizes.size, con_ms=1.0, peak=1000.0)
    rt = -(-P // 128)
    pairs = rt * (rt + 1) // 2
    stages = sum(-(-int(k) // 32) for k in sizes)
    # per stage of a tile pair: 14 f16 MMAs of 128x128x16 and one i8 MMA of 128x128x32
    assert w["f16_flops"] == pairs * stages * 14 * 2 * 128 * 128 * 16
    assert w["i8_ops"] == pairs * stages * 2 * 128 * 128 * 32
    assert w["f16_tflops"] == pytest.approx(w["f16_flops"] / 1e-3 / 1e12)


@pytest.mark.parametrize("P", [1, 5, 128, 129, 300, 1000])
def test_host_d2h_bytes_match_the_copies(P):
    B = 3
    upper = np.zeros((P, P), bool)  # [row i, column j]: the packed upper tiles
    for r0 in range(0, P, 128):
        upper[r0:r0 + 128, r0:P] = True
    assert np.all(upper | upper.T)  # the tiles and their transposes cover every element
    t = -(-P // 128)
    packed = t * (t + 1) // 2 * 128 * 128  # counts per slab, with each tile padded to 128 x 128
    assert packed >= int(upper.sum())
    assert bench.host_d2h_bytes(P, B) == B * (8 * int(upper.sum()) + 2 * packed)
    assert bench.host_d2h_bytes(P, B, wide=True) == B * (8 * int(upper.sum()) + 4 * packed)


def test_the_printed_line_is_short_and_keeps_its_keys():
    modes = ("fixed_i8", "split_f16", "split_f16_fine", "split_bf16", "fp32")
    x = 1.0 / 3.0
    prec = {m: {"max_abs": x, "max_rel": x, "max_rel_f2_ge_0.01": x, "max_comb": x, "vpair_bit_exact": True,
                "per_block": {"max_abs": [x] * 16}} for m in modes}
    cpu = {"value": x * 1e9, "unit": bench.UNIT, "cores": 16, "kind": "port", "sample": "s" * 200}
    line = {
        "metric": bench.METRIC, "value": x * 1e14, "unit": bench.UNIT, "n_gpus": 1, "steps": 20, "warmup": 5, "ms_per_step": 40 * x,
        "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "i8x4 (int32 exact)", "data": "synthetic",
        "config": {"workload": "c3", "populations": 1000, "samples": 10000, "snps": 1150000, "blocks": 714, "block_snps": "5 cM walk",
                   "precision": "fixed_i8", "l2": "inputs larger than L2 (no flush)", "cuda_graph": True, "parallelism": "1 GPU"},
        "gpu_launches": 100, "value_ordered_pairs": {"value": x * 2e14, "unit": "u" * 40},
        "clocks": {"sm_mhz": 1770.0, "sm_max_mhz": 1965.0, "reasons": ["sw_power_cap"]},
        "e2e": {"value": x * 1e13, "unit": bench.UNIT, "h2d_bytes_per_step": 1, "d2h_bytes_per_step": 2, "output_bytes_per_step": 3,
                "ms_per_step": 300 * x, "steps": 5},
        "roofline": {"bound": "tensor", "achieved": x * 2000, "peak": 1659.5, "unit": "TFLOP/s", "frac": x, "traffic": 1e10,
                     "peak_source": "measured", "kernel_ms": x, "decode_ms": x, "decode_hbm_gbs": x, "issued": {"i8_ops": x}},
        "cpu_baseline": {**cpu, "single_core": cpu}, "precision": {"against": "port CPU f2 on the cpu_baseline sample", **prec},
        "precision_all_blocks": {"pairs": "p" * 60, "blocks": 714, "oracle": "o" * 80, "max_abs": x, "max_comb_1e-9": x,
                                 "tolerance": {"rtol": 1e-6, "atol": 1e-9, "violations": 0}, "vpair_bit_exact": True,
                                 "precision": "fixed_i8", "per_block_max_abs": [x] * 714, "per_block_max_rel": [x] * 714},
        "other_arithmetics": {m: {"value": x, "ms_per_step": x, "contract_ms": x, "decode_ms": x} for m in modes[1:]},
        "per_block_launches": {"ms_per_step": x}, "fstats": {"ms": x, "cpu_baseline": cpu},
        "batched_requests": {"grouped": {"value": x, "ms_per_call": x, "device_span_ms": x, "equals_serial": True}},
        "other_configs": {c: {"populations": 5, **{m: {"ms_per_step": x, "value": x} for m in modes[:3]}, "cpu_baseline": cpu,
                              "precision": prec} for c in ("c2", "c4")},
    }
    short = bench.headline(line)
    assert len(bench.json.dumps(short)) < 2500
    for k in ("metric", "value", "unit", "n_gpus", "steps", "warmup", "ms_per_step", "higher_is_better", "scaling", "vs_baseline",
              "dtype", "data", "config", "clocks", "e2e", "gpu_launches", "roofline", "cpu_baseline"):
        assert k in short
    assert short["value"] == pytest.approx(line["value"], rel=1e-5) and short["config"] == line["config"]
    assert short["other_configs_ms"]["c4"]["split_f16"] == pytest.approx(x, rel=1e-5)
    # A quick run measures the headline alone.
    for k in ("e2e", "cpu_baseline", "precision", "precision_all_blocks", "per_block_launches", "fstats", "batched_requests",
              "other_configs"):
        line[k] = None
    line["other_arithmetics"] = {}
    assert bench.headline(line)["e2e"] is None
