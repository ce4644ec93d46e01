"""The line bench.py prints on stdout: the contract's keys whole, the sections short enough for the tail of a log."""
import json
import os
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)

import bench  # noqa: E402


def full_line():
    acc = {"rel_l2_vs_fp64_truth": 1.23456789e-7, "loads": {"count": 17, "rel_l2_max": 9.87654321e-7, "note": "x" * 200}}
    row = {"value": 1.23456789, "kernel_ms": 1.1, "setup_ms": 0.003, "iterations": 187, "reductions": 193,
           "reliable_updates": 3, "tolerance": 5e-6, "true_rel_residual": 4.9e-6, "coarse_dim": 444, "accuracy": acc}
    return {"metric": bench.METRIC, "value": 1.2, "unit": "ms", "n_gpus": 1, "steps": 20, "warmup": 5,
            "ms_per_step": 1.2, "higher_is_better": False, "scaling": "weak", "vs_baseline": None,
            "dtype": "f32 inner / f64 refinement", "data": "synthetic", "config": {"workload": "plate", "dof": 60492, "l2": "flushed between steps", "note": "y" * 150},
            "method": {"name": "mixed_two_level_cheb", "preconditioner": "z" * 90, "ctas": 148},
            "variants": {f"variant_{i}": dict(row) for i in range(7)},
            "roofline": {"achieved": 1.0, "frac": 0.1, "l2": {"peak": 2.0, "peak_source": "w" * 150}},
            "e2e": {"value": 1.5, "unit": "ms", "h2d_bytes_per_step": 241968, "d2h_bytes_per_step": 484000},
            "gpu_launches": 20, "clocks": {"sm_mhz": 1965, "sm_max_mhz": 1965, "reasons": []}, "accuracy": acc,
            "load_cases": {"cases": 4, "device_ms_per_case": 1.0, "iterations": list(range(64))},
            "learned": {"value": 40.0, "method": "m" * 120, "held_out": {"loads": 512, "ms_p50": 39.9}},
            "other_configs": {f"c{i}": {"best": "mixed", "best_ms": 1.0, "variants": {"v": row}} for i in range(4)},
            "batch": {"method": "mixed_two_level", "batch_ms": 260.0, "times": list(range(500)),
                      "methods": {f"m{i}": {"all": list(range(300))} for i in range(4)}},
            "cpu_baseline": {"value": 3200.0, "unit": "ms", "cores": 1, "sample": "s" * 200}}


def test_summary_keeps_the_contract_and_fits():
    line = full_line()
    short = json.loads(json.dumps(bench.summary(line)))
    for k in ("metric", "value", "unit", "n_gpus", "steps", "warmup", "ms_per_step", "higher_is_better", "scaling",
              "vs_baseline", "dtype", "data", "e2e", "gpu_launches", "clocks"):
        assert short[k] == line[k], k
    assert short["config"] == {"workload": "plate", "dof": 60492, "l2": "flushed between steps"}
    assert len(json.dumps(short)) < 2500
    assert short["variants_ms"]["variant_3"] == 1.2346 and short["method"] == "mixed_two_level_cheb"
    assert short["batch"]["batch_ms"] == 260.0 and short["learned"]["value"] == 40.0
    assert short["rel_l2_max"] == 9.87654321e-7 and short["other_configs_ms"]["c2"] == 1.0


def test_summary_without_sections():
    line = {k: v for k, v in full_line().items()
            if k not in ("load_cases", "learned", "other_configs", "batch", "accuracy", "cpu_baseline")}
    short = bench.summary(line)
    assert short["rel_l2_max"] is None and short["cpu_baseline"] is None and short["other_configs_ms"] == {}
