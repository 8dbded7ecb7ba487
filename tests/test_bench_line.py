"""The line that bench.py prints: short, whatever the report behind it holds, with the
headline's keys and the main figures of each configuration."""
import json
import sys
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent
sys.path.insert(0, str(ROOT))

import bench  # noqa: E402


def _report(padding):
    rate = {"value": 1.2345678901234567e11, "unit": "particle-steps/s",
            "ms_per_step": 10.117686367034912, "text": padding,
            "e2e": {"value": 1.15188634438e11, "call": padding},
            "cpu_baseline": {"value": 33153322.78533194, "sample": padding}}
    form = {"kernel_ms": 8.718534469604492, "particle_steps_per_s": 1.443e11,
            "fp64_error": {"sample": 512, "text": padding}}
    return {
        "metric": bench.METRIC, "value": 1.24434730661e11, "unit": bench.UNIT, "n_gpus": 1,
        "steps": 30, "warmup": 3, "ms_per_step": 10.117686367034912, "higher_is_better": True,
        "scaling": "weak", "vs_baseline": None, "dtype": "f32", "data": "synthetic",
        "config": {"seeds_per_rank": 1048576}, "e2e": rate["e2e"] | {"call": ""},
        "gpu_launches": 120, "clocks": {"sm_mhz": 1965.0, "sm_max_mhz": 1965.0, "reasons": []},
        "precision_forms": {"f32": {"fp64_error": padding}, "f16": form, "bf16": form},
        "fp64_error": padding, "true_rk4": form, "systems_forms": padding, "recording": rate,
        "ftle": rate, "batched": rate | {"f16": form, "plain_f32": form},
        "serving": {"latency_ms": {"p50_pooled": 12.2, "p99_pooled": 202.0, "p99_max": 511.0},
                    "particle_steps_per_s": 2.29e10, "runs": [padding] * 3}}


def test_line_is_short_and_keeps_the_main_figures():
    report = _report("x" * 5000)
    line = bench.headline(report)
    assert len(json.dumps(line)) < 2600
    for key in ("metric", "value", "unit", "n_gpus", "steps", "warmup", "ms_per_step",
                "higher_is_better", "scaling", "vs_baseline", "dtype", "data", "config", "e2e",
                "gpu_launches", "clocks"):
        assert line[key] == report[key]
    main = line["configurations"]
    assert main["recording"]["value"] == main["ftle"]["value"] == report["ftle"]["value"]
    assert main["batched"]["e2e"] == report["batched"]["e2e"]["value"]
    assert main["batched"]["f16"] == report["batched"]["f16"]["particle_steps_per_s"]
    assert main["serving"]["latency_ms"] == {"p50_pooled": 12.2, "p99_pooled": 202.0}
    assert main["kernel_ms"] == {"f16": 8.718534469604492, "bf16": 8.718534469604492}


def test_line_of_a_run_without_the_configurations():
    report = {"metric": bench.METRIC, "value": 1.0}
    assert bench.headline(report) == report
