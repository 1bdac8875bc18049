"""The benchmark's printed line: short enough to be kept whole, headline keys as they are.

Parity and error tables of a leg hold an entry for each member checked, and
the line with all of them is some 22 KB, of which a reader that keeps the end
of the output has no beginning.
"""
import json
import os
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
HEADLINE = ("metric", "value", "unit", "n_gpus", "steps", "warmup", "ms_per_step", "higher_is_better", "scaling",
            "vs_baseline", "dtype", "data", "gpu_launches")


def _line():
    x = 0.1234567890123456
    phases = {f"phase_{k}": x for k in range(16)}
    error = {f"max_error_{k}": x for k in range(8)}
    parity = {"ok": True, "members": {str(k): {"ok": True, "state_mismatches": [], **error} for k in range(16)},
              "ledgers": error, "note": "n" * 300, "substeps": 90}
    leg = {"value": 2.5e10 + x, "unit": "projections/s", "p99_latency_s": x, "parity": parity,
           "fp64_error": {"members": {str(k): error for k in range(16)}, "max_position_error_over_extent": x},
           "phase_ms_per_substep": phases, "workload": "w" * 400, "cpu_baseline": {"value": x, "sample": "s" * 300},
           "e2e": {"value": 1.5e10, "wall_s": x}, "load_sweep": [phases] * 3}
    return {"metric": "bond projections/s", "value": 26931657527.113033, "unit": "projections/s", "n_gpus": 1,
            "steps": 20, "warmup": 5, "ms_per_step": 51.25547790527344, "higher_is_better": True, "scaling": "weak",
            "vs_baseline": None, "dtype": "f32 (f64 ledgers)", "data": "synthetic", "gpu_launches": 8100,
            "config": {"workload": "impact", "nodes": 4194304},
            "e2e": {"value": 17422651572.605854, "unit": "projections/s", "h2d_bytes_per_step": 1639717546,
                    "d2h_bytes_per_step": 361499648, "note": "n" * 120},
            "roofline": {"bound": "hbm", "frac": x, "kernel": "kSolve", "note": "n" * 120},
            "clocks": {"sm_mhz": 2070.0, "sm_max_mhz": 2070.0, "reasons": []}, "phase_ms_per_substep": phases,
            "parity": {"ok": True, "ledgers": error, "note": "n" * 130}, "fp64_error": error,
            "cpu_baseline": {"value": x, "sample": "s" * 300},
            **{name: json.loads(json.dumps(leg)) for name in ("cantilever", "batched", "served", "cascade")}}


def test_printed_line_is_short_and_keeps_the_headline():
    sys.path.insert(0, ROOT)
    import bench

    line = _line()
    before = json.dumps(line)
    short = bench.headline(line)
    assert json.dumps(line) == before  # the detail is not touched
    text = json.dumps(short)
    assert "\n" not in text and len(text) < 6000 < len(before)
    for k in HEADLINE:
        assert short[k] == line[k], k
    for k in ("config", "e2e", "roofline", "clocks"):
        assert list(short[k]) == list(line[k]), k
        for q, v in line[k].items():
            assert short[k][q] == v or abs(short[k][q] / v - 1) < 1e-6, (k, q)
    for name in ("cantilever", "batched", "served", "cascade"):
        assert short[name]["parity"]["ok"] is True and abs(short[name]["value"] / line[name]["value"] - 1) < 1e-6
        assert short[name]["p99_latency_s"] > 0 and short[name]["e2e"]["value"] == line[name]["e2e"]["value"]


def test_figures_that_are_no_numbers_pass():
    sys.path.insert(0, ROOT)
    import bench

    assert str(bench.headline({"value": 1.0, "e2e": {"value": float("nan"), "n": 3, "s": "x"}})["e2e"]["value"]) == "nan"
