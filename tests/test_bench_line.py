"""The benchmark's printed line: the contract's keys whatever was measured, short
enough to be kept whole by whoever records it."""
import json
import os
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)


def _report(bench):
    num = 123456789.0123456789
    full = {k: num for k in bench.LINE_KEYS}
    full |= {"metric": bench.METRIC, "unit": bench.UNIT, "scaling": "weak", "dtype": "f32", "data": "synthetic",
             "config": bench._config(512), "higher_is_better": True, "vs_baseline": None,
             "cpu_baseline": {"value": num, "unit": bench.UNIT, "cores": 16, "kind": "port", "sample": "x" * 400},
             "clocks": {"sm_mhz": 2070.0, "sm_max_mhz": 2070.0, "reasons": ["sw_power_cap"], "samples": 99},
             "roofline": {k: num for k in bench.ROOFLINE_KEYS} | {"kernel_ms": {"rk4_fused_level": num}},
             "e2e": {k: num for k in bench.E2E_KEYS} | {"path": "x" * 2000}}
    for path in bench.LEG_FIGURES:
        d, *rest = path.split(".")
        at = full
        for k in [d, *rest][:-1]:
            at = at.setdefault(k, {"long": list(range(2000))})
        at[path.split(".")[-1]] = num
    return full


def test_line_is_short_and_keeps_the_contract():
    import bench
    text = json.dumps(bench.compact(_report(bench)))
    assert len(text) < 4096 and "\n" not in text
    line = json.loads(text)
    for k in ("metric", "value", "unit", "n_gpus", "steps", "warmup", "ms_per_step", "higher_is_better", "scaling",
              "vs_baseline", "dtype", "data", "config", "roofline", "cpu_baseline", "e2e", "clocks", "gpu_launches"):
        assert k in line, k
    assert {"value", "unit", "h2d_bytes_per_step", "d2h_bytes_per_step"} <= set(line["e2e"])
    assert {"sm_mhz", "sm_max_mhz", "reasons"} <= set(line["clocks"]) and line["config"]["grid"] == [512] * 3
    assert len(line["legs"]) == len(bench.LEG_FIGURES)


def test_line_of_a_run_without_the_legs():
    import bench
    full = {k: v for k, v in _report(bench).items() if k in bench.LINE_KEYS}
    full |= {"fp64": None, "e2e": None, "adjoint": None, "scale_1024": {"unavailable": "no room"}}
    line = bench.compact(full)
    assert line["legs"] == {"scale_1024.unavailable": "no room"}
    assert "e2e" not in line and "roofline" not in line and line["value"] == 123456789.0
