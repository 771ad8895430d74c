"""The benchmark's result line: one short JSON line with every key that its reader
needs, whatever the report beside it holds (lines of 20 KB were cut, and the result
with them)."""
import json

import bench

KEYS = {"metric": "m" * 90, "value": 1.4e9, "unit": "descriptors/s", "n_gpus": 1, "steps": 20, "warmup": 5,
        "ms_per_step": 13.3, "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f16x3",
        "data": "synthetic", "gpu_launches": 100}


def test_line_is_short_and_whole():
    report = dict(KEYS, precision_note="p" * 170, config=bench.workload_desc(19061120),
                  clocks={"sm_mhz": 1965.0, "sm_max_mhz": 1965.0, "reasons": ["sw_power_cap"], "samples": 99},
                  e2e={"value": 1.7e8, "unit": "descriptors/s", "h2d_bytes_per_step": 6, "d2h_bytes_per_step": 7},
                  roofline={"bound": "tensor", "frac": 0.43, "hbm_view": {"achieved": [1.0] * 1000}},
                  paths={p: {"value": 1.0, "rel_err_vs_fp64": {"x": [0.1] * 1000}} for p in bench.PATHS},
                  em={"config1": {"per_iteration": [0.1] * 1000}}, router_threshold_sweep=[{"a": 1.0}] * 1000)
    report.update({f"{p}_{k}": 1.2345678901234567e-05 for p in bench.PATHS for k in ("value", "rel_err_max")})
    text = bench.result_line(report)
    assert "\n" not in text and len(text) < 3000
    line = json.loads(text)
    assert {k: line[k] for k in KEYS} == KEYS
    for k in ("config", "clocks", "e2e"):
        assert line[k] == report[k]
    assert line["roofline"] == {"bound": "tensor", "frac": 0.43}
