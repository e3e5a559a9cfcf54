"""The benchmark's line keeps its keys and stays short, whatever the segments report."""
import json

import bench

KEYS = ("metric", "value", "unit", "n_gpus", "steps", "warmup", "ms_per_step", "higher_is_better", "scaling",
        "vs_baseline", "dtype", "data", "config", "e2e", "gpu_launches", "clocks", "roofline", "cpu_baseline")


def full_line():
    line = {k: 1.2345678901234567 for k in KEYS}
    line["metric"], line["dtype"] = bench.METRIC, bench.DTYPES["fp16x3"]
    line["config"] = {"workload": bench.WORKLOAD, "theta_shape": [8, 8, 2, 128, 2, 1024], "text": "x" * 120}
    line["roofline"] = {"text": "x" * 500}
    line["e2e"] = {"value": 78.4, "h2d_bytes_per_step": 536870912, "d2h_bytes_per_step": 536870912, "path": "x" * 200}
    line["cpu_baseline"] = {"value": 0.08, "sample": "x" * 120}
    line["clocks"] = {"sm_mhz": 2070.0, "sm_max_mhz": 2070.0, "reasons": ["sw_power_cap"]}
    line["kernels"] = {"tc_gemm": {"launches": 3, "ms": 5.78}}
    line["tc_tile_choices"] = ["128 256 1280 persist256 %d" % i for i in range(500)]
    line["u1_blocksparse"] = {"fp16x3": {"applies_per_s": 883.2}, "sector_gemms_mkn_per_step": [[1, 2, 3]] * 500}
    line["batched_eff_h1"] = {"ms_batched_graph": 0.8}
    line["gradient"] = {"error": "RuntimeError: " + "y" * 5000}
    line["dmrg_segment"] = {"time_ratio_fp64_over_mixed": 3.84, "runs": {"fp16x3": {"total_s": 1.01}}}
    return line


def test_line_is_short_and_complete():
    whole = full_line()
    line, detail = bench.headline(dict(whole))
    assert len(json.dumps(line)) <= bench.LINE_BYTES
    for k in KEYS:
        assert line[k] == whole[k], k
    for k in whole:
        assert (line if k in KEYS else detail)[k] == whole[k], k
    s = line["segments"]
    assert s["u1_fp16x3_applies_per_s"] == 883.2 and s["batched_64_ms"] == 0.8 and s["tile_choices"] == 500
    assert s["dmrg_step_fp64_over_mixed"] == 3.84 and "site_gradients_fp64_s" not in s
    assert line["segment_errors"]["gradient"].startswith("RuntimeError")


def test_line_without_segments():
    line, detail = bench.headline({k: 1 for k in KEYS})
    assert detail == {} and line["segments"] == {} and "segment_errors" not in line
