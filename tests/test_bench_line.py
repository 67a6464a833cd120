"""The line that bench.py prints stays short, whatever the full record holds: the first of
the two is what a log with a few kB of room keeps."""
import json

import bench


def test_short_line():
    row = {f"{k}_{m}": 1.234567890123456e-07 for k in ("u", "w", "uvs", "wvs", "vel_total", "gamma")
           for m in ("rel_l2", "max")}
    leg = {f"key_{k}": 123.45678901234567 for k in range(18)}
    line = {
        "metric": bench.METRIC, "value": 3356.1234567890123, "unit": bench.UNIT, "n_gpus": 1, "steps": 20, "warmup": 5,
        "ms_per_step": 19.07123456789, "higher_is_better": True, "scaling": "weak", "vs_baseline": None,
        "dtype": "d" * 60, "data": "d" * 40,
        "config": {"workload": "w" * 220, "instances": 64, "blobs_total": 8999596, "panels_total": 14501,
                   "parallelism": "single GPU", "l2": "l" * 60, "graph": "g" * 40},
        "gpu_launches": 560, "gpu_launches_note": "n" * 200, "setup_s": 12.345678,
        "clocks": {"sm_mhz": 1965.0, "sm_max_mhz": 1965.0, "samples": 51, "reasons": []},
        "roofline": {**{k: 123.45678901234567 for k in ("achieved", "peak", "frac", "traffic", "launch_ms",
                                                        "share_of_step", "pairs_represented_per_launch")},
                     "bound": "latency", "kernel": "k" * 40, "unit": "GB/s", "frac_is": "f" * 200},
        "e2e": {"value": 1099.123456789, "unit": bench.UNIT, "h2d_bytes_per_step": 145955013,
                "d2h_bytes_per_step": 215511760, "note": "n" * 600},
        "plain_gpu": {"value": 1.0, "unit": bench.UNIT, "ratio_batched_over_plain": 2.0, "how": "h" * 100},
        "cpu_baseline": {"value": 0.1276, "unit": bench.UNIT, "cores": 16, "kind": "reference", "sample": "s" * 300},
        "accuracy": {"simulations": 64, "pooled_rel_l2": {k: 1.2345678901e-7 for k in
                                                          ("u", "w", "uvs", "wvs", "vel_total", "gamma")},
                     "within_bounds": True, "per_simulation": [dict(row) for _ in range(64)]},
        "f64_value": 45.168, "f64": {"how": "h" * 300}, "nbody": {"n": 1 << 20, "pair_kernel_ms": 1.7,
                                                                  "gpairs_per_s": 643000.0},
        "serving": {"requests": 1000, "arrivals": "a" * 200, "realtime_live": {"batched": dict(leg, latency_p50_s=0.03)},
                    "saturated": {"batched": dict(leg, sim_steps_per_s=15193.0), "serial": dict(leg),
                                  "ratio_batched_over_serial": 4.65}},
    }
    short = bench.short_line(line)
    assert len(json.dumps(short)) <= 2700
    for k in ("metric", "value", "unit", "n_gpus", "steps", "warmup", "ms_per_step", "higher_is_better", "scaling",
              "vs_baseline", "dtype", "data", "config", "e2e", "gpu_launches", "clocks"):
        assert short[k] is line[k] or set(short[k]) <= set(line[k])
    assert short["e2e"]["value"] == line["e2e"]["value"] and "per_simulation" not in short["accuracy"]
    assert short["serving"]["ratio_batched_over_serial"] == 4.65 and short["serving"]["latency_p50_s"] == 0.03
    assert bench.short_line({"value": 1.0}) == {"value": 1.0}
