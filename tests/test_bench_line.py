"""The benchmark's printed line: the headline and what it is judged by, short enough to be kept whole.

A line of 20 kB (every leg, every roofline, the autotuner's table) was cut off at its beginning
by a reader that keeps the last 3000 characters, and with it the headline.
"""
import json
import os
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _everything():
    """As run_ours assembles it, with texts and tables of the real lengths."""
    leg = {"value": 3367.7294028732413, "unit": "updates/s", "ms_per_step": 28.208917236328126, "svd": "x" * 120,
           "speedup_vs_plain_fp64": 1.0242378281908266, "max_abs_err_vs_plain_fp64": {"n_i": 1e-16, "entropy": 1e-16},
           "within_error_bound": True}
    roof = {"kernel": "k_jacobi_persistent<double>", "bound": "fp64", "achieved": 0.22639859511370414,
            "peak": 1.054799014178178, "unit": "TFLOP/s", "frac": 0.21463671473953483, "traffic": None,
            "peak_source": "y" * 140, "algorithmic": "z" * 160, "flops_per_launch": 1.0, "launches": 60,
            "avg_launch_ms": 5.123456789012345, "share_of_timed": 0.6123456789012345, "other": {"a": "b" * 500}}
    sat = {"workload": "w" * 120, "steps": 3, "start": "s" * 120, "fp64": dict(leg, rsvd={"a": "c" * 900}),
           "mixed": dict(leg), "mixed_without_model": dict(leg), "ab_model": {"what": "d" * 200}}
    return {"metric": "two-site updates/sec (Trotter steps/sec = value/95)", "value": 3288.0345855042924,
            "unit": "updates/s", "n_gpus": 1, "steps": 20, "warmup": 5, "ms_per_step": 28.892640125751495,
            "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "c128 (f64)",
            "data": "synthetic", "config": {"workload": "v" * 60, "svd": "u" * 480, "L": 64}, "phases": {},
            "e2e": {"value": 3263.2767134442256, "unit": "updates/s", "h2d_bytes_per_step": 5147632.0,
                    "d2h_bytes_per_step": 4198440.0, "steps": 20, "path": "t" * 120},
            "gpu_launches": 994, "window_autotune": [{"step": 4, "default_ms": 2.29}] * 12, "roofline": roof,
            "roofline_hbm": None, "cpu_baseline": {"value": 1.69, "unit": "updates/s", "cores": 1, "sample": "r" * 180},
            "precision_form": leg, "mixed_form": leg, "saturated": sat, "saturated_random_start": sat,
            "saturated_chi512": sat, "autotune_table": [{"route": "q" * 30}] * 15,
            "clocks": {"sm_mhz": 2070.0, "sm_max_mhz": 2070.0, "reasons": [], "samples": 3}}


def test_line_is_short_and_complete():
    sys.path.insert(0, ROOT)
    import bench

    out = _everything()
    line = bench.bench_line(out, "bench_out/bench_details.json")
    text = json.dumps(line)
    assert len(text) < 2900
    for key in ("metric", "value", "unit", "n_gpus", "steps", "warmup", "ms_per_step", "higher_is_better", "scaling",
                "vs_baseline", "dtype", "data", "config", "e2e", "gpu_launches", "clocks"):
        assert line[key] == out[key]
    assert list(line)[:2] == ["metric", "value"]
    assert line["legs_updates_per_s"]["saturated"]["mixed"] == round(3367.7294028732413, 2)


def test_line_without_the_legs():
    import bench

    out = _everything()
    for name in bench.LEGS + bench.SATURATED_LEGS:
        out[name] = None
    assert "legs_updates_per_s" not in bench.bench_line(out, "x")
