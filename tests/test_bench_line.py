"""The benchmark's result line: every key a reader needs, short enough for one that keeps the end of the output."""
import json


def _result():
    phases = [[f"a_phase_of_the_call_{i}", 1.0 / 3.0] for i in range(40)]
    roof = {"bound": "tensor", "achieved": 1591.123456789, "peak": 1714.8, "unit": "TFLOP/s", "frac": 0.92712345678,
            "traffic": 123456789012.0, "kernel": "k_crt_gemm", "peak_note": "x" * 200, "traffic_note": "y" * 300}
    part = {"value": 117.123456789012, "unit": "TFLOP/s", "ms_per_step": 75.123456789, "steps": 20, "phases_ms": phases,
            "call_ms": [75.1] * 200, "sample": "s" * 120, "roofline": roof, "wall_s": 18.5}
    r = {"metric": "Cauchy", "value": 117.123456789012, "unit": "TFLOP/s", "n_gpus": 1, "steps": 20, "warmup": 5,
         "ms_per_step": 75.123456789012, "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "bf16",
         "data": "synthetic", "config": {"workload": "w" * 120, "n": 16384, "l2": "inputs larger than L2", "parallelism": "p" * 60},
         "latency_ms": {"p50": 75.123456, "p99": 75.5}, "phases_ms": {p: v for p, v in phases[:8]}, "gpu_launches": 160,
         "roofline": roof, "fp64_plain": dict(part), "rel_err": {"split_vs_fp64_path": 2.6e-13},
         "e2e": dict(part, h2d_bytes_per_step=2148007936, d2h_bytes_per_step=2147483648, median_call_tflops=112.3,
                     stalled_calls=0, redone_calls=0, first_call_phases_ms=phases, slowest_call_timeline_ms=phases),
         "cpu_baseline": dict(part, cores=16, kind="port"),
         "clocks": {"sm_mhz": 1812.0, "sm_max_mhz": 2070.0, "reasons": ["sw_power_cap"]}}
    return dict(r, extra={name: dict(part, kinds={"toeplitz": part, "dft": part}) for name in ("cfg0", "cfg1", "cfg3", "cfg4")})


def test_line_is_short_and_whole():
    import bench
    r = _result()
    assert len(json.dumps(r)) > 20000
    line = bench.compact_line(r)
    text = json.dumps(line)
    assert len(text) < 3500
    for key in ("metric", "value", "unit", "n_gpus", "steps", "warmup", "ms_per_step", "higher_is_better", "scaling", "vs_baseline",
                "dtype", "data", "config", "gpu_launches", "clocks", "roofline", "e2e", "cpu_baseline"):
        assert key in line
    assert line["value"] == r["value"] and line["ms_per_step"] == r["ms_per_step"]
    assert line["e2e"]["value"] == r["e2e"]["value"]
    assert line["e2e"]["h2d_bytes_per_step"] == r["e2e"]["h2d_bytes_per_step"]
    assert line["clocks"]["reasons"] == ["sw_power_cap"]
    assert [line["extra"][c]["value"] for c in ("cfg0", "cfg1", "cfg3", "cfg4")] == [117.12] * 4
