"""
The bench's printed line stays a few kilobytes, whatever its legs measured, and
keeps the keys and numbers of the headline.
"""
import json

import bench

ORDER = {"pixel_iter_per_s": 3.1e13, "wall_s": 17.5, "latency_ms": {"p50": 100.123456789, "p99": 9.9e3, "n": 2000},
         "latency_ms_by_side": {str(k): {"p50": 1.23456789, "p99": 2.3456789} for k in (256, 512, 1024, 2048)}}
LEG = {"workload": "w" * 400, "fe32": {"kernel_ms": 1.23456789, "value": 1e13, "full_steps": 10 ** 11},
       "vs_oracle": {"oracle_s": 1., **{f"output_{k}": 0.123456789 for k in range(60)}},
       "vs_exact": {"direct_s": 2., **{f"output_{k}": 0.123456789 for k in range(60)}}}


def test_line_is_short_and_whole():
    line = {"metric": bench.METRIC, "value": 1.0e14, "unit": "pixel-iter/s", "n_gpus": 1, "steps": 20,
            "warmup": 5, "ms_per_step": 7.4, "higher_is_better": True, "scaling": "weak", "vs_baseline": None,
            "dtype": "f32+i32exp", "data": "synthetic", "config": {"nx": 2048}, "gpu_launches": 20,
            "clocks": {"sm_mhz": 2070.0}, "e2e": {"value": 1.0e14, "h2d_bytes_per_step": 32768},
            "serving": {"rate_per_s": 200., **{k: ORDER for k in ("fifo", "shortest", "hrrn", "fifo_1gb")}},
            "supplementary": {f"leg_{k}": LEG for k in range(8)}}
    assert len(json.dumps(line)) > 20000
    out = json.loads(json.dumps(bench.short_line(line)))
    assert len(json.dumps(out)) < 4000
    for k in line:
        if k not in ("serving", "supplementary"):
            assert out[k] == line[k]
    assert out["serving"]["hrrn"] == {"pixel_iter_per_s": 3.1e13, "p50_ms": 100.123456789, "p99_ms": 9.9e3}
    assert out["supplementary"] == {f"leg_{k}.fe32.kernel_ms": 1.2346 for k in range(8)}


def test_line_without_the_legs():
    assert bench.short_line({"value": 1., "serving": None, "supplementary": None}) == {
        "value": 1., "serving": None, "supplementary": None}
