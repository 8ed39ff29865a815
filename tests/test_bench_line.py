"""The printed line of bench.py: every scalar and the named keys of every leg, short enough for a log that keeps the
last few KB of the output."""

from __future__ import annotations

import json

import bench


def test_summary_keeps_scalars_and_drops_series():
    line = {"metric": "m", "value": 1.5, "unit": "u", "n_gpus": 1, "vs_baseline": None, "gpu_launches": 3000,
            "config": {"workload": "w", "l2": "flushed"}, "clocks": {"sm_mhz": 2070, "reasons": []},
            "e2e": {"value": 2.0, "unit": "u", "h2d_bytes_per_step": 48, "d2h_bytes_per_step": 1 << 32,
                    "call_seconds": [0.1] * 500},
            "roofline": {"bound": "fp64", "achieved": 1.0, "peak": 2.0, "unit": "TFLOP/s", "frac": 0.5,
                         "terms": {"a": [1] * 500}},
            "field_sweep": {"fields": 64, "mixed_ms_total": 1.0, "per_field": [{"B": [0.1] * 3}] * 640},
            "autotune": {"mixed": {"seconds": 1.0}}, "serving": None, "cpu_baseline": {"value": 1.0, "unit": "u",
                                                                                     "cores": 16, "kind": "port"}}
    short = bench.summary(line)
    for key in ("metric", "value", "unit", "n_gpus", "vs_baseline", "gpu_launches", "config", "clocks", "serving",
                "cpu_baseline"):
        assert short[key] == line[key]
    assert short["e2e"] == {k: line["e2e"][k] for k in ("value", "unit", "h2d_bytes_per_step", "d2h_bytes_per_step")}
    assert set(short["roofline"]) == {"bound", "unit", "achieved", "peak", "frac"}
    assert "per_field" not in short["field_sweep"] and short["field_sweep"]["fields"] == 64
    assert len(json.dumps(short)) < 4096
