"""The line that bench.py prints: short enough for the tail of a log, with the keys that name and qualify the measurement unchanged."""
import json
import os
import sys

import pytest

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
import bench


def record(rows):
    table = [{"c": 256, "hw": 14, "k": 3, "s": 2, "layout": "nchw", "dtype": "f32", "pass": "bwd_data", "ms": 0.125, "tflops": 78.4} for _ in range(rows)]
    note = "word " * 100
    return {"metric": "quaternion conv2d fwd+bwd TFLOP/s", "value": 1240.3659615911226, "unit": "TFLOP/s", "n_gpus": 1, "steps": 20, "warmup": 5,
            "ms_per_step": 0.5090112209320068, "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f16", "data": "synthetic",
            "config": {"workload": "w" * 150, "parallelism": "dp1", "l2": "exceed", "flop_per_step_per_gpu": 631360192512.0},
            "clocks": {"sm_mhz": 1965, "sm_max_mhz": 1965, "reasons": ["sw_power_cap"]}, "gpu_launches": 80,
            "e2e": {"value": 43.72437911892352, "unit": "TFLOP/s", "h2d_bytes_per_step": 616824832, "d2h_bytes_per_step": 616824832,
                    "copy_roofline": {"frac": 0.9919, "note": note}},
            "parity": {"y": 2.4577e-4, "ok": True, "checked": note}, "roofline": {"bound": "tensor", "frac": 0.75586, "per_clock": {"f": 0.7}, "traffic_note": note},
            "kernel_sm_mhz": {k: {"short": 1965, "long": 1320.0, "long_launches": 12017} for k in ("forward", "backward_filter", "backward_data")},
            "qresnet18": {"value": 25699.0, "e2e": {"value": 1.0}, "glue": note, "layers": {"rows": table}},
            "dense": {"config": note, "f32": {"fwd_ms": 0.0214}}, "sweep": {"config": note, "rows": table}, "sweep_f32": {"config": note, "rows": table}}


@pytest.mark.parametrize("rows", [1, 60, 1000])
def test_line_is_short_and_keeps_its_keys(rows):
    r = record(rows)
    line = bench.compact(r)
    assert len(json.dumps(line)) <= bench.LINE_LIMIT
    for k in ("metric", "value", "unit", "n_gpus", "steps", "warmup", "ms_per_step", "higher_is_better", "scaling", "vs_baseline", "dtype", "data",
              "config", "clocks", "gpu_launches"):
        assert line[k] == r[k]
    for k in ("value", "unit", "h2d_bytes_per_step", "d2h_bytes_per_step"):
        assert line["e2e"][k] == r["e2e"][k]
    assert line["parity"]["ok"] is True and line["roofline"]["frac"] == 0.75586 and line["qresnet18"]["value"] == 25699.0
    assert line["sweep"] == {"rows": rows, "ms_sum": pytest.approx(0.125 * rows)}


def test_missing_legs():
    r = record(1)
    for k in ("sweep", "sweep_f32", "dense", "qresnet18"):
        del r[k]
    r["e2e"] = None                                              # a run of the kernels alone
    assert bench.compact(r).get("e2e") is None
