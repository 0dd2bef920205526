"""bench.py's result line: the keys of the metric, in less than the 3,000 characters that readers of an
output's end keep, whatever the record carries besides."""

import io
import json
from contextlib import redirect_stderr, redirect_stdout

import bench


def test_result_line_is_short(tmp_path):
    record = {
        "metric": "bh_steps_per_s_1M_fp64_theta0.5", "value": 76.61234567891, "unit": "steps/s",
        "n_gpus": 1, "steps": 20, "warmup": 5, "ms_per_step": 13.0534567891, "higher_is_better": True,
        "scaling": "weak", "vs_baseline": None, "dtype": "f64", "data": "synthetic",
        "config": bench.headline_config(1),
        "e2e": {"value": 71.7, "unit": "steps/s", "h2d_bytes_per_step": 83886080,
                "d2h_bytes_per_step": 75497472},
        "gpu_launches": 480,
        "roofline": {"kernel": "k", "bound": "fp64", "achieved": 1.0 / 3.0, "peak": 1.0, "unit": "TFLOP/s",
                     "frac": 1.0 / 3.0, "traffic": 1.0 / 7.0, "traffic_source": "x" * 120,
                     "peak_source": "y" * 80, "note": "z" * 2000, "work": {"accepted_cells": 1}},
        "roofline_build": {"phases": {str(k): "p" * 500 for k in range(5)}}, "tree": {"nodes": 1},
        "clocks": {"sm_mhz": 2070, "sm_max_mhz": 2070, "reasons": ["none"]},
        "cpu_baseline": {"value": 0.33, "unit": "steps/s", "cores": 16, "kind": "port",
                         "sample": "s" * 200, "build_s": 1.0, "traversal_s": 2.0},
        "also": {str(k): "w" * 1000 for k in range(20)},
    }
    out, err = io.StringIO(), io.StringIO()
    path = tmp_path / "detail.json"
    with redirect_stdout(out), redirect_stderr(err):
        bench.print_result(record, str(path))
    assert out.getvalue().count("\n") == 1 and len(out.getvalue()) < 2500
    line = json.loads(out.getvalue())
    assert json.loads(err.getvalue()) == record and json.loads(path.read_text()) == record
    left_out = {"also", "roofline_build", "tree"}
    assert set(line) == set(record) - left_out
    for key in set(line) - {"roofline", "cpu_baseline"}:
        assert line[key] == record[key]
    assert line["roofline"]["frac"] == record["roofline"]["frac"]
