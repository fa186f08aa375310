"""The benchmark's line on standard output: one JSON object of a few kilobytes
with every key of its contract, whatever the length of the full record."""
import json
import os
import sys

from conftest import ROOT

sys.path.insert(0, ROOT)


def test_line_is_short_and_complete():
    import bench

    its = list(range(1000))
    form = {"steps_per_s": 1 / 3, "ms_per_step": 2 / 3, "iterations_per_step": 4.5, "iterations": its,
            "max_residual": 9e-7, "converged": True, "launches": 7,
            "steps100": {"steps_per_s": 1 / 7, "iterations_mean": 3.3, "how": "x" * 200}}
    seq = {"ms_per_step": 2.0, "batch_speedup": 1.5, "how": "x" * 200}
    batch = {"value": 1e9, "unit": "voxel-updates/s", "ms_per_step": 3.0, "config": {"workload": "w", "sizes": [its] * 4},
             "forms": {"fp64": {"ms_per_step": 3.0, "sequential": seq, "iterations_last_step": its}}}
    line = {"metric": "m", "value": 2 / 3, "unit": "time-steps/s", "n_gpus": 1, "steps": 10, "warmup": 3,
            "ms_per_step": 100 / 3, "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f64",
            "data": "synthetic", "config": {"form": "proj"}, "roofline": {"frac": 0.75}, "roofline_mixed": {"x": its},
            "gpu_launches": 5, "clocks": {"sm_mhz": 2070, "reasons": []}, "forms": {f: form for f in "abcdefg"},
            "error_vs_fp64": {"a": {"max_rel": 1e-5, "rel_l2": 1e-6, "mask_dice": 1.0, "mask_level": "x" * 50}},
            "e2e": {"value": 1 / 3, "unit": "time-steps/s", "h2d_bytes_per_step": 8, "d2h_bytes_per_step": 8},
            "frontend": {"main_front_end_ms": 3.0, "components": {"max4d": {"ms": 0.5, "bytes_counted": "x" * 300}}},
            "batch": dict(batch, small_volumes=batch)}
    short = bench.short_line(line)
    text = json.dumps(short)
    assert len(text) < 8192 < len(json.dumps(line))
    for key in line:
        assert key in short or key == "roofline_mixed", key
    for key in ("value", "ms_per_step"):
        assert abs(short[key] - line[key]) <= 1e-6 * line[key]
    assert short["e2e"]["h2d_bytes_per_step"] == 8 and short["config"] == line["config"]
    assert short["forms"]["a"]["steps100"]["iterations_mean"] == 3.3
    assert short["batch"]["small_volumes"]["forms"]["fp64"]["speedup_over_sequential"] == 1.5
