"""The line that bench.py prints: every key of its contract and a few figures of each part, short enough for a reader
that keeps a few thousand characters (a line of 24 kB was cut and read as no result)."""
import json
import os
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)
import bench  # noqa: E402

CONTRACT = ["metric", "value", "unit", "n_gpus", "steps", "warmup", "ms_per_step", "higher_is_better", "scaling",
            "vs_baseline", "dtype", "data", "config", "e2e", "gpu_launches", "clocks"]


def test_printed_line_is_short_and_complete():
    number = 123456789.12345678
    line = {k: number for k in bench.HEAD}
    line.update({"e2e": {"call": "x" * 300, **{"k%d" % i: number for i in range(5)}}, "config": {"workload": "x" * 450},
                 "roofline": {"note": "x" * 420}, "cpu_baseline": {"sample": "x" * 170}, "clocks": {"reasons": []}})
    deep = {"plain_fits_per_s": number, "learned_fits_per_s": number, "note": "y" * 4000}
    line["learned_other_configs"] = {"as3d": deep, "multi": {**deep, "lr_selection": {"fits_per_s": number}}}
    line["frames"] = {"frames_per_s": number, "e2e": {"frames_per_s": number}, "note": "y" * 5000}
    head, parts = bench.printed(line)
    got = json.loads(head)
    assert "\n" not in head and len(head) < 5000
    assert all(k in got for k in CONTRACT)
    assert got["parts"]["frames.e2e.frames_per_s"] == number
    assert got["parts"]["learned_other_configs.multi.lr_selection.fits_per_s"] == number
    assert "consecutive_fit.rows_per_s" not in got["parts"]  # a part switched off
    full = json.loads(parts)
    assert full["frames"] == line["frames"] and "value" not in full
