"""The benchmark's printed line: one short JSON object with the headline's keys, however long
the record it summarises (the batch leg's autotuner tables alone are 15 KB)."""

import json
import os
import sys

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
import bench  # noqa: E402


def _record():
    step = {"ms_per_step": 1.0 / 3.0, "value": 2.0 / 3.0, "step_frac": 0.25,
            "kernels": {"k%d" % i: {"ms": 1.0 / 3.0, "gbs": 1e4 / 3.0} for i in range(20)}}
    forms = {f: {"modes": {m: dict(step, smem_bytes=[1] * 100) for m in ("fused", "phased")},
                 "tuned": {"o2-%d" % i: {"tile": [4, 8, 8], "ms": 1.0 / 3.0} for i in range(300)}}
             for f in ("fp32", "fp64")}
    fields = ("grid_mass", "grid_momentum", "grid_velocity", "particle_velocity")
    errors = {f: {k: {"normwise": 1e-7 / 3.0, "per_entry": 1e-5, "entries": 9} for k in fields}
              for f in ("fp32_tiled", "fp32_plain", "fp64_plain")}
    return {"metric": bench.METRIC, "value": 1e10 / 3.0, "unit": "particles/s", "n_gpus": 1,
            "steps": 20, "warmup": 5, "ms_per_step": 1.0 / 3.0, "higher_is_better": True,
            "scaling": "weak", "vs_baseline": None, "dtype": "f32", "data": "synthetic",
            "config": {"workload": "w" * 120, "grid": 256, "parallelism": "replicas"},
            "e2e": {"value": 1e9 / 3.0, "unit": "particles/s", "h2d_bytes_per_step": 10200547328,
                    "d2h_bytes_per_step": 6442450944},
            "gpu_launches": 60, "clocks": {"sm_mhz": 1965.0, "sm_max_mhz": 1965.0, "reasons": []},
            "roofline": {"bound": "hbm", "frac": 1.0 / 3.0}, "step_roofline": {"frac": 1.0 / 3.0},
            "kernels": step["kernels"], "fp64_plain": step, "fp64_plain_unsorted": step,
            "sort": {"sort_ms": 7.0, "tile": [4, 8, 8]}, "errors_vs_fp64": {"grid_mass": 1e-7},
            "errors_vs_oracle": dict(errors, sample="s" * 100),
            "advect_cubic": {"workload": "w" * 300, "fp32": step, "fp64": step},
            "polypic": {"workload": "w" * 300, "quadratic_27": {"fp32": step, "fp64": step}},
            "batch": {"forms": forms, "autotune_measurements": list(range(5000))}}


def test_line_is_short_and_complete():
    record = _record()
    text = bench.stdout_line(record)
    assert "\n" not in text and len(text) < 4096
    line = json.loads(text)
    for k in ("metric", "value", "unit", "n_gpus", "steps", "warmup", "ms_per_step",
              "higher_is_better", "scaling", "vs_baseline", "dtype", "data", "e2e",
              "gpu_launches", "clocks", "config"):
        assert line[k] == record[k]
    assert line["batch_ms"]["fp64"]["phased"] == float("%.6g" % (1.0 / 3.0))


def test_batch_record():
    record = {k: v for k, v in _record().items() if k in ("metric", "value", "ms_per_step")}
    record.update(_record()["batch"])
    line = json.loads(bench.stdout_line(record))
    assert line["value"] == record["value"] and "fused" in line["batch_ms"]["fp32"]
