"""The line bench.py prints: short enough to be read whole from the end of the
output, with every key of the measurement contract as measured."""
import json
import os
import sys

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, REPO)

import bench  # noqa: E402

CONTRACT = ("metric", "value", "unit", "n_gpus", "steps", "warmup", "ms_per_step", "higher_is_better", "scaling",
            "vs_baseline", "dtype", "data", "config", "e2e", "gpu_launches", "clocks")


def _report(filler):
    """A report with sections of a default run's kind, `filler` words in each."""
    deep = {f"step_{k}": {f"figure_{j}": 1.0 / (3 + j) for j in range(9)} for k in range(filler)}
    text = "what the number means " * filler
    res = {"metric": bench.METRIC, "value": 16058262.496975265, "unit": bench.UNIT, "n_gpus": 1, "steps": 2000,
           "warmup": 20, "ms_per_step": 0.2550711822509766, "higher_is_better": True, "scaling": "weak",
           "vs_baseline": None, "dtype": "f32 faces, f64 sums", "data": "synthetic (seeded meshes, poses and velocities)",
           "config": {"workload": "mixed_batch_4096_bodies_distinct_meshes", "bodies": 4096, "faces_per_step": 37828450,
                      "distinct_mesh_faces": 37828450, "surface": "flat", "current_mps": [0.2, 0.0, 0.0],
                      "density": 1025.0, "l2_policy": "inputs larger than L2 (mesh data > 129 MB)",
                      "processed_faces_per_step": 27966726, "parallelism": "single GPU"},
           "faces_per_s": 148305463855.88477,
           "e2e": {"value": 14483838.977730138, "unit": bench.UNIT, "h2d_bytes_per_step": 2588672,
                   "d2h_bytes_per_step": 688128, "steps": 500, "transfer": text},
           "kernel_ms": {"prep": 0.0111, "chunk": 0.2401, "finalize": 0.0143}, "gpu_launches": 6000,
           "clocks": {"sm_mhz": 2070.0, "sm_max_mhz": 2070.0, "power_w_max": 308.62, "samples": 14, "reasons": []}}
    for key in bench.SECTIONS:
        res[key] = {"value": 1.0 / 3.0, "kind": "port", "note": text, "deep": deep,
                    **{f"number_{k}": 1e6 / (7 + k) for k in range(8)}}
    res["rollout"]["exact"] = {"env_steps_per_s": 8242488.7652583355, **deep}
    return res


def test_line_is_short_and_keeps_the_contract():
    for filler in (1, 12, 300):
        res = _report(filler)
        line = bench.short_line(res)
        assert len(line) <= 3000 and "\n" not in line
        d = json.loads(line)
        for key in CONTRACT:
            if key != "e2e":
                assert d[key] == res[key], key
        assert all(d["e2e"][k] == res["e2e"][k] for k in ("value", "unit", "h2d_bytes_per_step", "d2h_bytes_per_step"))
        assert d["cpu_baseline"]["kind"] == "port"
    assert json.loads(bench.short_line(_report(1)))["rollout"]["exact_env_steps_per_s"] == 8242490.0
