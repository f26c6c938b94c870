"""The benchmark's line on stdout stays short enough to be read back whole, whatever its
legs hold, and carries every key that is read from it."""
import json
import sys
from pathlib import Path

sys.path.insert(0, str(Path(__file__).resolve().parents[1]))

KEYS = ("metric", "value", "unit", "n_gpus", "steps", "warmup", "ms_per_step", "higher_is_better", "scaling",
        "vs_baseline", "dtype", "data", "config", "e2e", "gpu_launches", "clocks", "roofline", "cpu_baseline")


def test_the_legs_go_elsewhere():
    import bench

    line = dict.fromkeys(KEYS, 1.0)
    line["config"] = {"workload": "x" * 500}
    line["cpu_baseline"] = {"value": 0.06, "sample": "y" * 400}
    line["roofline"] = {"note": "z" * 400}
    for leg in bench.LEGS:
        line[leg] = {"ms_per_step": 2.5, "s_per_iter": 0.1, "rows": [{"text": "w" * 100}] * 100}
    head, legs = bench.split_line(line)
    assert all(head[k] == line[k] for k in KEYS)
    assert len(json.dumps(head)) < 3000
    assert set(legs) == set(bench.LEGS) and legs["batch"] == line["batch"]
    assert head["legs"]["batch_ms_per_iter"] == 2.5 and head["legs"]["persistent_s_per_iter"] == 0.1


def test_legs_that_did_not_run():
    import bench

    line = dict.fromkeys(KEYS, 1.0)
    line.update(dict.fromkeys(bench.LEGS))  # (skipped legs are null)
    head, legs = bench.split_line(line)
    assert all(v is None for v in legs.values())
    assert all(v is None for k, v in head["legs"].items() if k != "on")
