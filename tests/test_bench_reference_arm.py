"""The benchmark's reference arm is the reference or nothing: where its driver
was not built the arm says so, and times no restatement in its name."""
import argparse
import json

import bench
import refio


def test_without_the_reference_driver_the_arm_is_unavailable(monkeypatch, capsys):
    monkeypatch.setattr(refio, "driver_available", lambda: False)
    monkeypatch.setattr(bench, "cpu_reference_sample", lambda *a, **k: {"kind": "port", "each": [1.0] * 8, "n": 1, "cores": 1})
    for name in ("RANK", "LOCAL_RANK", "WORLD_SIZE"):
        monkeypatch.delenv(name, raising=False)
    bench.run_reference_arm(argparse.Namespace(gpus=1, steps=2, warmup=3))
    line = json.loads(capsys.readouterr().out)
    assert line["impl"] == "reference" and line["unavailable"]
    assert "value" not in line and "config" not in line
