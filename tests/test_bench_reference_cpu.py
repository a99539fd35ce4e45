"""bench.py's reference arm where the reference is not built: one line that says so, and no error."""
import argparse
import json

import bench


def test_reference_arm_without_the_reference(monkeypatch, capsys):
    def missing():
        raise ModuleNotFoundError("No module named 'sr'")

    monkeypatch.setattr(bench, "reference_module", missing)
    assert bench.run_reference(argparse.Namespace(gpus=1, steps=2, warmup=3), 1, 0) == 0
    line = json.loads(capsys.readouterr().out)
    assert line["impl"] == "reference" and line["unavailable"] and "\n" not in line["unavailable"]
