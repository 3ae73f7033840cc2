"""The benchmark's reference arm times the reference's own code or nothing."""

import argparse
import json
import pathlib
import sys

sys.path.insert(0, str(pathlib.Path(__file__).resolve().parents[1]))
import bench  # noqa: E402


def test_reference_arm_without_the_reference_says_so(monkeypatch, capsys, tmp_path):
    """No number of this repository's own C port stands in for a reference that is not on the machine."""
    def timed(*_):
        raise AssertionError("something was timed in the reference's place")
    monkeypatch.setattr(bench, "ROOT", tmp_path)
    monkeypatch.setattr(bench, "cpu_decode_sample", timed)
    monkeypatch.setattr(bench, "model_path", timed)
    bench.run_reference(argparse.Namespace(gpus=1, steps=2, warmup=3), 0)
    line = json.loads(capsys.readouterr().out)
    assert line["impl"] == "reference" and line["unavailable"] and "value" not in line
