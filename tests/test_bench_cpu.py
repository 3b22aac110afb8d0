"""bench.py where the reference's sources are absent (no oracle library): both arms still keep their line."""
import argparse
import json

import numpy as np
import pytest

import bench
import oracle as O


@pytest.fixture
def no_oracle(monkeypatch, tmp_path):
    monkeypatch.setattr(O, "LIB_PATH", str(tmp_path / "liboracle.so"))
    monkeypatch.setattr(O, "_lib", None)


def test_reference_arm_says_unavailable(no_oracle, capsys):
    planes = [np.zeros((1500, 2000), np.uint8), np.zeros((750, 1000), np.uint8), np.zeros((750, 1000), np.uint8)]
    args = argparse.Namespace(gpus=1, steps=1, warmup=1, qindex=120)
    bench.cpu_reference(args, planes, 0)
    line = json.loads(capsys.readouterr().out)
    assert line["impl"] == "reference" and "oracle" in line["unavailable"] and set(line) == {"impl", "unavailable"}
    bench.cpu_reference(args, planes, 1)   # the other ranks print nothing
    assert capsys.readouterr().out == ""


def test_own_arm_reports_the_missing_baseline(no_oracle):
    planes = [np.zeros((1500, 2000), np.uint8), np.zeros((750, 1000), np.uint8), np.zeros((750, 1000), np.uint8)]
    assert "oracle" in bench.cpu_baseline(planes, 120)["unavailable"]
