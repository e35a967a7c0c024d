"""bench.py where the host build of the reference kernels is absent: the
reference arm says so and ends well, and the product's own line is not lost."""
import argparse
import json
import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)

import bench  # noqa: E402
import pipeline as PL  # noqa: E402


@pytest.fixture
def no_reference(monkeypatch, tmp_path):
    monkeypatch.setattr(PL, "HERE", str(tmp_path))


def test_reference_arm_is_unavailable(no_reference, capsys):
    assert bench.run_reference(argparse.Namespace(gpus=1, steps=1, warmup=3)) == 0
    lines = capsys.readouterr().out.strip().splitlines()
    assert len(lines) == 1
    d = json.loads(lines[0])
    assert d["impl"] == "reference" and d["unavailable"] and "\n" not in d["unavailable"]


def test_cpu_baseline_raises_its_own_error(no_reference):
    """The error that the product's arm reports in place of its CPU baseline."""
    with pytest.raises(bench.ReferenceUnavailable):
        bench.cpu_reference_run(64, 48, 1)
