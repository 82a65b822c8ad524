"""What bench.py calls a reference or a baseline is what it timed."""
import argparse
import os

import pytest

import bench
from kapsel_old_b200 import workload
from oracle import ref, spm, udf


@pytest.fixture
def no_reference(monkeypatch, tmp_path):
    monkeypatch.setattr(ref, "REF_DIR", str(tmp_path))


def _steps_of(monkeypatch, cls):
    """Counts the steps of an oracle class in place of taking them."""
    seen = []
    monkeypatch.setattr(cls, "__init__", lambda self, cfg: None)
    monkeypatch.setattr(cls, "run", lambda self, n: seen.append((cls.__name__, n)))
    return seen


def test_reference_arm_without_a_reference_build_is_unavailable(no_reference, monkeypatch):
    monkeypatch.setattr(spm, "SpmOracle", None)  # the restatement is not the reference
    line = bench.run_reference(argparse.Namespace(steps=2, warmup=3))
    assert set(line) == {"impl", "unavailable"} and line["impl"] == "reference"
    assert "\n" not in line["unavailable"]
