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


def test_port_baseline_of_an_electrolyte_is_the_electrolyte_step(no_reference, monkeypatch):
    seen = _steps_of(monkeypatch, spm.SpmOracle)
    monkeypatch.setattr(spm.ElectrolyteOracle, "__init__", lambda self, cfg: None)
    monkeypatch.setattr(spm.ElectrolyteOracle, "run", lambda self, n: seen.append(("ElectrolyteOracle", n)))
    cb = bench.cpu_baseline(udf.electrolyte_config((4, 4, 4), 1, seed=1, a=3.0), warmup=1, steps=2)
    assert seen == [("ElectrolyteOracle", 1), ("ElectrolyteOracle", 2)] and cb["kind"] == "port"


def test_no_port_baseline_of_the_sheared_step(no_reference, monkeypatch):
    # the numpy restatement has no Lees-Edwards step: its Navier-Stokes one is
    # another workload
    seen = _steps_of(monkeypatch, spm.SpmOracle)
    cb = bench.cpu_baseline(workload.shear_le_128_256(), warmup=1, steps=2)
    assert set(cb) == {"unavailable"} and not seen


def test_batch_baseline_carries_the_kind_and_cores_of_its_runs(monkeypatch):
    boxes = [{"np_xyz": (5, 5, 5)}, {"np_xyz": (6, 6, 6)}, {"np_xyz": (5, 5, 5)}]
    for kind, cores in (("port", 1), ("reference", 7)):
        monkeypatch.setattr(bench, "cpu_baseline", lambda c, warmup, steps: {"value": 2.0, "kind": kind, "cores": cores})
        cb = bench.cpu_baseline_batch(boxes)
        assert (cb["kind"], cb["cores"]) == (kind, cores) and cb["value"] == pytest.approx(2.0 / 3, abs=1e-5)
        assert ("OpenMP" in cb["sample"]) == (kind == "reference")
