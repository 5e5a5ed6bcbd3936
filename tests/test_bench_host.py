"""bench.py on a machine without the reference's CPU build (no GPU needed): the arms that time it say so
and the run goes on."""
from __future__ import annotations

import argparse
import json
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]


@pytest.fixture
def bench(monkeypatch, tmp_path):
    monkeypatch.syspath_prepend(str(ROOT))
    import bench as module
    from oracle import oracle as O

    monkeypatch.setattr(O, "REF_FAST_SO", tmp_path / "libcfdref_fast.so")
    monkeypatch.setattr(O, "REF_CLI", tmp_path / "cfd-bench")
    monkeypatch.setattr(O, "_ref", {})
    return module


def test_cpu_baselines_report_a_missing_build(bench):
    assert "libcfdref_fast.so" in bench.cpu_solid_baseline()["unavailable"]
    assert "cfd-bench" in bench.cpu_inplace_baselines()["unavailable"]


def test_reference_arm_reports_a_missing_build(bench, capsys):
    args = argparse.Namespace(gpus=1, steps=20, warmup=5, n=512)
    assert bench.run_reference_arm(args, 1, 2) == 0 and capsys.readouterr().out == ""
    assert bench.run_reference_arm(args, 0, 1) == 0
    line = json.loads(capsys.readouterr().out)
    assert line["impl"] == "reference" and "libcfdref_fast.so" in line["unavailable"]
