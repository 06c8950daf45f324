"""bench.py --impl reference measures the reference or says why it cannot: the
oracle's restatement is never timed in its place."""
from __future__ import annotations

import argparse
import json

import pytest


@pytest.fixture
def bench(oracle, monkeypatch, tmp_path):
    import bench as B

    oracle.lib()
    monkeypatch.setattr(oracle, "_REF_DIR", str(tmp_path))  # no compiled harness here ...
    monkeypatch.setattr(oracle, "_ref", None)
    monkeypatch.setenv("HPMC_SRC", str(tmp_path))  # ... and no tree
    return B


def test_unavailable_without_the_harness(bench, capsys):
    bench.run_reference(argparse.Namespace(lattice=16, steps=1, warmup=1), 0, 1)
    line = json.loads(capsys.readouterr().out)
    assert line["impl"] == "reference" and "value" not in line
    assert "reference harness not built" in line["unavailable"] and "\n" not in line["unavailable"]


def test_only_rank_0_prints(bench, capsys):
    bench.run_reference(argparse.Namespace(lattice=16, steps=1, warmup=1), 1, 2)
    assert capsys.readouterr().out == ""
