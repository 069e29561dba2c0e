"""bench.py where an optional CPU library is missing: our arm's line keeps its
GPU results, the reference arm says why it is unavailable."""
import json
import os
import sys
import types

import pytest

import oracle_lib

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))


@pytest.fixture
def bench(monkeypatch):
    import bench as b

    def missing(*a, **k):
        raise FileNotFoundError("library not built")

    monkeypatch.setattr(oracle_lib, "RefLib", missing)
    return b, lambda: monkeypatch.setattr(oracle_lib, "Oracle", missing)


def test_cpu_baseline_needs_no_reference_library(bench, monkeypatch):
    b, _ = bench
    import inspire_b200 as ib
    monkeypatch.setattr(b, "host_mem_available", lambda: None)
    cq = b.cpu_baseline(ib, 256, 120, timed=1)
    assert cq["value"] > 0 and cq["kind"] == "port", cq


def test_cpu_baseline_without_the_oracle(bench):
    b, no_oracle = bench
    no_oracle()
    import inspire_b200 as ib
    assert "not built" in b.cpu_baseline(ib, 256, 120)["unavailable"]


def test_reference_arm_without_its_library(bench, capsys):
    b, _ = bench
    b.run_reference(types.SimpleNamespace(n_entries=256, entry_bytes=120, warmup=0, steps=1, batch=1))
    line = json.loads(capsys.readouterr().out)
    assert line["impl"] == "reference" and "not built" in line["unavailable"]
