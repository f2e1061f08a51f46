"""bench.py's host baseline: the reference's figure where its library was built,
a reason in its place where it was not (the line is printed either way)."""
import importlib.util
import os

import pytest

from conftest import ROOT


@pytest.fixture(scope="module")
def bench():
    spec = importlib.util.spec_from_file_location("bench", os.path.join(ROOT, "bench.py"))
    m = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(m)
    return m


class _Workload:
    def cpu_reference(self, seconds, threads):
        return 12.3456, threads, f"a sample of {seconds} s", 1.0


def test_without_the_reference_library(bench, monkeypatch):
    from oracle.pyoracle import Reference
    monkeypatch.setattr(Reference, "available", staticmethod(lambda sse=False: False))
    got = bench.host_baseline(_Workload(), 2.0, 8)
    assert "libmanta_ref.so" in got["unavailable"] and "value" not in got


def test_with_it(bench, monkeypatch):
    from oracle.pyoracle import Reference
    monkeypatch.setattr(Reference, "available", staticmethod(lambda sse=False: not sse))
    assert bench.host_baseline(_Workload(), 2.0, 8) == {
        "value": 12.346, "unit": "Mrays/s", "cores": 8, "kind": "reference",
        "sample": "a sample of 2.0 s"}
