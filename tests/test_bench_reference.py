"""bench.py --impl reference measures the reference's own functions or says that they are not
there; the restatement in oracle/ never stands in for them."""
import argparse
import importlib.util
import os

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_reference_arm_is_unavailable_without_the_reference(hb, monkeypatch):
    spec = importlib.util.spec_from_file_location("bench_under_test", os.path.join(ROOT, "bench.py"))
    bench = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(bench)
    import oracle
    monkeypatch.setattr(oracle, "ref_available", lambda: False)
    monkeypatch.setattr(bench, "cpu_run", lambda *a: pytest.fail("something was timed"))
    args = argparse.Namespace(width=64, height=64, streams=1, gop=2, batch=1, gpus=1, steps=1, warmup=0)
    line = bench.run_reference(args, hb, 0, 1)
    assert line["impl"] == "reference" and line["unavailable"] and "value" not in line
