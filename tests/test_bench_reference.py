"""The benchmark's reference arm where the reference's kernel builds are absent: the CPU port's baselines."""
import argparse
import itertools

import bench


def test_cpu_port_arm(monkeypatch):
    values = itertools.count(1.0)
    monkeypatch.setattr(bench, "_ref_libs", lambda: None)
    monkeypatch.setattr(bench, "cpu_baseline_c1", lambda *a: ({"value": next(values), "kind": "port"}, None))
    out = bench.run_reference(argparse.Namespace(steps=3, warmup=2), 1, 0, 0, None)
    assert out["warmup"] == 2 and out["value"] == 4.0 and out["impl"] == "reference"      # the median of the timed ones: 3, 4, 5
    assert out["cpu_baseline"] == {"value": 4.0, "kind": "port"}
