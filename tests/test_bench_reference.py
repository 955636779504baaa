"""bench.py --impl reference where the reference's programs are not built: one line
that says so, and nothing of this repository timed in their place."""
import json
import os
import sys
import types

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_unavailable_without_the_programs(monkeypatch, capsys):
    sys.path.insert(0, ROOT)
    import bench

    def timed(*a):
        raise AssertionError("a CPU run in the reference's place")
    monkeypatch.setattr(bench, "_ref_bins", lambda: ("oracle_cli", "oracle_cli", "port"))
    monkeypatch.setattr(bench, "cpu_round_trip", timed)
    bench.run_reference(types.SimpleNamespace(gpus=1, steps=1, warmup=1), 0, 1)
    line = json.loads(capsys.readouterr().out)
    assert line["impl"] == "reference" and line["unavailable"] and "value" not in line
