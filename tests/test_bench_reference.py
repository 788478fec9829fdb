"""bench.py --impl reference times the reference's own code or says that it cannot: the
package's CPU checker does not stand in for it (no GPU)."""

import json
import types

import bench
from oracle import ref


def test_reference_arm_without_the_reference(monkeypatch, capsys):
    monkeypatch.setattr(ref, "available", lambda: False)
    args = types.SimpleNamespace(gpus=1, steps=1, warmup=0, events=4, cpu_sample_points=1000)
    assert bench.run_reference(args, 1, 0) == 0
    lines = capsys.readouterr().out.strip().splitlines()
    assert len(lines) == 1
    line = json.loads(lines[0])
    assert line["impl"] == "reference" and line["unavailable"] and "value" not in line
    assert bench.run_reference(args, 2, 1) == 0  # other ranks print nothing
    assert capsys.readouterr().out == ""
