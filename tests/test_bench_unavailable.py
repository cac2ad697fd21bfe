"""bench.py --impl reference where the reference has not been compiled: one line that says so, and exit code 0."""
import json
import sys
from pathlib import Path

REPO = Path(__file__).resolve().parent.parent


def test_reference_arm_without_the_reference(monkeypatch, capsys):
    monkeypatch.syspath_prepend(str(REPO))
    import bench
    import oracle

    def missing(*a, **k):
        raise OSError("libref_ops_fast.so: cannot open shared object file")

    monkeypatch.setattr(oracle, "RefStepper", missing)
    monkeypatch.setattr(oracle, "RefStripStepper", missing)
    monkeypatch.delenv("RANK", raising=False)
    args = type("A", (), dict(gpus=1, steps=1, warmup=3, workload="batch600"))()
    assert bench.run_reference(args) == 0
    line = json.loads(capsys.readouterr().out)
    assert line["impl"] == "reference" and "not compiled" in line["unavailable"]
