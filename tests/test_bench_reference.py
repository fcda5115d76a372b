"""bench.py --impl reference times the reference's own code or says that it cannot: nothing of this repository stands in
for it."""
import json
import sys

from oracle.api import Oracle, Reference


def test_unavailable_reference_is_not_replaced(monkeypatch, capsys):
    import bench

    def none(*_):
        raise AssertionError("the oracle stands in for the reference")

    monkeypatch.setattr(Reference, "available", staticmethod(lambda: False))
    monkeypatch.setattr(Oracle, "accel", none)
    monkeypatch.setattr(sys, "argv", ["bench.py", "--impl", "reference", "--steps", "1", "--warmup", "0", "--rays", "100",
                                      "--subdiv", "2", "--nrandom", "10"])
    monkeypatch.delenv("RANK", raising=False)
    assert bench.main() == 0
    line = json.loads(capsys.readouterr().out.strip())
    assert line["impl"] == "reference" and line["unavailable"] and "value" not in line


def test_other_ranks_print_nothing(monkeypatch, capsys):
    import bench
    monkeypatch.setattr(sys, "argv", ["bench.py", "--impl", "reference", "--gpus", "2"])
    monkeypatch.setenv("RANK", "1")
    assert bench.main() == 0 and capsys.readouterr().out == ""
