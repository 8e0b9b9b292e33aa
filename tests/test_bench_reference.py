"""bench.py --impl reference without the reference's host build: one line that
says so, no number of the oracle's restatement, exit code 0."""
import json
import sys

from conftest import ROOT


def test_unavailable(monkeypatch, capsys):
    monkeypatch.syspath_prepend(str(ROOT))
    import bench
    import pyoracle

    def absent(*a, **k):
        raise FileNotFoundError("oracle/_ref")

    monkeypatch.setattr(pyoracle, "Reference", absent)
    monkeypatch.delenv("RANK", raising=False)
    monkeypatch.setattr(sys, "argv", ["bench.py", "--impl", "reference", "--steps", "1", "--warmup", "0"])
    assert bench.main() in (0, None)
    line = json.loads(capsys.readouterr().out.strip().splitlines()[-1])
    assert line["impl"] == "reference" and line["unavailable"] and "value" not in line
