"""bench.py --impl reference where the reference's library was not built: one JSON line that says so, exit status 0."""
import json
import sys

from conftest import ROOT


def test_unavailable(monkeypatch, capsys):
    import importlib.util
    import oracle
    spec = importlib.util.spec_from_file_location("bench_arm", ROOT / "bench.py")
    bench = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(bench)

    def missing(*a):
        raise FileNotFoundError("libltref.so not built")

    monkeypatch.setattr(oracle, "RefLib", missing)
    monkeypatch.setattr(sys, "argv", ["bench.py", "--impl", "reference", "--steps", "1"])
    assert bench.main() == 0
    line = json.loads(capsys.readouterr().out)
    assert line["impl"] == "reference" and "not built" in line["unavailable"]
