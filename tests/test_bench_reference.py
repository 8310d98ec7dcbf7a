"""bench.py where the reference library has not been built: the reference arm
says so on its one line, and the sections that would time it lose their own
field only."""
import argparse
import json
import os
import sys

from conftest import ROOT

sys.path.insert(0, ROOT)
import bench  # noqa: E402


def test_missing_reference(monkeypatch, capsys, tmp_path):
    monkeypatch.setattr(bench, "REF_OPENBLAS", str(tmp_path / "none.so"), raising=False)
    monkeypatch.setattr(bench, "host_threads", lambda: 1)
    monkeypatch.setitem(sys.modules, "refbind", None)  # not reached
    bench.run_reference(argparse.Namespace(n=64, warmup=1, steps=1, gpus=1), 0)
    line = json.loads(capsys.readouterr().out.strip())
    assert line["impl"] == "reference" and line["unavailable"]
    assert "unavailable" in bench.reference_ir_cpu("spd", None, None)
