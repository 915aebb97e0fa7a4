"""bench.py's reference arm times the reference's own build or nothing: without
it the arm says so on one line, and never times this repository's restatement."""
import json
import os
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_reference_arm_without_the_reference_build(monkeypatch, capsys, tmp_path, oracle_lib):
    monkeypatch.syspath_prepend(ROOT)
    import bench
    monkeypatch.setattr(oracle_lib, "reference_bench_binary", lambda: (str(tmp_path / "absent"), "x86-64-v3"))
    monkeypatch.setattr(sys, "argv", ["bench.py", "--impl", "reference", "--edge", "8", "--steps", "2", "--warmup", "1"])
    bench.main()
    lines = capsys.readouterr().out.splitlines()
    assert len(lines) == 1
    rec = json.loads(lines[0])
    assert rec["impl"] == "reference" and rec["unavailable"] and "value" not in rec
