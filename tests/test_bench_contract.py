"""bench.py's reference arm (Banshee's own CPU tracer, oracle/_ref) prints the
one JSON line the benchmark contract asks for; runs on CPU."""
import json
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_reference_arm_json_line():
    from oracle import oracle
    if not oracle.available("ref"):
        pytest.skip("oracle/_ref not built")
    out = subprocess.run([sys.executable, os.path.join(ROOT, "bench.py"), "--impl", "reference", "--steps", "2",
                          "--warmup", "3", "--ref-rows", "2"], capture_output=True, text=True, timeout=600, cwd=ROOT)
    assert out.returncode == 0, out.stderr[-2000:]
    lines = [l for l in out.stdout.splitlines() if l.startswith("{")]
    assert len(lines) == 1
    d = json.loads(lines[0])
    assert d["impl"] == "reference" and d["metric"] == "Msamples/s at 1080p" and d["unit"] == "Msamples/s"
    assert d["higher_is_better"] is True and d["n_gpus"] == 1 and d["steps"] == 2 and d["warmup"] == 3
    assert d["value"] > 0 and d["cpu_baseline"]["value"] == d["value"]
    assert d["cpu_baseline"]["kind"] == "reference" and d["cpu_baseline"]["cores"] >= 1
    assert d["e2e"] == {"value": d["value"], "unit": "Msamples/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0}
    assert d["config"]["workload"].startswith("C3")


def test_reference_arm_without_the_reference(monkeypatch, capsys):
    """Where the reference is not built the arm says so in one line and exits with 0."""
    import argparse
    import bench
    from oracle import oracle
    monkeypatch.setattr(oracle, "REF_SO", os.path.join(ROOT, "oracle", "no_such_library.so"))
    rc = bench.run_reference_arm(argparse.Namespace(gpus=1, steps=2, warmup=3, ref_rows=2), 0)
    lines = capsys.readouterr().out.splitlines()
    assert rc == 0 and len(lines) == 1
    d = json.loads(lines[0])
    assert d["impl"] == "reference" and d["unavailable"] and set(d) == {"impl", "unavailable"}
