"""bench.py's reference arm runs on the host cores only, so its JSON line can
be checked without a GPU: one line, the contract's keys, the reference's own
kernels (kind "reference") and a zero-copy e2e object."""
import json
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_reference_arm_json_line():
    from oracle import build as ob
    try:
        if ob.build_ref() is None:
            pytest.skip("reference kernel sections not available")
    except Exception as e:  # no reference sources on this machine
        pytest.skip("reference host build unavailable: %s" % e)
    r = subprocess.run([sys.executable, "bench.py", "--impl", "reference", "--steps", "1", "--warmup", "1"],
                       cwd=ROOT, capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stderr[-2000:]
    lines = [l for l in r.stdout.splitlines() if l.startswith("{")]
    assert len(lines) == 1
    d = json.loads(lines[0])
    for k in ("metric", "value", "unit", "n_gpus", "steps", "warmup", "ms_per_step", "higher_is_better",
              "scaling", "vs_baseline", "dtype", "data", "config", "cpu_baseline", "e2e"):
        assert k in d, k
    assert d["impl"] == "reference"
    assert d["metric"] == "Westervelt Gcell-updates/s" and d["higher_is_better"] is True
    assert d["value"] > 0 and d["steps"] == 1 and d["warmup"] == 1
    assert d["cpu_baseline"]["kind"] == "reference" and d["cpu_baseline"]["value"] == d["value"]
    assert d["e2e"]["value"] == d["value"] and d["e2e"]["h2d_bytes_per_step"] == 0
    assert d["config"]["workload"]


@pytest.mark.parametrize("cause", ["no sources", "no compiler"])
def test_reference_arm_without_the_reference_reports_no_number(monkeypatch, capsys, cause):
    """Where the reference's kernels cannot be built, the arm says so and times nothing in
    their place."""
    import argparse

    import bench
    from oracle import build as ob

    def build_ref(*a, **k):
        if cause == "no sources":
            return None
        raise RuntimeError("command failed: g++\nsecond line")
    monkeypatch.setattr(ob, "build_ref", build_ref)
    bench.run_reference(argparse.Namespace(gpus=1, steps=1, warmup=1), 1, 0)
    lines = capsys.readouterr().out.splitlines()
    assert len(lines) == 1
    d = json.loads(lines[0])
    assert d["impl"] == "reference" and d["unavailable"] and "\n" not in d["unavailable"]
    assert "value" not in d and "e2e" not in d
