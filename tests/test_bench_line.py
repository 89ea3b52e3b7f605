"""bench.py prints its line without the reference's CPU harness (a clone on which it was never built): the CPU baseline is
reported as failed and everything else is measured."""
import json
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_baseline_that_cannot_start_is_reported(monkeypatch):
    import bench
    from oracle import refio
    monkeypatch.setattr(refio, "harness_available", lambda *a: False)
    monkeypatch.setattr(bench, "SAMPLE_NX", 8)
    monkeypatch.setattr(bench, "SAMPLE_NY", 4)
    run, said = bench.begin_cpu_baseline(3)
    assert run is None and said["value"] is None and said["sample"].startswith("failed: ") and "harness" in said["sample"]


@pytest.mark.gpu
def test_line_without_the_harness():
    code = ("import sys; sys.argv = ['bench.py', '--nx', '120', '--ny', '30', '--steps', '1', '--warmup', '3']\n"
            "from oracle import refio; refio.harness_available = lambda *a: False\n"
            "import bench; bench.main()")
    r = subprocess.run([sys.executable, "-c", code], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    lines = [ln for ln in r.stdout.splitlines() if ln.startswith("{")]
    assert len(lines) == 1
    out = json.loads(lines[0])
    assert out["cpu_baseline"]["value"] is None and "harness" in out["cpu_baseline"]["sample"]
    for key in ("metric", "value", "unit", "n_gpus", "steps", "warmup", "ms_per_step", "e2e", "gpu_launches", "roofline", "clocks"):
        assert key in out, key
    assert out["e2e"]["h2d_bytes_per_step"] > 0 and out["gpu_launches"] > 0
