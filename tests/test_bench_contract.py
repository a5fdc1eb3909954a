"""bench.py's reference arm runs on the CPU: its JSON line must carry the
contract's keys (the GPU arm is exercised on a B200)."""
from __future__ import annotations

import json
import subprocess
import sys
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]


def test_reference_arm_line():
    from oracle import build
    if build.build_ref() is None:
        pytest.skip("reference engine library not available")
    out = subprocess.run([sys.executable, str(ROOT / "bench.py"), "--impl", "reference", "--steps", "1",
                          "--warmup", "1", "--ref-step-s", "1.5"], cwd=ROOT, capture_output=True, text=True,
                         timeout=600)
    assert out.returncode == 0, out.stderr[-2000:]
    line = json.loads(out.stdout.strip().splitlines()[-1])
    for k in ("metric", "value", "unit", "n_gpus", "steps", "warmup", "ms_per_step", "higher_is_better", "scaling",
              "vs_baseline", "dtype", "data", "config", "impl", "cpu_baseline", "e2e"):
        assert k in line, k
    assert line["impl"] == "reference" and line["value"] > 0
    assert line["e2e"]["h2d_bytes_per_step"] == 0 and line["e2e"]["d2h_bytes_per_step"] == 0
    assert line["cpu_baseline"]["kind"] in ("reference", "port") and line["cpu_baseline"]["cores"] >= 1
    assert line["config"]["workload"] == "solid82k_1deg"


def test_roofline_rate_is_one_the_device_ran_at():
    """k_raster and k_columns overlap: spans of 100 and 60 ms in a sweep of 110 ms
    moved their bytes in 110 ms."""
    import importlib.util
    spec = importlib.util.spec_from_file_location("bench", ROOT / "bench.py")
    bench = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(bench)
    klog = {"k_raster": dict(launches=10, ms=100.0, timed=10), "k_strip": dict(launches=10, ms=60.0, timed=10)}
    r = bench._rates(klog, 110e6, 110.0)
    assert r["achieved"] == pytest.approx(1.0) and r["avg_launch_ms"] == pytest.approx(11.0)
    assert r["bytes_per_launch"] == pytest.approx(11e6)
