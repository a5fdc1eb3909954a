"""The rasterizer's candidate masks (tomo_shell2026_b200/csrc/tomo_span.cuh) on
the host: tests/mask_check.cpp compiles the same header with g++ (IEEE single
precision, no contraction) and, for random small, large, sliver, axis-aligned
and almost collinear triangles, checks that every box pixel the reference's
barycentric test accepts is a candidate.  The exact test runs on candidates
only, so this is the masks' exactness condition."""
from __future__ import annotations

import shutil
import subprocess
from pathlib import Path

import pytest

HERE = Path(__file__).resolve().parent


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
@pytest.mark.parametrize("seed", [21, 22])
def test_masks_hold_every_accepted_pixel(tmp_path, seed):
    exe = tmp_path / "mask_check"
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-fno-fast-math", str(HERE / "mask_check.cpp"),
                    "-o", str(exe)], check=True)
    out = subprocess.run([str(exe), "100000", str(seed)], capture_output=True, text=True)
    m = dict(zip(*[iter(out.stdout.strip().splitlines()[-1].split())] * 2))
    assert out.returncode == 0 and int(m["violations"]) == 0, out.stdout[-2000:]
    accepted, cand, box = int(m["accepted"]), int(m["candidates"]), int(m["pixels"])
    # the masks hold every accepted pixel and little else
    assert 0 < accepted <= cand < 0.5 * box


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_masks_at_any_pixel_size(tmp_path):
    """tests/mask_range_check.cpp: the masks' cell grid stays within the pixel box
    and holds every accepted pixel, for pixel sizes up to the largest float."""
    exe = tmp_path / "mask_range_check"
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-fno-fast-math", "-fwrapv",
                    str(HERE / "mask_range_check.cpp"), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe), "2000", "31"], capture_output=True, text=True)
    m = dict(zip(*[iter(out.stdout.strip().splitlines()[-1].split())] * 2))
    assert out.returncode == 0 and int(m["violations"]) == 0, out.stdout[-2000:]
    assert int(m["cases"]) > 10000 and int(m["accepted"]) > 10000
