"""Bed pixel counts (k_bed) for windows on either side of the 31-pixel limit of
the ballot scan, at the grid's edges, against the oracle (the bed's mass is part
of Mss, and every bed pixel of the best orientation is exported)."""
from __future__ import annotations

import numpy as np
import pytest

from tomo_shell2026_b200 import meshgen, native
from tomo_shell2026_b200.options import BED_BRIM, BED_RAFT, BED_SKIRT, PrintOptions

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("outer,inner", [(1.0, 0.0), (2.9, 1.0), (8.0, 3.5), (31.0, 12.0), (33.0, 30.0)])
@pytest.mark.parametrize("bed", [BED_BRIM, BED_RAFT, BED_SKIRT])
def test_bed_windows(oracle, bed, outer, inner):
    m = meshgen.perturbed_sphere(320, 24.0, 4, with_hull=False)
    ypr = meshgen.ypr_grid([0.0, 40.0, 115.0], [0.0, 33.0])
    opts = PrintOptions(bed_type=bed, bed_inner=inner, bed_outer=outer, bed_thickness=0.7)
    got, want = native.sweep(m, ypr, opts), oracle.sweep(m, ypr, opts)
    assert np.array_equal(got.Mss.view(np.int32), np.asarray(want["Mss"], np.float32).view(np.int32))
    assert got.optID == want["optID"]
    assert got.n_bed[got.optID] == got.pixels[5].shape[0] and got.n_bed.min() > 0


@pytest.mark.parametrize("bed", [-1, 4, 77])
@pytest.mark.parametrize("outer", [3.0, 33.0])
def test_unknown_bed_type_lays_no_bed(oracle, bed, outer):
    """A bed type that is none of brim, raft and skirt has no candidate pixel
    (IsBedCandidate, STomoSh_INT3.cpp:1331-1373), for either window scan."""
    m = meshgen.perturbed_sphere(320, 24.0, 4, with_hull=False)
    ypr = meshgen.ypr_grid([0.0, 40.0, 115.0], [0.0, 33.0])
    opts = PrintOptions(bed_type=bed, bed_outer=outer, bed_thickness=0.7)
    got, want = native.sweep(m, ypr, opts), oracle.sweep(m, ypr, opts)
    assert got.n_bed.max() == 0 and got.pixels[5].shape[0] == 0
    assert np.array_equal(got.Mss.view(np.int32), np.asarray(want["Mss"], np.float32).view(np.int32))
