"""Strip plans (Engine::plan_strips, adapt_after): the height a caller forces is the
height that runs, and results never depend on the plan."""
from __future__ import annotations

import numpy as np
import pytest

from tests.test_golden import bits
from tomo_shell2026_b200 import meshgen, native
from tomo_shell2026_b200.options import PrintOptions

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def default_options():
    yield
    for key, value in ((native.TOMO_OPT_STRIP_H, 0), (native.TOMO_OPT_BATCH, 256), (native.TOMO_OPT_NORMAL_SMEM, 0)):
        native.set_option(key, value)


def plates(n, a=200.0, b=140.0, gap=3.0):
    """n thin plates above one another: 2 n pixels in every column."""
    box = np.array([(0, 2, 1), (0, 3, 2), (4, 5, 6), (4, 6, 7), (0, 1, 5), (0, 5, 4), (1, 2, 6), (1, 6, 5), (2, 3, 7),
                    (2, 7, 6), (3, 0, 4), (3, 4, 7)])
    v = [(x, y, gap * k + z) for k in range(n) for z in (0.0, 1.0) for x, y in ((0, 0), (a, 0), (a, b), (0, b))]
    return meshgen.mesh_from_arrays(np.array(v, float), np.vstack([box + 8 * k for k in range(n)]), "plates",
                                    with_hull=False)


def _same(got, ref):
    for k in ("Mo", "Mss", "Vtc", "VoF", "VssF"):
        assert np.array_equal(bits(getattr(got, k)), bits(getattr(ref, k))), k
    assert np.array_equal(got.Vss64, ref.Vss64) and got.optID == ref.optID


@pytest.mark.parametrize("h,scale", [(8, 1.0), (8, 2.4), (8, 2.7), (4, 5.3)])
def test_forced_height_runs(h, scale):
    """Grids whose forced strips need fewer CTAs per SM than the default plan's."""
    m = meshgen.perturbed_sphere(2000, 100.0, 5, scale=scale, with_hull=False)
    ypr = meshgen.ypr_grid([0.0, 70.0], [0.0, 40.0])
    ref = native.sweep(m, ypr, PrintOptions())
    native.set_option(native.TOMO_OPT_STRIP_H, h)
    got = native.sweep(m, ypr, PrintOptions())
    st = native.stats()
    assert h * st["grid"] <= 5900
    assert st["strip_h"] == h and st["overflow_reruns"] == 0
    _same(got, ref)


@pytest.mark.parametrize("h", [2, 8])
def test_adaptation_keeps_a_forced_height(h):
    m = plates(7)
    ypr = np.ascontiguousarray(meshgen.ypr_grid(np.arange(0, 20, 0.25), [0.0, 3.0]))   # 160
    ref = native.sweep(m, ypr, PrintOptions())
    native.set_option(native.TOMO_OPT_STRIP_H, h)
    native.set_option(native.TOMO_OPT_BATCH, 32)
    s = native.Session(m, ypr, PrintOptions())
    for _ in range(2):   # the second sweep starts where the first adapted to
        s.run_device()
        assert native.stats()["strip_h"] == h
        assert np.array_equal(bits(s.finish()[2]), bits(ref.Mss))


@pytest.mark.parametrize("radius", [1160.0, 1500.0])
def test_wide_grids_hold_a_solid(radius):
    """One-column strips of a grid far wider than the reference's: a part that fills
    it is not run twice."""
    m = meshgen.perturbed_icosphere(4, radius, 5, with_hull=False)
    ypr = meshgen.ypr_grid([0.0, 50.0], [0.0, 40.0])
    got = native.sweep(m, ypr, PrintOptions())
    st = native.stats()
    assert st["grid"] > 2500 and st["strip_h"] == 1 and st["overflow_reruns"] == 0
    native.set_option(native.TOMO_OPT_NORMAL_SMEM, 150528)
    _same(got, native.sweep(m, ypr, PrintOptions()))


def test_adaptation_steps_are_worth_a_check():
    """One-column strips that hold a few pixels too few: the first check of the sweep
    already gets the rest of it through (up to the next budget's own room)."""
    m = plates(22, 140.0, 200.0)   # 8,800 pixels and more in a column of the grid
    ypr = np.ascontiguousarray(meshgen.ypr_grid(np.arange(0, 10, 0.25), [0.0, 1.0, 2.0]))   # 120
    ref = native.sweep(m, ypr, PrintOptions())
    native.set_option(native.TOMO_OPT_STRIP_H, 1)
    native.set_option(native.TOMO_OPT_BATCH, 30)
    got = native.sweep(m, ypr, PrintOptions())
    assert 0 < native.stats()["overflow_reruns"] <= 30
    _same(got, ref)


@pytest.mark.parametrize("far", [5.0e3, 3.0e9, 1.0e20, 3.0e38])
def test_meshes_beyond_any_grid_are_refused(far):
    """Extents past the largest grid, also those whose span is no int."""
    m = plates(1, 30.0, 20.0)
    v = m.vertices.copy()
    v[0, 0] = far
    bad = meshgen.MeshArrays(v, m.faces, m.vertex_normals, m.face_normals, m.area)
    ypr = meshgen.ypr_grid([0.0, 30.0], [0.0])
    with pytest.raises(native.TomoError, match="mesh extent exceeds the supported slot grid"):
        native.sweep(bad, ypr, PrintOptions())
    with pytest.raises(native.TomoError, match="above the static limit"):
        native.sweep_static(bad, ypr, PrintOptions())
