"""Strip plans (Engine::plan_strips): the height a caller forces is the
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
