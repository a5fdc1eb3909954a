"""tomoSweepStatic re-runs what overflows its strips, and only that: the same
orientations as TomoSh_CUDA, whose strips hold as much."""
from __future__ import annotations

import numpy as np
import pytest

from tests.test_golden import bits
from tests.test_gpu_plan import plates
from tomo_shell2026_b200 import meshgen, native
from tomo_shell2026_b200.options import PrintOptions

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,a,b", [(1, 150.0, 150.0), (2, 150.0, 127.5), (2, 150.0, 150.0), (3, 120.0, 102.0)])
def test_static_reruns_as_many_as_the_sweep(n, a, b):
    m = plates(n, a, b, gap=10.0)
    ypr = meshgen.ypr_grid(np.arange(0, 360, 10), [0.0])   # 36: two whole batches and four
    opts = PrintOptions()
    ref = native.sweep(m, ypr, opts)
    want = native.stats()["overflow_reruns"]
    opt, Mo, Mss, Vtc = native.sweep_static(m, ypr, opts)
    st = native.stats()
    assert (st["static_overflow_reruns"], st["static_prio_reruns"], st["static_safe_reruns"]) == (want, 0, 0)
    assert opt == ref.optID
    for got, k in ((Mo, "Mo"), (Mss, "Mss"), (Vtc, "Vtc")):
        assert np.array_equal(bits(got), bits(getattr(ref, k))), k


@pytest.mark.parametrize("n,shell", [(3, False), (5, False), (9, True), (12, False), (28, False)])
def test_static_overflows_of_many_sizes(oracle, n, shell):
    """Re-runs of a few thousand pixels a strip (all of a batch's at once) up to as
    many as the large strips hold, against the oracle; past that the call refuses."""
    m = plates(n, 165.0, 120.0, gap=3.0)
    ypr = np.concatenate([meshgen.ypr_grid(np.arange(0, 360, 24), [0.0]), meshgen.ypr_grid([0.0, 40.0], [1.0, 90.0])])
    opts = PrintOptions(shell_mesh=shell, explicit_ss=not shell, bed_type=2 * shell, bed_outer=2.0, bed_thickness=0.9)
    if n == 28:
        with pytest.raises(native.TomoError, match="exceed the static scratch"):
            native.sweep_static(m, ypr, opts)
        return
    native.sweep(m, ypr, opts)
    ref = native.stats()
    want = oracle.sweep(m, ypr, opts)
    opt, Mo, Mss, Vtc = native.sweep_static(m, ypr, opts)
    st = native.stats()
    assert opt == want["optID"] and st["static_overflow_reruns"] > 0
    for k in ("overflow_reruns", "prio_reruns", "safe_reruns"):
        assert st["static_" + k] == ref[k], k
    for got, k in ((Mo, "Mo"), (Mss, "Mss"), (Vtc, "Vtc")):
        assert np.array_equal(bits(got), bits(np.asarray(want[k], np.float32))), k
