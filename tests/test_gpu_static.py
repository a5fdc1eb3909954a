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
