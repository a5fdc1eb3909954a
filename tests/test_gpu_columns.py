"""The column stage (k_columns) where its classes meet: stacks of n sheets put n
raw pixels in a column and up to 2 n along the sheets' diagonals -- one or two
(closed form), up to 32 (several columns side by side in a warp), up to 128 (a
warp per column), longer, and either side of the 63-pixel cap.  Bit for bit
against the oracle, with the bed's last-pixel bookkeeping on and off."""
from __future__ import annotations

import numpy as np
import pytest

from tomo_shell2026_b200 import meshgen, native
from tomo_shell2026_b200.options import BED_NONE, BED_RAFT, PrintOptions

pytestmark = pytest.mark.gpu


def _stack(n, seed):
    """n sheets over one another, wound up or down by a seeded choice, a few of
    them doubled (equal keys) and a few tilted."""
    rng = np.random.default_rng(seed)
    V, F = [], []
    for k in range(n):
        w = rng.uniform(4.0, 9.0)
        z = 1.25 * (k if k % 7 else max(k - 1, 0))
        t = rng.uniform(-0.6, 0.6) if k % 5 == 0 else 0.0
        b = len(V)
        V += [(0.3, 0.2, z), (0.3 + w, 0.2, z + t), (0.3 + w, 0.2 + w, z), (0.3, 0.2 + w, z - t)]
        f = [(b, b + 1, b + 2), (b, b + 2, b + 3)]
        F += f if rng.random() < 0.5 else [t3[::-1] for t3 in f]
    return meshgen.mesh_from_arrays(np.array(V), np.array(F), f"stack{n}", with_hull=False)


@pytest.mark.parametrize("bed", [BED_NONE, BED_RAFT])
@pytest.mark.parametrize("explicit_ss", [True, False])
@pytest.mark.parametrize("n", [1, 2, 3, 16, 17, 31, 33, 62, 64, 65, 127, 129, 150])
def test_column_classes(oracle, n, explicit_ss, bed):
    m = _stack(n, n)
    ypr = meshgen.ypr_grid([0.0, 0.7, 90.0, 183.0], [0.0, 1.1, 35.0])
    opts = PrintOptions(explicit_ss=explicit_ss, bed_type=bed, bed_outer=2.0 if bed else 0.0,
                        bed_thickness=0.97 if bed else 0.0)
    got, want = native.sweep(m, ypr, opts), oracle.sweep(m, ypr, opts)
    for k in ("Vo64", "Vss64", "Vtc64"):
        assert np.array_equal(getattr(got, k), want[k]), k
    for k in ("Mo", "Mss", "Vtc"):
        assert np.array_equal(getattr(got, k).view(np.int32), np.asarray(want[k], np.float32).view(np.int32)), k
    assert got.optID == want["optID"]
