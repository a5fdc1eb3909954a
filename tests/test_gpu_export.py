"""The pixel export kernels against the column dump of the same orientation, on
the 256 grid and on a grid whose slots do not fill the last block: every type's
pixels in slot order, sentinels and support voxels included."""
from __future__ import annotations

import numpy as np
import pytest

from tomo_shell2026_b200 import meshgen, native
from tomo_shell2026_b200.options import PrintOptions

pytestmark = pytest.mark.gpu


def _expected(d):
    out = [[] for _ in range(11)]
    for sl in np.nonzero(d["cols"][:, 0])[0]:
        nd, nfin = d["cols"][sl, :2]
        k = d["keys"][sl, :nd].astype(np.int64)
        rows = [(int(t) if nd > 1 else 0, int(a >> 16) - 32768, int(a & 0xFFFF) - 32768)
                for t, a in zip(d["types"][sl, :nd], k)]
        rows += {2: [(8, 0, 0), (1024, 0, 0)], 1: [(int(d["cols"][sl, 6]), 0, 0)]}.get(int(nfin - nd), [])
        x, y = divmod(int(sl), d["G"])
        s0 = s1 = -1
        for t, z, nz in rows:
            for b in range(11):
                if b != 4 and (t >> b) & 1:
                    out[b].append((x, y, z, 0, 0, nz))
            s0, s1 = (z if t & 4 else s0), (z if t & 8 else s1)
            if s0 > -1 and s1 > -1:
                out[4] += [(x, y, zz, 0, 0, 0) for zz in range(s0, s1 - 1, -1)]
                s0 = s1 = -1
    return out


@pytest.mark.parametrize("explicit_ss", [True, False])
@pytest.mark.parametrize("scale", [1.0, 2.7])
def test_export_matches_column_dump(scale, explicit_ss):
    m = meshgen.perturbed_sphere(900, 45.0, 8, scale=scale, with_hull=False)
    ypr = np.array([[0.4, 1.1, 0.2]], np.float32)
    opts = PrintOptions(explicit_ss=explicit_ss)
    got = native.sweep(m, ypr, opts).pixels
    want = _expected(native.Session(m, ypr, opts).columns(0))
    for k in range(11):
        assert np.array_equal(got[k], np.array(want[k], np.int16).reshape(-1, 6)), f"type {k}"
