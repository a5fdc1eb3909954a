"""Sweeps whose buffers do not fit the device: batches shrink until they do, with
the same results and no error left behind; what does not fit at all is an error,
after which the library works again.  TOMO_OPT_MEM_LIMIT stands in for a small
device."""
from __future__ import annotations

import numpy as np
import pytest

from tests.test_golden import bits
from tomo_shell2026_b200 import meshgen, native
from tomo_shell2026_b200.options import PrintOptions

pytestmark = pytest.mark.gpu

YPR = meshgen.ypr_grid(np.arange(0, 360, 15), np.arange(0, 70, 5))   # 336


@pytest.fixture(autouse=True)
def fresh_library():
    """No buffers of earlier calls before, no limit and no batch after."""
    native.Batch.release()
    native.lib().OnDestroy()
    yield
    native.set_option(native.TOMO_OPT_MEM_LIMIT, 0)
    native.Batch.release()
    native.lib().OnDestroy()


def _limits():
    return [int(2 ** (k / 2)) for k in range(25, 43)]   # 5.7 MiB to 1.4 GiB, in KiB


def test_shrunk_sweeps_match_and_leave_no_error():
    m = meshgen.perturbed_sphere(3000, 60.0, 8, with_hull=False)
    opts = PrintOptions(explicit_ss=False)
    ref = native.sweep(m, YPR, opts)
    shrunk = refused = 0
    for kib in _limits():
        native.lib().OnDestroy()
        native.set_option(native.TOMO_OPT_MEM_LIMIT, kib)
        try:
            got = native.sweep(m, YPR, opts)
        except native.TomoError:
            refused += 1
            native.set_option(native.TOMO_OPT_MEM_LIMIT, 0)
            got = native.sweep(m, YPR, opts)   # nothing of the refusal is left
        else:
            shrunk += native.kernel_log()["k_raster"]["launches"] > 2 + 1   # two batches and the export
        assert native.lib().tomoGetLastError() == 0 and native.lib().tomoGetLastErrorString() == b"", kib
        for k in ("Mo", "Mss", "Vtc", "VoF", "VssF"):
            assert np.array_equal(bits(getattr(got, k)), bits(getattr(ref, k))), (kib, k)
        assert np.array_equal(got.Vss64, ref.Vss64) and got.optID == ref.optID
    assert shrunk > 0 and refused > 0


def test_shrunk_batches_keep_every_mesh_in_place():
    """One workspace for meshes of different needs: a mesh whose batch shrinks must
    not leave an earlier one short (its capture would have to allocate)."""
    opts = PrintOptions()
    meshes = [meshgen.perturbed_icosphere(2, 30.0, 11, with_hull=False),
              meshgen.perturbed_sphere(20000, 55.0, 12, with_hull=False),
              meshgen.perturbed_icosphere(3, 140.0, 13, with_hull=False)]
    refs = [native.sweep(m, YPR, opts) for m in meshes]
    shrunk = 0
    for order in ((0, 1, 2), (2, 1, 0)):
        for kib in _limits():
            native.Batch.release()
            native.lib().OnDestroy()
            native.set_option(native.TOMO_OPT_MEM_LIMIT, kib)
            try:
                b = native.Batch([meshes[i] for i in order], [YPR] * 3, opts, autotune=False)
                for _ in range(2):   # the capture and a replay
                    b.run()
            except native.TomoError as e:
                assert "out of memory" in str(e), (kib, e)
                continue
            assert native.lib().tomoGetLastError() == 0
            shrunk += any(b.config(k)["batch"] < 256 for k in range(3))
            for k, i in enumerate(order):
                got = b.results(k)
                assert np.array_equal(bits(got["Mss"]), bits(refs[i].Mss)), (kib, i)
                assert np.array_equal(got["Vss64"], refs[i].Vss64) and got["optID"] == refs[i].optID
    assert shrunk > 0
