"""The triangle-centric rasterizer (k_raster) at the sizes where its work split
changes: triangle counts around a warp's 32, too few triangles to fill the chip
(several lanes per triangle), boxes of more cells than a lane takes (finished
by the whole warp), large and small triangles in one warp.  Bit for bit against
the oracle."""
from __future__ import annotations

import numpy as np
import pytest

from tomo_shell2026_b200 import meshgen, native
from tomo_shell2026_b200.options import PrintOptions

pytestmark = pytest.mark.gpu


def _cube(edge):
    v = np.array([[x, y, z] for x in (0, 1) for y in (0, 1) for z in (0, 1)], float) * edge
    f = [(0, 1, 3), (0, 3, 2), (4, 6, 7), (4, 7, 5), (0, 4, 5), (0, 5, 1), (2, 3, 7), (2, 7, 6), (0, 2, 6), (0, 6, 4),
         (1, 5, 7), (1, 7, 3)]
    return v, np.array(f)


def _mesh(kind):
    if kind == "cube":
        return meshgen.mesh_from_arrays(*_cube(110.0), with_hull=False)
    if kind == "cube_and_sphere":   # two kinds of triangles interleaved in every warp
        v, f = _cube(90.0)
        m = meshgen.perturbed_sphere(320, 30.0, 3, with_hull=False)
        g = m.faces + 8
        order = np.argsort(np.concatenate([np.arange(12) * 25.0, np.arange(g.shape[0])]), kind="stable")
        return meshgen.mesh_from_arrays(np.vstack([v, m.vertices + 40.0]), np.vstack([f, g])[order], with_hull=False)
    n = int(kind)
    m = meshgen.random_mesh(n, n, extent=90.0)
    return meshgen.mesh_from_arrays(m.vertices, m.faces, with_hull=False)


@pytest.mark.parametrize("n_ypr", [1, 9, 300])
@pytest.mark.parametrize("kind", ["cube", "cube_and_sphere", "1", "31", "33", "257"])
def test_raster_splits(oracle, kind, n_ypr):
    m = _mesh(kind)
    ypr = np.random.default_rng(n_ypr).uniform(0.0, 2.0 * np.pi, (n_ypr, 3)).astype(np.float32)
    opts = PrintOptions(shell_mesh=kind == "cube_and_sphere")
    got, want = native.sweep(m, ypr, opts), oracle.sweep(m, ypr, opts)
    for k in ("Vo64", "Vss64", "Vtc64"):
        assert np.array_equal(getattr(got, k), want[k]), k
    for k in ("Mo", "Mss", "Vtc"):
        assert np.array_equal(getattr(got, k).view(np.int32), np.asarray(want[k], np.float32).view(np.int32)), k
    assert got.optID == want["optID"]


@pytest.mark.parametrize("dvoxel", [14.0, 300.0, 1.0e7, 1.0e10, -1.0e10])
def test_raster_at_any_pixel_size(oracle, dvoxel):
    """Pixel centres far outside the triangles: the cells stay those of the pixel
    box and the triangles fall back to their centroids."""
    m = _mesh("cube_and_sphere")
    ypr = np.random.default_rng(3).uniform(0.0, 2.0 * np.pi, (5, 3)).astype(np.float32)
    opts = PrintOptions(dVoxel=dvoxel)
    got, want = native.sweep(m, ypr, opts), oracle.sweep(m, ypr, opts)
    for k in ("Vo64", "Vss64", "Vtc64"):
        assert np.array_equal(getattr(got, k), want[k]), k
    assert np.array_equal(got.entries, want["entries"]) and got.optID == want["optID"]
