"""The network's kernels at the sample counts where their work splits: below,
at and past an eight (k_mlp_pass), eights that do not fill the eight partial
sums (k_mlp_update), a warp's eight and a CTA's 64 samples (k_mlp_forward)."""
from __future__ import annotations

import numpy as np
import pytest

from oracle import mlp_oracle as mo
from tomo_shell2026_b200 import surrogate

pytestmark = pytest.mark.gpu


def _data(n, seed):
    rng = np.random.default_rng(seed)
    yaw, pitch = rng.uniform(0, 2 * np.pi, n), rng.uniform(0, np.pi / 3, n)
    x = np.stack([np.sin(yaw), np.cos(yaw), np.sin(pitch), np.cos(pitch)], 1).astype(np.float32)
    return x, (np.sin(3 * yaw) + pitch).astype(np.float32)


@pytest.mark.parametrize("n", [1, 7, 8, 9, 63, 64, 65, 72, 513])
def test_sample_counts(n):
    surrogate.mlp_init(5)
    p = surrogate.mlp_params()
    x, y = _data(n, n)
    loss, g = surrogate.mlp_grad(x, y)
    ref_loss, ref = mo.loss_and_grad(p.astype(np.float64), x.astype(np.float64), y.astype(np.float64))
    # chains of at most 128 products and n / 64 + 16 sums of values near one, each
    # rounded at 2^-24: below 2e-5 of the larger of one and the largest gradient
    assert np.max(np.abs(g - ref)) <= 2e-5 * max(1.0, np.max(np.abs(ref)))
    assert abs(loss - ref_loss) <= 2e-5 * max(1.0, ref_loss)
    out = surrogate.mlp_predict(x)
    want = mo.forward(p.astype(np.float64), x.astype(np.float64))[-1][:, 0]
    assert np.max(np.abs(out - want)) <= 2e-5


def test_predictions_do_not_depend_on_the_count():
    """Eights of samples go to the CTAs in turn: the same bits for a sample whatever
    the number of samples, around one eight per CTA and eight per CTA."""
    surrogate.mlp_init(6)
    x, _ = _data(9480, 3)
    full = surrogate.mlp_predict(x)
    for n in (1, 8, 9, 100, 1183, 1184, 1185, 1193, 9471, 9472, 9473):
        assert np.array_equal(surrogate.mlp_predict(x[:n]).view(np.int32), full[:n].view(np.int32)), n
