"""Gradients whose sums leave the range that the sweep and the escapes' sky keep
in three floats (2^100): the gradient is linear in dLoss/dimage, so a loss
scaled by a power of two scales it exactly, up to the order of its sums."""

import numpy as np
import pytest

from kittlespt_gb300 import scenes as S

from tests.test_gpu_parity import make_renderer

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("largest", [60, 99, 101, 110, 116])   # log2 of the largest parameter's gradient
def test_scaled_loss(largest):
    w, h, spp, depth = 40, 30, 4, 4
    sc = S.scene_small(w, h, spp, depth)
    a = np.random.default_rng(8).random((h, w, 4), np.float32)
    r = make_renderer(sc)
    try:
        base, _ = r.adjoint(0, spp, a)
        k = largest - int(np.floor(np.log2(np.abs(base).max())))
        scaled, _ = r.adjoint(0, spp, np.ldexp(a, k).astype(np.float32))
    finally:
        r.shutdown()
    assert np.isfinite(scaled).all()
    # the same terms (fewer than 2^15), times 2^k: 2^15 * 2^-53 of their absolute sum, taken to be within 100 of the sum
    np.testing.assert_allclose(scaled, np.ldexp(base, k), rtol=4e-10)
