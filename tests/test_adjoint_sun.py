"""The sun's Jacobian (k_adjoint_constants, one block) against the FP64 sky.

In frames of depth 0 the sky enters a hit pixel only by its sun light
samples: with weights W per channel, the pixels' radiance sums to W * S (S the
sun's radiance) and the gradient of that sum for sky parameter k is the sum
over the channels of W * dS/dk.  W follows from the image and the oracle's S,
dS/dk from its central differences.  The single-precision S is within 1e-3 of
the oracle's (tests/test_adjoint.py), the differences (h = 1e-3) within 1e-5 of
the derivatives: 2e-3 of the terms' sizes bounds the whole."""

import math

import numpy as np
import pytest

from kittlespt_gb300 import scenes as S
from oracle import oracle as O

from tests.test_adjoint import _renderer, _sky_theta_fixed

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("theta_deg,mie_scale,rayleigh_height", [(5.0, 1.0, 8000.0), (17.0, 1.0, 7994.0),
                                                                 (45.0, 4.0, 8000.0), (85.0, 0.25, 4000.0)])
def test_sun_jacobian(theta_deg, mie_scale, rayleigh_height):
    w, h, spp = 40, 30, 4
    sc = S.scene_small(w, h, spp, 0)
    sc.env["sun_theta"] = math.radians(theta_deg)
    sc.env["mie"] *= np.float32(mie_scale)
    sc.env["rayleigh_height"] = rayleigh_height
    hit = O.Scene(sc).render_samples(0, 1)["first_hit"][..., 0] >= 0
    r = _renderer(sc)
    try:
        image = r.adjoint(0, spp, np.zeros((h, w, 4), np.float32), want_image=True)[1]
        hit &= image.max(-1) < 1.0e8 / spp   # a sample clamped at 1e8 has no derivative
        adj = np.zeros((h, w, 4), np.float32)
        adj[hit] = 1.0
        grad, image = r.adjoint(0, spp, adj, want_image=True)
    finally:
        r.shutdown()
    sky, fixed = _sky_theta_fixed(sc)
    sun = np.array([fixed[:3]], np.float32)
    weight = image[hit][:, :3].astype(np.float64).sum(0) / O.sky_double(sun, sky, fixed)[0]
    assert (weight > 0).all()
    for k in range(6):
        step = 1e-3 * abs(sky[k])
        up, down = sky.copy(), sky.copy()
        up[k] += step
        down[k] -= step
        d = (O.sky_double(sun, up, fixed) - O.sky_double(sun, down, fixed))[0] / (2.0 * step)
        assert abs(grad[len(grad) - 6 + k] - (weight * d).sum()) <= 2e-3 * np.abs(weight * d).sum(), k
