"""Sky radiance of short and long lists of directions: several lanes march a
direction where the list is short (8 or 2, by its length), one where it is
long, with the same result bit for bit."""

import math

import numpy as np
import pytest

from kittlespt_gb300 import scenes as S

from tests.test_gpu_parity import make_renderer

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

LONG = 400003   # more than any GPU of this kind holds threads for


def _sky(r, dirs):
    d = torch.from_numpy(np.ascontiguousarray(dirs)).cuda()
    out = torch.zeros((len(dirs), 3), dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    r.sky_device(len(dirs), d.data_ptr(), out.data_ptr())
    r.synchronize()
    return out.cpu().numpy().view(np.int32)


@pytest.mark.parametrize("arith", [0, 1])
@pytest.mark.parametrize("theta_deg", [-4.0, 5.0, 80.0])   # the light rays meet the ground, graze, leave
def test_lanes_give_the_same_sky(arith, theta_deg):
    sc = S.scene_small(16, 16, 1, 1)
    sc.env["sun_theta"] = math.radians(theta_deg)
    sc.sky_arith = arith
    i = np.arange(LONG) + 0.5
    y = 1.0 - 2.0 * ((i * 0.6180339887) % 1.0)   # every stretch of the list covers the sphere
    phi = i * 2.39996323
    dirs = np.stack([np.sqrt(1.0 - y * y) * np.cos(phi), y, np.sqrt(1.0 - y * y) * np.sin(phi)], 1).astype(np.float32)
    r = make_renderer(sc)
    try:
        want = _sky(r, dirs)
        assert np.isfinite(want.view(np.float32)).all() and (want != 0).any()
        for n in (1, 7, 8, 9, 1021, 19001, 20011, 50021, 80009, 131072):
            np.testing.assert_array_equal(_sky(r, dirs[n:2 * n]), want[n:2 * n])
    finally:
        r.shutdown()
