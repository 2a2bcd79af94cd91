"""The escapes' sky gradient, whose Jacobians the replay's sky pass stores per
path: one wave, several (the stored Jacobians are reused wave by wave) and the
split halves give the same gradient."""

import numpy as np
import pytest

from kittlespt_gb300 import scenes as S

from tests.test_gpu_parity import make_renderer

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("w,h,spp,depth", [(64, 48, 4, 3), (33, 35, 3, 6), (7, 5, 1, 1)])
def test_waves_and_halves(w, h, spp, depth):
    sc = S.scene_small(w, h, spp, depth)
    a = np.random.default_rng(5).random((h, w, 4), np.float32)
    grads, images = [], []
    for cap in (0, 1024):
        r = make_renderer(sc)
        try:
            if cap:
                r.set_tuning(wave_cap=cap)
            g, image = r.adjoint(0, spp, a, want_image=True)
            grads.append(g)
            images.append(image)
            if not cap:
                d = torch.from_numpy(a).cuda()
                img = torch.zeros((h, w, 4), dtype=torch.float32, device="cuda")
                out = torch.zeros(len(g), dtype=torch.float64, device="cuda")
                torch.cuda.synchronize()
                r.adjoint_forward_device(0, spp, img.data_ptr())
                r.adjoint_backward_device(d.data_ptr(), out.data_ptr())
                r.synchronize()
                grads.append(out.cpu().numpy())
                images.append(img.cpu().numpy())
        finally:
            r.shutdown()
    assert np.any(grads[0][-6:] != 0.0)
    # the same single-precision terms (fewer than 2^17) summed in double in another order:
    # 2^17 * 2^-53 = 1.5e-11 of the terms' absolute sum, taken to be within 100 of the sum
    for g, im in zip(grads[1:], images[1:]):
        np.testing.assert_allclose(g, grads[0], rtol=1.5e-9)
        np.testing.assert_allclose(im, images[0], rtol=3e-6)   # up to 4 samples, added by atomics
