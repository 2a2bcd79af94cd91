"""The bloom chain of images whose levels take a pixel's taps from one block of
texels (100,000 pixels and more: kpt_post.cu), against the oracle's chain: the
levels' down and up steps and level 0's tent in the tonemap, odd sizes, with
and without the Karis average."""

import numpy as np
import pytest

from kittlespt_gb300 import scenes as S
from oracle import oracle as O

from tests.test_gpu_parity import make_renderer

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

LOG_ERROR = 6.3e-6


def _tolerance(post, expo):
    """Per channel, how far the display image may be off through CUDA's and the
    C library's log2f, exp2f (1, 2 and 1 ulp) and powf (4 and 1 ulp) alone; the
    rest of the chain is the same IEEE operations.

    The logarithm of a value and of the exposure range are off by at most
    9.1e-6 together (2 ulps of numbers below 16, 2^-20 each, and the range's
    three ulps of exp2f, over its 16.5 stops), as from an exposure off by 6.3e-6
    of itself; what that and the polynomial's rounding make of it is probed: twice
    the spread over nine exposures in that range.  The powf of the look and the
    EOTF: 5 * 2^-24 of their result each, 2.4 * 1.5 times and once into the linear
    values, which the last matrix (rows of absolute sum 2.93) mixes, times the slope of
    the sRGB curve; and its own powf."""
    probes = [post(np.float32(expo * (1.0 + k * LOG_ERROR / 4))) for k in range(-4, 5)]
    spread = np.max(probes, axis=0) - np.min(probes, axis=0)
    ref = probes[4][..., :3].astype(np.float64)
    lin = np.where(ref <= 0.04045, ref / 12.92, ((ref + 0.055) / 1.055) ** 2.4)
    slope = np.where(lin <= 0.0031308, 12.92, 1.055 / 2.4 * np.maximum(lin, 0.0031308) ** (1 / 2.4 - 1))
    ulps = 5 * 2.0 ** -24
    powf = 2.93 * (2.4 * 1.5 + 1.0) * ulps * lin.max(-1, keepdims=True) * slope + 1.055 * ulps
    return probes[4], 2.0 * spread[..., :3] + powf


@pytest.mark.parametrize("karis", [0, 1])
@pytest.mark.parametrize("w,h", [(401, 301), (901, 483), (1283, 911)])   # one, two, two levels with blocks
def test_large_levels_match_the_oracle(w, h, karis):
    sc = S.scene_full(w, h, 1, 2, n_variants=2, subdiv=3, grid=4, n_lights=4)
    sc.settings["bloom"], sc.settings["karis"], sc.settings["auto_exposure"] = 1, karis, 0
    sc.settings["bloom_final_blend"] = 0.8
    r = make_renderer(sc)
    try:
        r.execute_rendering(16.0, 1)
        r.synchronize()
        render, img = r.read_render(), r.get_render_target()
    finally:
        r.shutdown()
    expo = float(O.exposure_scalar(sc.exposure))

    def post(with_karis):
        bl = O.bloom(render, bool(with_karis), float(sc.settings["bloom_internal_blend"]))
        return lambda x: O.post_image(render, bl, 0.8, float(x))

    ref, tol = _tolerance(post(karis), expo)
    err = np.abs(img[..., :3].astype(np.float64) - ref[..., :3])
    assert (err <= tol).all(), f"{(err > tol).sum()} values off, worst {(err / tol).max()} times the bound, {err.max()}"
    # the bound tells the chain from one that differs in its taps' weights
    other = np.abs(post(1 - karis)(expo)[..., :3] - ref[..., :3])
    assert (other > 10 * tol).mean() > 0.05
