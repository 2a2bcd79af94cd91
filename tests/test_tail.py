"""The tail of a wave (k_tail: each path's later levels in one go) against the
wave taken level by level, which a context with stage timing on renders:
accumulation, display image, ray counts and per-level counts bit for bit."""

import numpy as np
import pytest

from kittlespt_gb300 import _lib as K
from kittlespt_gb300 import scenes as S

from tests.test_gpu_parity import bits, make_renderer

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _frames(sc, timed, **tuning):
    r = make_renderer(sc)
    try:
        if tuning:
            r.set_tuning(**tuning)
        if timed:
            K.check(r._L.kpt_enable_timing(r.ctx, 1))
        out = []
        for k in range(2):
            r.execute_rendering(16.0, sc.spp)
            st = r.stats()
            out.append((r.read_accumulation(), r.get_render_target(), r.level_counts(),
                        (st.path_rays, st.shadow_rays, st.path_box_tests, st.path_inst_xforms, st.overflows)))
        return out
    finally:
        r.shutdown()


def _every_lobe(w, h, spp, depth):
    return S.scene_full(w, h, spp, depth, n_variants=2, subdiv=3, grid=4, n_lights=4)


CASES = {
    "every_lobe": (lambda: _every_lobe(96, 54, 4, 8), {}),          # lights, transmission, roulette, one path a warp
    "spheres": (lambda: S.scene_small_n(200, 150, 3, 6, 12), {}),   # long chains, several paths a warp
    "tail_at_the_last_level_but_one": (lambda: _every_lobe(33, 17, 2, 3), {}),
    "no_tail": (lambda: _every_lobe(33, 17, 2, 2), {}),
    "few_paths": (lambda: S.scene_small(7, 3, 1, 8), {}),
    "several_waves": (lambda: _every_lobe(96, 54, 4, 6), dict(wave_cap=4096)),
    "sorted": (lambda: _every_lobe(96, 54, 4, 6), dict(sort_rays=1)),
    "sky_as_the_reference": (lambda: _every_lobe(96, 54, 4, 6), dict()),
    "level_3": (lambda: S.scene_small_n(512, 400, 2, 6, 8), {}),    # 409,600 items
    "level_4": (lambda: _every_lobe(640, 480, 2, 7), {}),           # 614,400 items
}


@pytest.mark.parametrize("which", list(CASES))
def test_tail_equals_the_levels(which):
    make, tuning = CASES[which]
    sc = make()
    sc.settings["bloom"] = sc.settings["auto_exposure"] = 1
    if which == "sky_as_the_reference":
        sc.sky_arith = 1
    tail, levels = _frames(sc, False, **tuning), _frames(sc, True, **tuning)
    for (acc, img, counts, rays), (acc2, img2, counts2, rays2) in zip(tail, levels):
        np.testing.assert_array_equal(bits(acc), bits(acc2))
        np.testing.assert_array_equal(bits(img), bits(img2))
        np.testing.assert_array_equal(counts, counts2)
        assert rays == rays2
