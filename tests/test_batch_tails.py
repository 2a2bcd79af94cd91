"""A batch whose jobs end differently: some path by path (their wave's tail),
some level by level, the latter going on past the others' last level."""

import pytest

from kittlespt_gb300 import scenes as S

from tests.test_batch import _outputs, _renderers, _same

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


# (width, height, samples, depth): up to 300,000 samples of a wave the tail starts at level 2,
# above 1,250,000 not before level 5
@pytest.mark.parametrize("sizes", [
    [(64, 36, 2, 4), (960, 540, 3, 5)],                                   # tail from 2 of 4; levels 0 to 5
    [(64, 36, 2, 3), (960, 540, 3, 4), (64, 36, 2, 2), (33, 9, 1, 4)],    # tails of 3 and 4, no tail of 2
    [(640, 360, 2, 4), (96, 54, 4, 8), (960, 540, 3, 8)],                 # tails from 3, 2 and 5
])
def test_jobs_end_once(sizes):
    from kittlespt_gb300.renderer import Batch
    jobs = [(S.scene_full(w, h, spp, depth, n_variants=2, subdiv=3, grid=3, n_lights=4) if k % 2 else
             S.scene_small_n(w, h, spp, depth, 4), spp) for k, (w, h, spp, depth) in enumerate(sizes)]
    spp = [n for _, n in jobs]
    alone, together = _renderers(jobs), _renderers(jobs)
    try:
        with Batch(0) as b:
            for _ in range(2):
                for r, n in zip(alone, spp):
                    r.execute_rendering(16.0, n)
                b.submit(together, spp)
                b.wait()
        _same(_outputs(together), _outputs(alone))
        for r, q in zip(together, alone):
            s, t = r.stats(), q.stats()
            assert (s.path_rays, s.shadow_rays, s.adapted_luminance) == (t.path_rays, t.shadow_rays, t.adapted_luminance)
    finally:
        for r in alone + together:
            r.shutdown()
