"""Refit of meshes of few and many triangles, one after another in one context
(its refit memory is kept and grows): every box is the bounds of the triangles
under it, hits are the oracle's brute force, for leaves of 1 to 8 triangles,
meshes that are one leaf and leaves of more triangles than lanes work on one."""

import copy

import numpy as np
import pytest

from kittlespt_gb300 import scenes as S
from oracle import oracle as O

from tests.test_gpu_parity import bits, global_prim, gpu_trace, make_renderer
from tests.test_refit import _expected_boxes

pytestmark = pytest.mark.gpu


def _triangles(n, seed, same=False):
    rng = np.random.default_rng(seed)
    pos = rng.uniform(-2.0, 2.0, (1 if same else n, 1, 3)) + rng.normal(0.0, 0.2, (1 if same else n, 3, 3))
    return np.ascontiguousarray(np.broadcast_to(pos, (n, 3, 3)), np.float32)


@pytest.mark.parametrize("sizes", [[1, 8, 9], [17, 300], [5000, 2, 40001]])
@pytest.mark.parametrize("same", [False, True])
def test_sizes(sizes, same):
    sc = S.scene_small(32, 32, 1, 2)
    if same:   # all triangles alike: no split parts them
        sizes = [min(n, 40) for n in sizes]
    meshes = []
    for k, n in enumerate(sizes):
        pos = _triangles(n, 10 + k, same)
        nrm = np.tile(np.float32([0.0, 1.0, 0.0]), (n, 3, 1))
        meshes.append(S.Mesh(pos, nrm, np.zeros((n, 3, 2), np.float32), np.zeros(n, np.int32)))
    sc.meshes = meshes
    sc.instances = [S.Instance(k, S.translate(0.0, 0.0, -1.0 * k).astype(np.float32), 0) for k in range(len(sizes))]
    sc2 = copy.deepcopy(sc)
    o, d = S.random_rays(20000, 4, center=(0, 0, 0), radius=6.0)
    r = make_renderer(sc)
    try:
        for k, n in enumerate(sizes):
            pos = (meshes[k].positions * np.float32(0.8) + _triangles(n, 50 + k, same) * np.float32(0.2)).astype(np.float32)
            sc2.meshes[k] = S.Mesh(pos, meshes[k].normals, meshes[k].uvs, meshes[k].material)
            r.refit_mesh(k, pos)
        for k in range(len(sizes)):
            blas = r.get_blas(k)
            assert np.array_equal(blas["boxes"], _expected_boxes(blas, sc2.meshes[k].positions))
        inst, tri, t = gpu_trace(r, o, d)
    finally:
        r.shutdown()
    ref = O.Scene(sc2).trace(o, d, brute=True)
    np.testing.assert_array_equal(bits(t), bits(ref["t"]))
    if not same:
        np.testing.assert_array_equal(global_prim(sc2, inst, tri), ref["prim"])
