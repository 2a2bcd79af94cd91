"""The queue traversal at the sizes where its warps work differently, against
the oracle bit for bit: leaves of 1 to 9 triangles and one of 40 (a group of
lanes tests 4 or 8 of a leaf at a time), queues of fewer rays than the grid
has warps, of about one ray per warp and of several warps' worth, ray ranges
that end at, before and after a hit, meshes whose root is a leaf, and the
camera rays' tiles over ragged images."""

import numpy as np
import pytest

from kittlespt_gb300 import scenes as S
from oracle import oracle as O

from tests.test_gpu_parity import bits, global_prim, make_renderer, render_samples

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _mesh(ntris, seed, clump=False):
    """ntris random triangles; clump: all with one centroid, which no split
    separates (one leaf)."""
    rng = np.random.default_rng(seed)
    pos = rng.normal(0.0, 0.5, (ntris, 3, 3)).astype(np.float32)
    if clump:   # integer corners that sum to zero: equal centroids exactly
        pos[:, 0] = rng.integers(-4, 5, (ntris, 3))
        pos[:, 1] = rng.integers(-4, 5, (ntris, 3))
        pos[:, 2] = -(pos[:, 0] + pos[:, 1])
        pos *= np.float32(0.125)
    n = np.cross(pos[:, 1] - pos[:, 0], pos[:, 2] - pos[:, 0])
    n /= np.maximum(np.linalg.norm(n, axis=1, keepdims=True), 1e-12)
    return S.Mesh(pos, np.repeat(n[:, None], 3, 1).astype(np.float32), np.zeros((ntris, 3, 2), np.float32),
                  np.zeros(ntris, np.int32))


def _scene(sizes, clump=0):
    base = S.scene_small(8, 8, 1, 2)
    meshes = [_mesh(k, 10 + k) for k in sizes] + ([_mesh(clump, 99, True)] if clump else [])
    inst = [S.Instance(k, (S.translate(0.7 * k, 0.2 * (k % 3), -0.4 * (k % 2)) @ S.rot_y(0.3 * k)).astype(np.float32), 0)
            for k in range(len(meshes))]
    return S.Scene(meshes, inst, base.materials, base.camera, base.env, base.settings, base.exposure, 8, 8, 1)


def _rays(sc, n, seed):
    """Towards points inside the scene's triangles, every eighth with an axis-parallel direction."""
    rng = np.random.default_rng(seed)
    ex = sc.expanded()
    k = rng.integers(0, ex["positions"].shape[0], n)
    model = np.concatenate([np.repeat(m[None], c, 0) for m, c in zip(ex["models"], ex["mesh_count"])])[k]
    p = np.einsum("nk,nkj->nj", rng.dirichlet((1.0, 1.0, 1.0), n), ex["positions"][k])
    p = np.einsum("nij,nj->ni", model[:, :3, :3], p) + model[:, :3, 3]
    d = rng.normal(size=(n, 3))
    d[::8] = np.eye(3)[rng.integers(0, 3, d[::8].shape[0])]
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    return (p - 4.0 * d).astype(np.float32), d.astype(np.float32)


def _closest(r, o, d, tmin=0.0, tmax=float("inf")):
    n = o.shape[0]
    to, td = torch.from_numpy(o).cuda(), torch.from_numpy(d).cuda()
    inst = torch.empty(n, dtype=torch.int32, device="cuda")
    tri, t = torch.empty_like(inst), torch.empty(n, dtype=torch.float32, device="cuda")
    uv = torch.empty((n, 2), dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    r.trace_device(n, to.data_ptr(), td.data_ptr(), inst.data_ptr(), tri.data_ptr(), t.data_ptr(), uv.data_ptr(),
                   tmin, tmax)
    r.synchronize()
    return inst.cpu().numpy(), tri.cpu().numpy(), t.cpu().numpy(), uv.cpu().numpy()


SCENES = {"leaves_1_to_9": ([1, 2, 3, 4, 5, 6, 7, 8, 9], 0), "one_triangle": ([1], 0), "root_leaf_of_40": ([3], 40),
          "deep": ([3000, 17], 40)}


@pytest.mark.parametrize("n", [1, 31, 33, 4863, 4865, 20000])
@pytest.mark.parametrize("which", list(SCENES))
def test_queue_matches_oracle(which, n):
    sc = _scene(*SCENES[which])
    o, d = _rays(sc, n, n)
    orc = O.Scene(sc)
    r = make_renderer(sc)
    try:
        for tmin, tmax in ((0.0, np.inf), (3.5, np.inf), (0.0, 4.0), (3.9, 4.1)):
            ref = orc.trace(o, d, tmin, tmax)
            inst, tri, t, uv = _closest(r, o, d, tmin, tmax)
            np.testing.assert_array_equal(global_prim(sc, inst, tri), ref["prim"])
            hit = ref["prim"] >= 0
            np.testing.assert_array_equal(bits(t[hit]), bits(ref["t"][hit]))
            np.testing.assert_array_equal(bits(uv[hit]), bits(ref["bary"][hit][:, 1:]))
    finally:
        r.shutdown()


@pytest.mark.parametrize("n", [1, 33, 4865, 20000])
@pytest.mark.parametrize("which", list(SCENES))
def test_occlusion_ranges(which, n):
    """Each ray with a range that ends just before its closest hit, at it
    (open: not occluded), just after it, at zero, below zero and nowhere."""
    sc = _scene(*SCENES[which])
    o, d = _rays(sc, n, 7 * n)
    t = O.Scene(sc).trace(o, d)["t"]
    tmax = np.choose(np.arange(n) % 6, [np.nextafter(t, np.float32(0.0)), t, np.nextafter(t, np.float32(np.inf)),
                                        np.zeros_like(t), np.full_like(t, -1.0), np.full_like(t, np.inf)])
    tmax = tmax.astype(np.float32)
    r = make_renderer(sc)
    try:
        to, td, tm = (torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in (o, d, tmax))
        out = torch.empty(n, dtype=torch.uint8, device="cuda")
        torch.cuda.synchronize()
        r.occluded_device(n, to.data_ptr(), td.data_ptr(), tm.data_ptr(), out.data_ptr())
        r.synchronize()
    finally:
        r.shutdown()
    np.testing.assert_array_equal(out.cpu().numpy() != 0, t < tmax)


@pytest.mark.parametrize("w,h", [(8, 4), (9, 5), (1, 33), (7, 3), (257, 2), (40, 31)])
def test_camera_tiles(w, h):
    """Every pixel of images that 8 x 4 tiles cover exactly, with narrow and
    low tiles at the edges, or only with those: first hits and albedo."""
    sc = S.scene_small(w, h, 1, 1)
    ref = O.Scene(sc).render_samples(0, 1)
    r = make_renderer(sc)
    try:
        rad, hit, alb = render_samples(r, sc, 1)
    finally:
        r.shutdown()
    np.testing.assert_array_equal(global_prim(sc, hit[..., 0], hit[..., 1]), ref["first_hit"][..., 0])
    on = ref["first_hit"][..., 0] >= 0
    np.testing.assert_array_equal(bits(alb[..., :3][on]), bits(ref["albedo"][on][..., :3]))
