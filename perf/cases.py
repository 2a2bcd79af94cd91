"""The work that programs give this renderer, as measurable cases.

Kinds of case, each one call sequence a program makes through the public
Python API (``kittlespt_gb300.renderer``):

* ``frame``     one frame from a new camera position and its display image
                (previews, stills, offline sequences);
* ``live``      one interactive frame: the camera and one object have moved,
                temporal accumulation, FSR or bilinear upscaling, lens effects;
* ``animate``   a deforming mesh: refit, then a frame;
* ``batch``     many small render requests submitted together;
* ``adjoint``   one gradient evaluation of an image loss, with the records
                kept between the two halves (``split``) or as one host call;
* ``rays``      ray queries against a committed scene: closest hits, occlusion
                or diffuse bounce chains;
* ``sky``       sky radiance of many directions (an environment map).

Scenes are the families of ``kittlespt_gb300.scenes``: the sphere pair with
more spheres, the grid of displaced icospheres under emissive quads, random
triangles.  Mesh geometry is the same for every seed (a program loads the same
files); cameras, materials, placements, the sun and the rays differ.
"""

import functools
import math

import numpy as np
import torch

from kittlespt_gb300 import scenes as S
from kittlespt_gb300.renderer import Batch, Renderer


def listed():
    return [
        # the smallest frame: a thumbnail or viewport preview, where latency and launches count
        dict(name="preview_256", kind="frame", scene="spheres", objects=2, width=256, height=256, spp=1, depth=4,
             post=False, karis=False, sky_arith=1),
        # an ordinary still with the whole post chain, odd in both directions, in the host build's sky arithmetic
        dict(name="still_853x481", kind="frame", scene="icospheres", objects=25, width=853, height=481, spp=3,
             depth=8, post=True, karis=True, sky_arith=0),
        # the full frame of the benchmark: 64 instances, 16 samples, depth 8
        dict(name="full_1080p_16spp", kind="frame", scene="icospheres", objects=64, width=1920, height=1080, spp=16,
             depth=8, post=True, karis=False, sky_arith=1),
        # an interactive viewport: one sample per frame, history, FSR to 1080p, lens effects, one object moving
        dict(name="live_fsr_1080p", kind="live", scene="icospheres", objects=64, width=1920, height=1080, spp=1,
             depth=4, upscale=2, effects=True),
        # an animated mesh: 20,480 triangles refit, then a frame at half size
        dict(name="animate_20480", kind="animate", subdiv=5, width=640, height=360, spp=2, depth=5),
        # a render service's queue: a dozen requests of mixed sizes, spp, depths and scenes
        dict(name="batch_12_mixed", kind="batch", jobs=12, max_side=512, max_spp=12, max_depth=8),
        # inverse rendering, large: the differentiation workload of the benchmark, records kept
        dict(name="adjoint_512_32spp", kind="adjoint", width=512, height=512, spp=32, depth=6, split=True),
        # inverse rendering, small and odd, as one call on host arrays
        dict(name="adjoint_97x61_8spp", kind="adjoint", width=97, height=61, spp=8, depth=4, split=False),
        # picking and small probes: few rays, launch latency
        dict(name="probe_1021_rays", kind="rays", scene="spheres", size=2, rays=1021, query="closest", bounces=0),
        # an ambient-occlusion bake: many short occlusion rays over the instanced scene
        dict(name="occlusion_700001", kind="rays", scene="icospheres", size=64, rays=700001, query="any", bounces=0),
        # the traversal stress of the benchmark: 2M random triangles, 1M rays, 4 diffuse bounces
        dict(name="chains_2M_tris", kind="rays", scene="triangles", size=2000000, rays=1048576, query="bounces",
             bounces=4),
        # a 512 x 256 sky map
        dict(name="sky_map_131072", kind="sky", dirs=131072, sky_arith=1),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["frame", "frame", "frame", "live", "animate", "batch", "adjoint", "rays", "rays", "sky"])
    if kind == "frame":
        w = _log(rng, 64, 1920)
        return dict(kind=kind, scene=rng.choice(["spheres", "icospheres"]), objects=_log(rng, 1, 64), width=w,
                    height=max(33, int(w * rng.uniform(0.5, 0.5625))), spp=_log(rng, 1, 16), depth=rng.randint(1, 8),
                    post=rng.random() < 0.6, karis=rng.random() < 0.3, sky_arith=rng.randint(0, 1))
    if kind == "live":
        w = _log(rng, 320, 1920)
        return dict(kind=kind, scene=rng.choice(["spheres", "icospheres"]), objects=_log(rng, 2, 64), width=w,
                    height=int(w * 0.5625), spp=rng.randint(1, 4), depth=rng.randint(2, 6),
                    upscale=rng.randint(0, 2), effects=rng.random() < 0.5)
    if kind == "animate":
        w = _log(rng, 128, 960)
        return dict(kind=kind, subdiv=rng.randint(2, 6), width=w, height=int(w * 0.5625), spp=rng.randint(1, 4),
                    depth=rng.randint(2, 6))
    if kind == "batch":
        return dict(kind=kind, jobs=rng.randint(2, 16), max_side=_log(rng, 96, 512), max_spp=rng.randint(2, 12),
                    max_depth=rng.randint(3, 8))
    if kind == "adjoint":
        w = _log(rng, 48, 512)
        return dict(kind=kind, width=w, height=max(33, int(w * rng.uniform(0.6, 1.0))), spp=_log(rng, 2, 32),
                    depth=rng.randint(2, 6), split=rng.random() < 0.6)
    if kind == "rays":
        scene = rng.choice(["spheres", "icospheres", "triangles"])
        query = rng.choice(["closest", "any", "bounces"])
        size = _log(rng, 1000, 2000000) if scene == "triangles" else _log(rng, 1, 64)
        return dict(kind=kind, scene=scene, size=size, rays=_log(rng, 100, 1048576), query=query,
                    bounces=rng.randint(1, 4) if query == "bounces" else 0)
    return dict(kind=kind, dirs=_log(rng, 500, 131072), sky_arith=rng.randint(0, 1))


# ----------------------------------------------------------------------------
# scenes

@functools.lru_cache(maxsize=None)
def _icosphere(subdiv, seed):
    return S.displaced_icosphere(subdiv, 0.1, seed=seed)


@functools.lru_cache(maxsize=2)
def _triangles(n):
    return S.random_triangles(n, seed=3)


@functools.lru_cache(maxsize=None)
def _sphere():
    return S.uv_sphere(64, 32, 1.0, 0)


def _camera(g, width, height):
    eye = np.array([0.0, 4.0, 22.0]) + g.uniform(-1.0, 1.0, 3)
    return S.Camera.look_at(eye, (0.0, 1.0, 0.0), 45.0, width, height)


def _any_material(g):
    alb, rough = tuple(g.uniform(0.1, 0.9, 3)), float(g.uniform(0.05, 1.0))
    kind = int(g.integers(0, 3))
    if kind == 1:
        return S.material(albedo=alb, roughness=rough, transmission=1.0, ior=1.5)
    return S.material(albedo=alb, roughness=rough, metallic=1.0 if kind == 2 else 0.0)


def _scene(g, family, objects, width, height, spp, depth, post=False, karis=False, sky_arith=1):
    st = S.settings(max_depth=depth, bloom=post, karis=karis, auto_exposure=post)
    env = S.environment(sun_theta=math.radians(g.uniform(15.0, 60.0)), sun_phi=g.uniform(0.0, 2.0 * math.pi))
    inst = []
    if family == "spheres":
        mats = [S.material(albedo=(0.5, 0.5, 0.5), roughness=0.5)] + [_any_material(g) for _ in range(4)]
        meshes = [_sphere(), S.quad(20.0, 20.0, 0.0, True, 0)]
        inst.append(S.Instance(1, S.translate(0, -1.0, 0).astype(S.F32), 0))
        for k in range(objects):
            x, z = ((-1.5, 0.0), (1.5, 0.0))[k] if k < 2 else (g.uniform(-6, 6), g.uniform(-6, 2))
            inst.append(S.Instance(0, S.translate(x, 0, z).astype(S.F32), 1 + k % 4))
        eye = np.array([0.0, 1.0, 5.0]) + g.uniform(-0.2, 0.2, 3)
        cam = S.Camera.look_at(eye, (0.0, 0.0, 0.0), 45.0, width, height)
    elif family == "triangles":
        mats = [S.material()]
        meshes = [_triangles(objects)]
        inst.append(S.Instance(0, np.eye(4, dtype=S.F32), 0))
        cam = S.Camera.look_at((0.5, 0.5, 3.0), (0.5, 0.5, 0.5), 45.0, width, height)
    else:
        mats, grid = [], max(1, math.ceil(math.sqrt(objects)))
        meshes = [_icosphere(6, s) for s in S.FULL_FRAME_VARIANT_SEEDS]
        meshes.append(S.quad(0.5, 0.5, 0.0, facing_up=False, mat_id=0))
        half = (grid - 1) / 2.0
        for k in range(objects):
            mats.append(_any_material(g))
            model = (S.translate((k // grid - half) * 3.0, 0.0, (k % grid - half) * 3.0)
                     @ S.rot_y(g.uniform(0.0, 2.0 * math.pi)) @ S.scale(g.uniform(0.5, 1.5)))
            inst.append(S.Instance(int(g.integers(0, 5)), model.astype(S.F32), k))
        mats.append(S.material(albedo=(0.8, 0.8, 0.8), emission=(1.0, 1.0, 1.0), emission_scale=20.0))
        for k in range(16):
            model = S.translate((k // 4 - 1.5) * 6.0, 3.0, (k % 4 - 1.5) * 6.0)
            inst.append(S.Instance(5, model.astype(S.F32), len(mats) - 1))
        cam = _camera(g, width, height)
    sc = S.Scene(meshes, inst, np.stack(mats), cam, env, st, S.exposure(), width, height, spp)
    sc.sky_arith, sc.temporal_arith = sky_arith, 1
    return sc


class _State:
    """What the program keeps: its renderers (closed with the state) and buffers."""

    def __init__(self, **kw):
        self.renderers, self.batch, self.step = [], None, 0
        self.__dict__.update(kw)

    def open(self, scene):
        r = Renderer(0)
        r.initialize()
        self.renderers.append(r)
        r.set_blas_build(True)
        r.load_scene(scene)
        return r

    def __del__(self):
        if self.batch is not None:
            self.batch.close()
        for r in self.renderers:
            r.shutdown()


def _rng(seed):
    return np.random.Generator(np.random.PCG64(seed))


def _jobs(case):
    """The requests of a batch: scene family, objects, size, samples, depth."""
    g = _rng(case["jobs"] * 4096 + case["max_side"])
    for _ in range(case["jobs"]):
        w = int(g.integers(64, case["max_side"] + 1))
        yield ("spheres" if g.integers(0, 2) == 0 else "icospheres", int(g.integers(1, 33)), w, max(48, w * 9 // 16),
               int(g.integers(1, case["max_spp"] + 1)), int(g.integers(2, case["max_depth"] + 1)))


def _rays(g, case, scene):
    """Origins and directions (and lengths, for occlusion) that the query meets."""
    n = case["rays"]
    if case["scene"] == "triangles":
        o, d = S.random_rays(n, seed=int(g.integers(0, 1 << 30)))
        reach = g.uniform(0.05, 1.5, n)
    elif case["query"] == "any":
        # points about the objects, directions of the upper hemisphere
        at = np.stack([i.model[:3, 3] for i in scene.instances])[g.integers(0, len(scene.instances), n)]
        v = g.normal(size=(n, 3))
        o = at + 1.6 * v / np.linalg.norm(v, axis=1, keepdims=True)
        d = g.normal(size=(n, 3))
        d /= np.linalg.norm(d, axis=1, keepdims=True)
        d[:, 1] = np.abs(d[:, 1])
        reach = g.uniform(0.5, 8.0, n)
    else:
        # from about the camera to points of the scene
        o = np.tile(np.asarray(scene.camera.inv_view)[:3, 3], (n, 1)) + g.normal(size=(n, 3)) * 0.05
        to = g.uniform(-1.0, 1.0, (n, 3)) * ((3.0, 1.0, 2.0) if case["scene"] == "spheres" else (12.0, 1.5, 12.0))
        d = (to - o) / np.linalg.norm(to - o, axis=1, keepdims=True)
        reach = np.full(n, 30.0)
    return o.astype(S.F32), d.astype(S.F32), reach.astype(S.F32)


def _directions(n, seed):
    g = _rng(seed)
    d = g.normal(size=(n, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    d[:, 1] = np.abs(d[:, 1])   # the sky dome
    return d.astype(S.F32)


def prepare(case, seed):
    kind, g = case["kind"], _rng(seed)
    if kind in ("frame", "live"):
        sc = _scene(g, case["scene"], case["objects"], case["width"], case["height"], case["spp"], case["depth"],
                    post=case.get("post", True), karis=case.get("karis", False), sky_arith=case.get("sky_arith", 1))
        st = _State(case=case, scene=sc)
        r = st.open(sc)
        if kind == "live":
            r.set_renderer_settings(temporal_accumulation=1, upscale=case["upscale"],
                                    postprocess_effects=int(case["effects"]))
    elif kind == "animate":
        mesh = _icosphere(case["subdiv"], 0)
        mats = np.stack([_any_material(g), S.material(albedo=(0.5, 0.5, 0.5), roughness=0.5)])
        inst = [S.Instance(0, np.eye(4, dtype=S.F32), 0), S.Instance(1, S.translate(0, -1.2, 0).astype(S.F32), 1)]
        sc = S.Scene([mesh, S.quad(20.0, 20.0, 0.0, True, 1)], inst, mats,
                     S.Camera.look_at((0.0, 1.0, 4.0), (0.0, 0.0, 0.0), 45.0, case["width"], case["height"]),
                     S.environment(sun_theta=math.radians(g.uniform(15.0, 60.0))),
                     S.settings(max_depth=case["depth"], bloom=True, auto_exposure=True), S.exposure(),
                     case["width"], case["height"], case["spp"])
        sc.sky_arith = 1
        st = _State(case=case, scene=sc, poses=[])
        st.open(sc)
        axis = g.normal(size=3)
        for k in range(4):   # the poses of the animation
            w = 1.0 + 0.1 * np.sin(3.0 * (mesh.positions @ axis) + k)[..., None]
            st.poses.append(np.ascontiguousarray(mesh.positions * w, S.F32))
    elif kind == "batch":
        st = _State(case=case, spp=[])
        for family, objects, w, h, spp, depth in _jobs(case):
            st.open(_scene(g, family, objects, w, h, spp, depth, post=family == "icospheres"))
            st.spp.append(spp)
        st.batch = Batch(0)
    elif kind == "adjoint":
        sc = S.scene_small(case["width"], case["height"], case["spp"], case["depth"])
        for m in sc.materials:
            m["albedo"], m["roughness"] = g.uniform(0.1, 0.9, 3), g.uniform(0.05, 1.0)
        st = _State(case=case)
        r = st.open(sc)
        shape = (case["height"], case["width"], 4)
        target = g.uniform(0.0, 2000.0, shape).astype(S.F32)
        if case["split"]:
            st.target = torch.from_numpy(target).cuda()
            st.image = torch.zeros(shape, dtype=torch.float32, device="cuda")
            st.grad = torch.zeros(4 * len(sc.materials) + 6, dtype=torch.float64, device="cuda")
            st.stream = torch.cuda.ExternalStream(r.stream())
        else:
            st.adjoint = np.sign(target - 1000.0).astype(S.F32)
    elif kind == "rays":
        sc = _scene(g, case["scene"], case["size"], 64, 64, 1, 1)
        st = _State(case=case)
        st.open(sc)
        st.o, st.d, st.reach = (torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in _rays(g, case, sc))
        n = case["rays"] * (case["bounces"] + 1)
        if case["query"] == "any":
            st.hit = torch.zeros(n, dtype=torch.uint8, device="cuda")
        else:
            st.inst = torch.zeros(n, dtype=torch.int32, device="cuda")
            st.tri, st.t = torch.zeros_like(st.inst), torch.zeros(n, dtype=torch.float32, device="cuda")
            st.uv = torch.zeros((n, 2), dtype=torch.float32, device="cuda")
    else:
        sc = _scene(g, "spheres", 1, 64, 64, 1, 1, sky_arith=case["sky_arith"])
        st = _State(case=case)
        st.open(sc)
        st.dirs = torch.from_numpy(_directions(case["dirs"], seed)).cuda()
        st.out = torch.zeros((case["dirs"], 3), dtype=torch.float32, device="cuda")
    for r in st.renderers:
        r.synchronize()
    return st


def run(st):
    case, kind = st.case, st.case["kind"]
    r = st.renderers[0]
    if kind == "frame":
        r.set_camera_inverse(st.scene.camera.inv_proj, st.scene.camera.inv_view)   # a new view: accumulation restarts
        r.execute_rendering(16.0, case["spp"])
        return r.get_render_target()
    if kind == "live":
        st.step += 1
        view = np.array(st.scene.camera.inv_view)
        view[0, 3] += 0.02 * (st.step % 16)                      # a slow pan
        r.set_camera_inverse(st.scene.camera.inv_proj, view)
        model = np.array(st.scene.instances[1].model)
        model[1, 3] += 0.3 * math.sin(0.1 * st.step)             # an object bobbing
        r.set_mesh_transform(1, model)
        r.execute_rendering(16.0, case["spp"])
        return r.get_render_target()
    if kind == "animate":
        st.step += 1
        r.refit_mesh(0, st.poses[st.step % 4])
        r.execute_rendering(16.0, case["spp"])
        return r.get_render_target()
    if kind == "batch":
        for x in st.renderers:
            x.reset_accumulation()
        st.batch.submit(st.renderers, st.spp)
        st.batch.wait()
        return [x.get_render_target() for x in st.renderers]
    if kind == "adjoint":
        if not case["split"]:
            grad, image = r.adjoint(0, case["spp"], st.adjoint, want_image=True)
            return {"grad": grad, "image": image}
        with torch.cuda.stream(st.stream):
            r.adjoint_forward_device(0, case["spp"], st.image.data_ptr())
            adjoint = torch.sign(st.image - st.target)           # dLoss/dimage of the L1 loss
            r.adjoint_backward_device(adjoint.data_ptr(), st.grad.data_ptr())
        return {"grad": st.grad, "image": st.image}
    if kind == "rays":
        n, o, d = case["rays"], st.o.data_ptr(), st.d.data_ptr()
        if case["query"] == "any":
            r.occluded_device(n, o, d, st.reach.data_ptr(), st.hit.data_ptr())
            return st.hit
        if case["query"] == "closest":
            r.trace_device(n, o, d, st.inst.data_ptr(), st.tri.data_ptr(), st.t.data_ptr(), st.uv.data_ptr())
            return {"inst": st.inst, "tri": st.tri, "t": st.t, "uv": st.uv}
        r.trace_bounces_device(n, o, d, case["bounces"], st.inst.data_ptr(), st.tri.data_ptr(), st.t.data_ptr())
        return {"inst": st.inst, "tri": st.tri, "t": st.t}
    r.sky_device(case["dirs"], st.dirs.data_ptr(), st.out.data_ptr())
    return st.out


def _scene_bytes(family, objects):
    """Geometry a path or ray set reads at least once: nodes, triangles, shading records."""
    tris = objects if family == "triangles" else 3970 if family == "spheres" else 5 * 81920
    return tris * 48.0


def _ray_flops(family, objects):
    """One ray down the tree once: two boxes a level, a few triangles."""
    tris = objects if family == "triangles" else 3970 * max(1, objects) if family == "spheres" else 81920 * objects
    return 40.0 * math.log2(max(2, tris)) + 200.0


def work(case):
    kind = case["kind"]
    if kind in ("frame", "live"):
        scale = 2.5 if case.get("upscale") else 1.0
        pixels = case["width"] * case["height"]
        traced = pixels / scale / scale
        ray = _ray_flops(case["scene"], case["objects"])
        return {"bytes": 16.0 * pixels + _scene_bytes(case["scene"], case["objects"]),
                "flops": traced * (ray + case["spp"] * (ray + 300.0)) + 100.0 * pixels}
    if kind == "animate":
        tris, pixels = 20 * 4 ** case["subdiv"], case["width"] * case["height"]
        ray = _ray_flops("triangles", tris)
        return {"bytes": 36.0 * tris + 48.0 * tris + 16.0 * pixels,
                "flops": 60.0 * tris + pixels * (ray + case["spp"] * (ray + 300.0))}
    if kind == "batch":
        total = {"bytes": 0.0, "flops": 0.0}
        for family, objects, w, h, spp, _ in _jobs(case):
            ray = _ray_flops(family, objects)
            total["bytes"] += 16.0 * w * h + _scene_bytes(family, objects)
            total["flops"] += w * h * (ray + spp * (ray + 300.0))
        return total
    if kind == "adjoint":
        pixels = case["width"] * case["height"]
        ray = _ray_flops("spheres", 2)
        return {"bytes": 48.0 * pixels, "flops": pixels * (ray + case["spp"] * (ray + 900.0))}
    if kind == "rays":
        n, out = case["rays"], 1.0 if case["query"] == "any" else 20.0 if case["query"] == "closest" else 12.0
        return {"bytes": n * (28.0 + out * (case["bounces"] + 1)) + _scene_bytes(case["scene"], case["size"]),
                "flops": n * _ray_flops(case["scene"], case["size"])}
    return {"bytes": 24.0 * case["dirs"], "flops": case["dirs"] * 16.0 * (8 * 20.0 + 40.0)}


# ----------------------------------------------------------------------------
# 64-bit values

def _exact_rays(case, seed):
    """Closest hits by brute force over every triangle of every instance."""
    g = _rng(seed)
    sc = _scene(g, case["scene"], case["size"], 64, 64, 1, 1)
    o, d, reach = (torch.from_numpy(x.astype(np.float64)).cuda() for x in _rays(g, case, sc))
    n = o.shape[0]
    best = torch.full((n,), math.inf, dtype=torch.float64, device="cuda")
    uv = torch.zeros((n, 2), dtype=torch.float64, device="cuda")
    for inst in sc.instances:
        inv = torch.from_numpy(np.linalg.inv(inst.model.astype(np.float64))).cuda()
        lo, ld = o @ inv[:3, :3].T + inv[:3, 3], d @ inv[:3, :3].T
        p = torch.from_numpy(sc.meshes[inst.mesh].positions.astype(np.float64)).cuda()
        v0, e1, e2 = p[:, 0], p[:, 1] - p[:, 0], p[:, 2] - p[:, 0]
        step = max(1, (1 << 22) // p.shape[0])
        for a in range(0, n, step):
            rd, ro = ld[a:a + step, None], lo[a:a + step, None]
            pv = torch.cross(rd.expand(-1, p.shape[0], -1), e2[None].expand(rd.shape[0], -1, -1), dim=-1)
            det = (e1 * pv).sum(-1)
            tv = ro - v0
            u = (tv * pv).sum(-1) / det
            qv = torch.cross(tv, e1[None].expand_as(tv), dim=-1)
            v = (rd * qv).sum(-1) / det
            t = (e2 * qv).sum(-1) / det
            ok = (det.abs() >= 1.0e-5) & (u >= 0) & (u <= 1) & (v >= 0) & (u + v <= 1) & (t > 1.0e-5)
            m, k = torch.where(ok, t, torch.inf).min(dim=1)
            closer = m < best[a:a + step]
            best[a:a + step] = torch.where(closer, m, best[a:a + step])
            hit = torch.stack([u.gather(1, k[:, None])[:, 0], v.gather(1, k[:, None])[:, 0]], 1)
            uv[a:a + step] = torch.where(closer[:, None], hit, uv[a:a + step])
    return {"inst": None, "tri": None, "t": best, "uv": uv}


def _exact_sky(case, seed):
    """Single scattering over 16 view and 8 light steps from 1 m above the ground."""
    g = _rng(seed)
    e = _scene(g, "spheres", 1, 64, 64, 1, 1).env
    d = torch.from_numpy(_directions(case["dirs"], seed).astype(np.float64)).cuda()
    phi, theta = float(e["sun_phi"]), float(e["sun_theta"])
    sun = torch.tensor([math.cos(phi) * math.cos(theta), math.sin(theta), math.sin(phi) * math.cos(theta)],
                       dtype=torch.float64, device="cuda")
    earth, top = 6378137.0, 6438137.0
    hr, hm = float(e["rayleigh_height"]), float(e["mie_height"])
    sr = torch.tensor([float(x) for x in e["rayleigh"]], dtype=torch.float64, device="cuda")
    sm, am = float(e["mie"]), float(e["mie_absorption"])

    def leave(o, w):   # distance to the top of the atmosphere
        b = (o * w).sum(-1)
        return -b + torch.sqrt(b * b - (o * o).sum(-1) + top * top)

    def height(p):
        return torch.linalg.norm(p, dim=-1) - earth

    o = torch.tensor([0.0, earth + 1.0, 0.0], dtype=torch.float64, device="cuda").expand_as(d)
    step = leave(o, d) / 16.0
    ir, im = torch.zeros_like(d), torch.zeros_like(d)
    dr, dm = torch.zeros_like(step), torch.zeros_like(step)
    for i in range(16):
        p = o + ((i + 0.5) * step)[:, None] * d
        h = height(p)
        r, m = torch.exp(-h / hr) * step, torch.exp(-h / hm) * step
        dr, dm = dr + r, dm + m
        ls = leave(p, sun) / 8.0
        lr, lm, lit = torch.zeros_like(step), torch.zeros_like(step), torch.ones_like(step, dtype=torch.bool)
        for j in range(8):
            q = height(p + ((j + 0.5) * ls)[:, None] * sun)
            lit &= q >= 0
            lr, lm = lr + torch.exp(-q / hr) * ls, lm + torch.exp(-q / hm) * ls
        tr = torch.exp(-(sr * (dr + lr)[:, None] + (sm + am) * (dm + lm)[:, None])) * lit[:, None]
        ir, im = ir + tr * r[:, None], im + tr * m[:, None]
    mu = (d * sun).sum(-1)[:, None]
    k = 0.76
    phase_r = 3.0 * (1.0 + mu * mu) / (16.0 * math.pi)
    phase_m = 3.0 * (1.0 - k * k) * (1.0 + mu * mu) / (8.0 * math.pi * (2.0 + k * k)
                                                      * (1.0 + k * k - 2.0 * k * mu) ** 1.5)
    return (sr * ir * phase_r + sm * im * phase_m) * 6.0e5 * float(e["sun_emission_factor"])


def exact(case, seed):
    if case["kind"] == "sky":
        return _exact_sky(case, seed)
    if case["kind"] == "rays" and case["query"] == "closest":
        tris = _scene_bytes(case["scene"], case["size"]) / 48.0
        tris *= case["size"] if case["scene"] != "triangles" else 1
        if tris * case["rays"] <= 2.0e9:
            return _exact_rays(case, seed)
    return None   # sampled light transport (decisions follow the rounding), whole numbers, or too long
