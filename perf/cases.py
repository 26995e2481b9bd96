"""Timed cases: the work a program has this library do, through its public entry points.

Seven kinds of work, each with the sizes it is met at:

  frame      one frame of one view, the camera moving along its path from frame to
             frame: corrected ReSTIR GI, with the learned cache's inference, or the
             reference's own settings (compat_reference)
  views      one frame of several views over several scenes in one launch set
  dynamic    one frame of an animated world: vertices of a mesh and every instance
             transform change, then the frame
  build      the BVH of an uploaded scene, then a batch of rays through it
  trace      closest-hit / any-hit rays on device buffers
  query      the same through host arrays (upload, trace, read back)
  cache      the learned cache on host arrays: gradients of a batch, then a prediction
             of every sample

Scenes, cameras and settings are the benchmark's (bench.py) and the tests': the
procedural generator from 40 to 16384 objects (8.8 thousand to 4 million triangles),
the Cornell box, depth 4 (10 in reference mode), resolutions from 256 x 256 to
3840 x 2160.  A seed picks the scene, the camera's start and the random streams.

Frames come back as views of the renderer's device images: the RGBA8 image, and the
linear image where the case asks for it (write_hdr).
"""
from __future__ import annotations

import math

import numpy as np
import torch

import xvk_ray_gb300 as xr
from xvk_ray_gb300 import _lib as L

PATH_FRAMES = 32          # the camera path's length, played forward and back
ANIM_FRAMES = 16          # animation frames a dynamic case keeps in host memory
VIEW_RES = ((256, 256), (512, 512), (1280, 720), (1920, 1080))


def listed():
    return [
        # an interactive preview: the smallest frame, where launches and latency count
        dict(name="frame_cornell_256", kind="frame", objects=0, w=256, h=256, mode="restir", hdr=True, spatial=True),
        # an editor viewport of an odd size over a mid-sized scene under a sky, with temporal
        # reuse only (the reference UI's other setting)
        dict(name="frame_853x479_94k_temporal", kind="frame", objects=400, w=853, h=479, mode="restir", hdr=True,
             spatial=False, sky=True),
        # the benchmark's frame: 1920 x 1080, 998,442 triangles
        dict(name="frame_1080p_1m", kind="frame", objects=4096, w=1920, h=1080, mode="restir", hdr=False, spatial=True),
        # the same with paths ending in a trained cache (inference in every frame)
        dict(name="frame_1080p_1m_cache", kind="frame", objects=4096, w=1920, h=1080, mode="cache", hdr=True,
             spatial=True),
        # a user of the reference at its own settings: 10 bounces, its reservoir layout, textures
        dict(name="frame_1080p_94k_reference", kind="frame", objects=400, w=1920, h=1080, mode="reference", hdr=False,
             spatial=True),
        # render farm: views of uneven size over four scenes, one launch set per frame
        dict(name="views_8_over_4_scenes", kind="views", views=8, scenes=4, objects=40, top=2048, w=0, h=0),
        # large streams: two 4K cameras over four million triangles
        dict(name="views_2x4k_4m", kind="views", views=2, scenes=1, objects=16384, top=16384, w=3840, h=2160),
        # a game loop: the scene as one instance, moving instances around it, a mesh deforming
        dict(name="dynamic_1080p_1m_256", kind="dynamic", objects=4096, w=1920, h=1080, instances=256),
        # scene load: the acceleration structure of a million triangles
        dict(name="build_1m", kind="build", objects=4096, rays=65536),
        # batch visibility on the device: incoherent closest hits, as light baking asks for
        dict(name="trace_closest_2m_rays_1m", kind="trace", objects=4096, rays=1 << 21, any_hit=False),
        # gameplay queries: a few line-of-sight rays through host arrays
        dict(name="query_any_1000_rays_94k", kind="query", objects=400, rays=1000, any_hit=True),
        # the learned cache on its own: a batch's gradients and its predictions (the hash
        # table's 64 MB of gradients stay on the device, as in training)
        dict(name="cache_65536", kind="cache", samples=65536),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["frame", "frame", "frame", "views", "dynamic", "build", "trace", "query", "cache"])
    objects = _log(rng, 40, 4096)
    if kind == "frame":
        w = _log(rng, 200, 1920)
        return dict(kind=kind, objects=rng.choice([0, objects, objects]), w=w, h=max(64, int(w * rng.uniform(0.5, 1.0))),
                    mode=rng.choice(["restir", "restir", "cache", "reference"]), hdr=rng.random() < 0.5,
                    spatial=rng.random() < 0.75, sky=rng.random() < 0.25)
    if kind == "views":
        scenes = rng.randint(1, 4)
        return dict(kind=kind, views=rng.randint(scenes, 8), scenes=scenes, objects=_log(rng, 40, 400), top=objects,
                    w=0 if rng.random() < 0.5 else _log(rng, 200, 1920), h=_log(rng, 200, 1080))
    if kind == "dynamic":
        return dict(kind=kind, objects=objects, w=_log(rng, 256, 1920), h=_log(rng, 256, 1080),
                    instances=_log(rng, 2, 256))
    if kind == "build":
        return dict(kind=kind, objects=_log(rng, 40, 8192), rays=_log(rng, 1000, 65536))
    if kind == "trace":
        return dict(kind=kind, objects=objects, rays=_log(rng, 1000, 1 << 21), any_hit=rng.random() < 0.5)
    if kind == "query":
        return dict(kind=kind, objects=objects, rays=_log(rng, 1, 65536), any_hit=rng.random() < 0.5)
    return dict(kind="cache", samples=128 * _log(rng, 1, 1024))


# ---- inputs -----------------------------------------------------------------

EXTENT = 40.0


def _scene(objects, seed, extent=EXTENT, lights=16):
    if objects == 0:
        return xr.Scene.cornell()
    # the object density of the benchmark's scene at 4096 objects and more, its extent below
    ext = extent * max(1.0, objects / 4096.0) ** 0.5
    return xr.Scene.procedural(seed=1 + seed % 100003, n_objects=objects, n_lights=lights, extent=ext, sphere_subdiv=2)


def _reference_materials(scene, rng):
    """The scene as the reference can render it: Lambertian and light materials only, a
    third of them textured (planar coordinates)."""
    model = scene.materials[:, 7].view(np.uint32)
    model[model != L.XR_MAT_DIFFUSE_LIGHT] = L.XR_MAT_LAMBERTIAN
    scene.textures = [rng.integers(0, 256, (n, 2 * n, 4), dtype=np.uint8) for n in (64, 256)]
    tex = scene.materials[:, 4].view(np.int32)
    tex[1::3] = rng.integers(0, 2, tex[1::3].shape)
    tex[model == L.XR_MAT_DIFFUSE_LIGHT] = -1
    p = scene.vertices
    p[:, 6] = p[:, 0] - np.floor(p[:, 0])
    p[:, 7] = p[:, 2] - np.floor(p[:, 2])
    return scene


def _rays(scene, n, seed, any_hit):
    """Rays from points of the scene's volume in uniform directions; segments of a few
    units for visibility."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    v = scene.vertices[:, 0:3]
    lo = torch.tensor(np.maximum(v.min(0), [-60.0, 0.0, -60.0]).astype(np.float32), device="cuda")
    hi = torch.tensor(np.minimum(v.max(0), [60.0, 8.0, 60.0]).astype(np.float32), device="cuda")
    r = torch.empty(n, 8, device="cuda")
    r[:, 0:3] = lo + (hi - lo) * torch.rand(n, 3, generator=g, device="cuda")
    r[:, 3] = 1e-4
    d = torch.randn(n, 3, generator=g, device="cuda")
    r[:, 4:7] = d / d.norm(dim=1, keepdim=True)
    r[:, 7] = 1.0 + 20.0 * torch.rand(n, generator=g, device="cuda") if any_hit else 1e4
    return r.contiguous()


CACHE_LO, CACHE_INV = (-1.0, -1.0, -1.0), 0.5    # the scene cube [-1, 1]^3


def _cache_weights(seed):
    """Weights of a trained cache's magnitude: table N(0, 0.3), MLP uniform as initialised."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    table = torch.randn(16 * (1 << 19) * 2, generator=g, device="cuda") * 0.3
    mlp = torch.rand(17408, generator=g, device="cuda") * 2 - 1
    mlp[:16384] *= math.sqrt(6.0 / 128.0)
    mlp[16384:] *= math.sqrt(6.0 / 80.0)
    mlp[16384 + 3 * 64:] = 0.0
    return mlp.cpu().numpy(), table.cpu().numpy()


def _cache_samples(n, seed):
    """Samples on the walls and boxes of a room: positions on planes, unit normals and
    directions, radiance targets with a bright tail."""
    rng = np.random.default_rng(seed)
    s = np.zeros(n, xr.api.CACHE_SAMPLE_DTYPE)
    p = rng.uniform(-0.95, 0.95, (n, 3)).astype(np.float32)
    axis = rng.integers(0, 3, n)
    side = rng.choice(np.array([-0.9, -0.3, 0.25, 0.9], np.float32), n)
    p[np.arange(n), axis] = side
    s["pos"] = p
    nrm = np.zeros((n, 3), np.float32)
    nrm[np.arange(n), axis] = -np.sign(side)
    s["normal"] = nrm
    d = rng.standard_normal((n, 3)).astype(np.float32)
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    d *= np.where((d * nrm).sum(1, keepdims=True) < 0, -1.0, 1.0).astype(np.float32)
    s["wo"] = d
    s["albedo"] = rng.uniform(0.1, 0.9, (n, 3)).astype(np.float32)
    s["roughness"] = rng.uniform(0.05, 1.0, n).astype(np.float32)
    s["kind"] = rng.choice(np.array([0, 0, 1, 5], np.uint32), n)
    s["target"] = rng.exponential(0.5, (n, 3)).astype(np.float32) * rng.choice(np.array([0.1, 1.0, 8.0], np.float32),
                                                                               (n, 1), p=[0.5, 0.45, 0.05])
    return s


class _Context:
    """Closes its renderer once neither a state nor an image of it is held any more."""

    def __init__(self, renderer):
        self.r = renderer

    def __del__(self):
        self.r.close()


class _DeviceArray:
    """A renderer's device image for torch (no copy; torch holds this object as long as
    the tensor lives, and with it the renderer whose memory it is)."""

    def __init__(self, context, ptr, shape, typestr):
        self.context = context
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": shape, "typestr": typestr, "version": 2}


class _Camera:
    """One view's camera on its path: 0.01 units and 0.2 degrees a frame, 32 frames
    forward, then back."""

    def __init__(self, cam, w, h, bounces, sky, yaw):
        self.cam = L.XrCamera.from_buffer_copy(cam)
        self.cam.yaw_deg += yaw
        self.w, self.h, self.bounces, self.sky = w, h, bounces, sky
        self.prev, self.f = None, 0

    def next(self):
        s = 1.0 if (self.f // PATH_FRAMES) % 2 == 0 else -1.0
        self.cam.position[2] -= 0.01 * s
        self.cam.yaw_deg += 0.2 * s
        self.prev = xr.camera_ubo(self.cam, self.w, self.h, self.prev, self.f, self.bounces, sky=self.sky)
        self.f += 1
        return self.prev


class _State:
    def open(self, w, h):
        self.r = xr.Renderer(w, h)
        self.context = _Context(self.r)


def _images(st, n):
    """The frame's images: the RGBA8 one (its buffer alternates) and the linear one."""
    out = []
    for which in (L.XR_OUT_LDR8, L.XR_OUT_HDR) if st.hdr else (L.XR_OUT_LDR8,):
        ptr = st.r.output_device_ptr(which)
        if ptr not in st.images:
            st.images[ptr] = torch.as_tensor(_DeviceArray(st.context, ptr, (n, 4),
                                                          "|u1" if which == L.XR_OUT_LDR8 else "<f4"), device="cuda")
        out.append(st.images[ptr])
    return out


def prepare(case, seed):
    st = _State()
    st.kind = kind = case["kind"]
    st.images = {}
    st.hdr = bool(case.get("hdr"))
    if kind == "cache":
        st.open(8, 8)
        st.r.cache.reset(1 + seed % 1000)
        st.r.cache.set_bounds(CACHE_LO, CACHE_INV)
        mlp, table = _cache_weights(seed)
        st.r.cache.write(L.XR_CACHE_MLP, mlp)
        st.r.cache.write(L.XR_CACHE_GRID, table)
        st.samples = _cache_samples(case["samples"], seed)
        return st
    if kind in ("build", "trace", "query"):
        scene = _scene(case["objects"], seed)
        st.open(8, 8)
        st.r.upload_scene(scene)
        if kind != "build":
            st.r.build_bvh()
        st.n = case["rays"]
        st.any_hit = bool(case.get("any_hit"))
        rays = _rays(scene, st.n, seed, st.any_hit)
        if kind == "query":
            st.rays = rays.cpu().numpy()
        else:
            st.rays = rays
            st.prim = torch.empty(st.n, dtype=torch.int32, device="cuda")
            st.t = torch.empty(st.n, device="cuda")
            st.bary = torch.empty(st.n, 2, device="cuda")
        return st
    w, h = case["w"], case["h"]
    yaw = (seed % 97) * 0.37
    if kind == "views":
        n = case["scenes"]
        objs = [int(round(case["objects"] * (case["top"] / case["objects"]) ** (k / max(1, n - 1)))) if n > 1
                else case["top"] for k in range(n)]
        scenes = [_scene(o, seed + 10 * k, lights=64 if o > 8192 else 16) for k, o in enumerate(objs)]
        views = [(v * n // case["views"], *((w, h) if w else VIEW_RES[v % len(VIEW_RES)])) for v in range(case["views"])]
        st.open(8, 8)
        st.r.upload_scenes(scenes)
        st.r.set_views(views, xr.params_default(8, 8, seed=1 + seed % 65521))
        st.r.set_graphs(True)
        st.cams = [_Camera(scenes[s].camera, vw, vh, 4, False, yaw + (90.0 if n == 1 else 7.0) * v)
                   for v, (s, vw, vh) in enumerate(views)]
        st.n = sum(vw * vh for _, vw, vh in views)
        return st
    scene = _scene(case["objects"], seed)
    st.n = w * h
    if kind == "dynamic":
        small = [xr.Scene.procedural(seed=77 + seed % 1000 + k, n_objects=6, n_lights=0, extent=1.0, sphere_subdiv=2)
                 for k in range(2)]
        st.open(w, h)
        st.r.set_params(xr.params_default(w, h, seed=1 + seed % 65521))
        st.r.upload_scenes([scene] + small)
        st.verts, st.inst = [], []
        for f in range(ANIM_FRAMES):
            v = small[1].vertices.copy()
            v[:, 1] += (0.1 * np.sin(2.0 * v[:, 0] + 2.0 * np.pi * f / ANIM_FRAMES)).astype(np.float32)
            st.verts.append(v)
            st.inst.append(_instances(case["instances"], f, seed))
        st.cams = [_Camera(scene.camera, w, h, 4, False, yaw)]
        return st
    ref = case["mode"] == "reference"
    if ref:
        scene = _reference_materials(scene, np.random.default_rng(seed))
        p = xr.params_reference(w, h, write_hdr=int(st.hdr))
    else:
        p = xr.params_default(w, h, seed=1 + seed % 65521, write_hdr=int(st.hdr), spatial_on=int(case["spatial"]))
    st.open(w, h)
    st.r.set_params(p)
    st.r.upload_scene(scene)
    st.r.build_bvh()
    if case["mode"] == "cache":
        cp = xr.cache_params_default()
        cp.enabled, cp.train = 1, 0
        st.r.cache.set_params(cp)
        mlp, table = _cache_weights(seed)
        st.r.cache.write(L.XR_CACHE_MLP, mlp)
        st.r.cache.write(L.XR_CACHE_GRID, table)
    st.r.set_graphs(True)
    # the Cornell box keeps its light in view: a small turn only
    st.cams = [_Camera(scene.camera, w, h, 10 if ref else 4, bool(case.get("sky")),
                       yaw if case["objects"] else (seed % 97) * 0.02)]
    return st


def _instances(count, f, seed):
    """The big scene in place and `count` copies of the two small ones circling in it."""
    rec = np.zeros(count + 1, xr.api.INSTANCE_DTYPE)
    m = rec["object_to_world"].reshape(-1, 3, 4)
    m[0, :, :3] = np.eye(3)
    k = np.arange(count)
    a = 2 * np.pi * k / count + 0.01 * f * (1 + k % 3) + (seed % 89) * 0.05
    rad = 6.0 + 30.0 * (k % 16) / 16.0
    s = 0.5 + 0.5 * (k % 4)
    m[1:, 0, 0], m[1:, 0, 2] = s * np.cos(3 * a), s * np.sin(3 * a)
    m[1:, 2, 0], m[1:, 2, 2] = -s * np.sin(3 * a), s * np.cos(3 * a)
    m[1:, 1, 1] = s
    m[1:, 0, 3], m[1:, 1, 3], m[1:, 2, 3] = rad * np.cos(a), 1.0 + k % 5, rad * np.sin(a)
    rec["scene"][1:] = 1 + k % 2
    return rec


def run(st):
    r = st.r
    if st.kind == "frame":
        r.render(st.cams[0].next())
        return _images(st, st.n)
    if st.kind == "views":
        r.render_views([c.next() for c in st.cams])
        return _images(st, st.n)
    if st.kind == "dynamic":
        f = st.cams[0].f % ANIM_FRAMES
        r.update_vertices(2, st.verts[f])
        r.set_instances(st.inst[f])
        r.render(st.cams[0].next())
        return _images(st, st.n)
    # an occluded ray's triangle is any that lies in its way: what is asked is whether there is one
    if st.kind == "query":
        prim, t, bary = r.trace(st.rays, st.any_hit)
        return (prim >= 0,) if st.any_hit else (prim, t, bary)
    if st.kind == "cache":
        loss = r.cache.train(st.samples, apply=False)
        return loss, r.cache.read(L.XR_CACHE_MLP_GRAD), r.cache.query(st.samples)
    if st.kind == "build":
        r.build_bvh()
    L.check(L.load().xr_trace_rays_device(r.ctx, st.rays.data_ptr(), st.n, int(st.any_hit), st.prim.data_ptr(),
                                          st.t.data_ptr(), st.bary.data_ptr()), r.ctx)
    if not st.any_hit:
        return st.prim, st.t, st.bary
    r.sync()   # the comparison below runs on torch's stream
    return st.prim >= 0


# ---- the work of a pass ------------------------------------------------------

# Triangles per object of the procedural generator, and bytes of a triangle and its share
# of the vertices as uploaded (16 B of indices, half a vertex of position and normal).
TRIS_PER_OBJECT, TRI_BYTES = 244, 16 + 16
# Per path segment: a slab test of one 8-wide node per factor of eight of the triangle
# count (8 children, 6 multiply-adds and 6 comparisons each) and one triangle test.
NODE_FLOPS, TRI_FLOPS = 8 * 18, 60


def _ray_flops(objects):
    tris = max(36, objects * TRIS_PER_OBJECT)
    return math.log(tris, 8) * NODE_FLOPS + TRI_FLOPS


def _frame_work(pixels, objects, bounces, spatial, hdr, cache=False, reference=False):
    """Per pixel: the previous frame's G-buffer and reservoir read (20 + 32 B) and this
    frame's written, the image, and the rays of the path (half of them reach the next
    bounce) and of spatial reuse (half the neighbours need one)."""
    wide = 4 if reference else 1
    b = pixels * (2 * (20 + 32 * wide) + 4 + (16 if hdr else 0) + (32 if spatial else 0))
    rays = sum(0.5 ** k for k in range(bounces)) + (2.5 if spatial and not reference else 0.0)
    f = pixels * rays * (_ray_flops(objects) + 200)
    if cache:
        f += 0.25 * pixels * 2 * 17408
        b += 0.25 * pixels * 16 * 8 * 4
    return b, f


def work(case):
    kind = case["kind"]
    o = case.get("objects", 0)
    if kind == "frame":
        ref = case["mode"] == "reference"
        b, f = _frame_work(case["w"] * case["h"], o, 10 if ref else 4, case["spatial"], case["hdr"],
                           case["mode"] == "cache", ref)
    elif kind == "views":
        b = f = 0.0
        for v in range(case["views"]):
            w, h = (case["w"], case["h"]) if case["w"] else VIEW_RES[v % len(VIEW_RES)]
            x = _frame_work(w * h, case["top"], 4, True, False)
            b, f = b + x[0], f + x[1]
    elif kind == "dynamic":
        b, f = _frame_work(case["w"] * case["h"], o + 6 * case["instances"], 4, True, False)
        b += 1300 * 36 + case["instances"] * 56
    elif kind == "build":
        t = max(36, o * TRIS_PER_OBJECT)
        b, f = t * (TRI_BYTES + 48 + 14) + case["rays"] * 48, t * 100 + case["rays"] * _ray_flops(o)
    elif kind in ("trace", "query"):
        b, f = case["rays"] * (32 + 16), case["rays"] * _ray_flops(o)
    else:
        n = case["samples"]
        b = n * (2 * 72 + 12) + n * 3 * 16 * 8 * 4 + 17408 * 4
        f = n * 2 * 17408 * 4
    return {"bytes": float(b), "flops": float(f)}


# ---- 64-bit results -----------------------------------------------------------

def exact(case, seed):
    """Closest hits by testing every triangle, and the cache's network with its gradients,
    in 64 bits.  A frame has no such value: its paths and reservoirs branch on random
    numbers."""
    if case["kind"] == "cache":
        return _exact_cache(case, seed) if case["samples"] <= 65536 else None
    if case["kind"] in ("trace", "build", "query") and not case.get("any_hit"):
        if case["rays"] * max(36, case["objects"] * TRIS_PER_OBJECT) <= 4e10:
            return _exact_hits(case, seed)
    return None


def _exact_hits(case, seed):
    scene = _scene(case["objects"], seed)
    rays = _rays(scene, case["rays"], seed, False).double()
    tri = torch.tensor(scene.vertices[:, 0:3][scene.global_indices().reshape(-1, 3).astype(np.int64)],
                       device="cuda").double()
    a, e1, e2 = tri[:, 0], tri[:, 1] - tri[:, 0], tri[:, 2] - tri[:, 0]
    n, inf = rays.shape[0], float("inf")
    best, u_b, v_b = (torch.full((n,), x, device="cuda", dtype=torch.float64) for x in (inf, 0.0, 0.0))
    nt = torch.cross(e1, e2, dim=1)
    step = max(1, (1 << 24) // tri.shape[0])
    for i in range(0, n, step):
        o, d = rays[i:i + step, 0:3], rays[i:i + step, 4:7]
        # o + t d = a + u e1 + v e2, by Cramer's rule with triple products as matrix products
        det = -(d @ nt.T)
        oa_n = o @ nt.T - (a * nt).sum(1)
        t = oa_n / det
        c = torch.cross(o, d, dim=1)     # (o - a) x d = o x d - a x d
        u = (c @ e2.T - d @ torch.cross(e2, a, dim=1).T) / det
        v = -(c @ e1.T - d @ torch.cross(e1, a, dim=1).T) / det
        ok = (u >= 0) & (v >= 0) & (u + v <= 1) & (t >= 1e-4) & (t <= 1e4) & (det != 0)
        t = torch.where(ok, t, torch.full_like(t, inf))
        m, k = t.min(dim=1)
        best[i:i + step] = m
        u_b[i:i + step] = u.gather(1, k[:, None])[:, 0]
        v_b[i:i + step] = v.gather(1, k[:, None])[:, 0]
    hit = torch.isfinite(best)
    t = torch.where(hit, best, torch.full_like(best, -1.0))
    bary = torch.stack([torch.where(hit, u_b, torch.zeros_like(u_b)), torch.where(hit, v_b, torch.zeros_like(v_b))], 1)
    return [None, t, bary]


LEVEL_RES = (16, 22, 30, 42, 58, 80, 111, 153, 212, 294, 406, 561, 776, 1072, 1482, 2048)


def _exact_cache(case, seed):
    mlp, table = (torch.tensor(x, device="cuda", dtype=torch.float64) for x in _cache_weights(seed))
    s = _cache_samples(case["samples"], seed)

    def col(name):
        return torch.tensor(np.ascontiguousarray(s[name]), device="cuda").double()

    n = len(s)
    p = ((col("pos") - torch.tensor(CACHE_LO, device="cuda", dtype=torch.float64)) * CACHE_INV).clamp(0, 1)
    feats = []
    T = 1 << 19
    for lv, res in enumerate(LEVEL_RES):
        x = p * res
        i0 = x.floor().clamp(0, res - 1)
        f = x - i0
        i0 = i0.long()
        tl = table[2 * T * lv:2 * T * (lv + 1)].reshape(T, 2)
        acc = torch.zeros(n, 2, device="cuda", dtype=torch.float64)
        for k in range(8):
            b = torch.tensor([k & 1, (k >> 1) & 1, (k >> 2) & 1], device="cuda")
            c = i0 + b
            w = torch.where(b.bool(), f, 1 - f).prod(1, keepdim=True)
            if (res + 1) ** 3 <= T:
                idx = c[:, 0] + (res + 1) * (c[:, 1] + (res + 1) * c[:, 2])
            else:
                idx = (c[:, 0] ^ (c[:, 1] * 2654435761) ^ (c[:, 2] * 805459861)) & (T - 1)
            acc = acc + w * tl[idx]
        feats.append(acc)
    nrm, wo, kind = col("normal"), col("wo"), torch.tensor(s["kind"].astype(np.int64), device="cuda")
    refl = 2 * (nrm * wo).sum(1, keepdim=True) * nrm - wo
    x = torch.cat(feats + [nrm, wo, refl, col("albedo"), col("roughness")[:, None], (kind == 1).double()[:, None],
                           (kind == 5).double()[:, None], torch.ones(n, 1, device="cuda", dtype=torch.float64),
                           torch.zeros(n, 16, device="cuda", dtype=torch.float64)], 1)
    W = [mlp[4096 * l:4096 * l + 4096].reshape(64, 64).clone().requires_grad_() for l in range(4)]
    W.append(mlp[16384:].reshape(16, 64).clone().requires_grad_())
    for w in W[:4]:
        x = torch.relu(x @ w.T)
    y = (x @ W[4].T)[:, :3]
    # the relative L2 loss, its denominator held constant
    loss = ((y - col("target")) ** 2 / (y.detach() ** 2 + 0.01)).mean()
    loss.backward()
    return float(loss.detach()), torch.cat([w.grad.reshape(-1) for w in W]), y.detach()
