"""BVH builds over primitives without area, the smallest inputs and boxes that coincide:
the build ends in a tree of bounded depth, and hits are the oracle's bit for bit."""
import numpy as np
import pytest

import xvk_ray_gb300 as xr
from oracle import binding as ob
from tests.helpers import affine, box_scene, random_rays
from tests.test_gpu_traversal_queue import _rays, _soup

pytestmark = pytest.mark.gpu


def _with_triangles(extra):
    """The Cornell box behind the triangles `extra` (k x 3 x 3)."""
    base = xr.Scene.cornell()
    k = len(extra)
    v = np.zeros((3 * k, 9), np.float32)
    v[:, :3] = np.asarray(extra, np.float32).reshape(-1, 3)
    v[:, 4] = 1.0
    v[:, 8] = base.vertices[0, 8]
    idx = np.concatenate([np.arange(3 * k, dtype=np.uint32), base.global_indices().astype(np.uint32) + 3 * k])
    return xr.Scene(np.concatenate([v, base.vertices]), idx, base.materials, np.zeros((1, 2), np.uint32), base.camera)


def _alone(tri):
    """A scene of these triangles alone."""
    v = np.zeros((3 * len(tri), 9), np.float32)
    v[:, :3] = np.asarray(tri, np.float32).reshape(-1, 3)
    v[:, 4] = 1.0
    base = xr.Scene.cornell()
    return xr.Scene(v, np.arange(3 * len(tri), dtype=np.uint32), base.materials[:1].copy(), np.zeros((1, 2), np.uint32),
                    base.camera)


def _check(scene, rays, max_depth):
    op, ot, obary = ob.OracleScene.from_scene(scene).trace(rays)
    hit = op >= 0
    with xr.Renderer(8, 8) as r:
        r.upload_scene(scene)
        r.build_bvh()
        gp, gt, gb = r.trace(rays)
        st = r.stats()
    assert st.error_flags == 0 and st.bvh_triangles == scene.n_triangles
    assert st.bvh_depth <= max_depth
    assert np.array_equal(gp, op)
    assert np.array_equal(gt[hit].view(np.uint32), ot[hit].view(np.uint32))
    assert np.array_equal(gb[hit].view(np.uint32), obary[hit].view(np.uint32))


@pytest.mark.parametrize("builder", ["ploc", "lbvh"])
@pytest.mark.parametrize("n", [4, 5, 8])
@pytest.mark.parametrize("kind", ["point", "line"])
def test_triangles_without_area(kind, n, builder, monkeypatch):
    """Points and axis-parallel segments: every SAH cost of their subtree is 0."""
    monkeypatch.setenv("XR_BVH_BUILDER", builder)
    tri = np.full((n, 3, 3), 0.5)
    if kind == "line":
        tri[:, :, 0] = np.arange(3 * n).reshape(n, 3) * 0.01
    rays = random_rays(np.random.default_rng(n), 2000, [-1, 0, -1], [1, 2, 1])
    _check(_alone(tri), rays, n)
    _check(_with_triangles(tri), rays, n + 4)


@pytest.mark.parametrize("builder", ["ploc", "karras"])
def test_instances_of_empty_scenes_at_one_point(builder, monkeypatch):
    """Instances of a scene without triangles are point boxes at their origin."""
    monkeypatch.setenv("XR_TLAS_BUILDER", builder)
    rng = np.random.default_rng(3)
    scene = box_scene(rng, 12, 2.0)
    empty = xr.Scene(scene.vertices, scene.indices[:0].copy(), scene.materials, scene.ranges, scene.camera)
    inst = [(1, affine(np.eye(3), [1, 2, 3]))] * 5 + [(0, affine(np.eye(3), [0, 0, 0]))]
    rays = random_rays(rng, 2000, -4, 4)
    world = ob.OracleWorld([ob.OracleScene.from_scene(s) for s in (scene, empty)])
    world.set_instances(inst)
    c = world.trace_instanced(rays)
    with xr.Renderer(8, 8) as r:
        r.upload_scenes([scene, empty])
        r.set_instances(inst)
        g = r.trace_instanced(rays)
        assert r.stats().error_flags == 0
    for x, y in zip(g, c):
        assert np.array_equal(np.asarray(x).view(np.uint32), np.asarray(y).view(np.uint32))


def _log2(n):
    return max(int(np.ceil(np.log2(n))), 1)


@pytest.mark.parametrize("builder", ["ploc", "lbvh"])
@pytest.mark.parametrize("n", [1, 2, 3, 4, 65, 200, 2047, 2049, 3000])
@pytest.mark.parametrize("kind", ["one", "point", "row"])
def test_boxes_that_tie(kind, n, builder, monkeypatch):
    """One triangle many times, one point many times, a row of equal triangles: merged boxes
    of equal area everywhere, and still a tree no deeper than a balanced binary one."""
    monkeypatch.setenv("XR_BVH_BUILDER", builder)
    tri = np.tile(np.array([[[-0.5, -0.5, 0.0], [0.5, -0.5, 0.25], [0.0, 0.5, 0.0]]]), (n, 1, 1))
    if kind == "point":
        tri[:] = 0.25
    if kind == "row":
        tri[:, :, 0] += (np.arange(n)[:, None] - n // 2) * 1.25
    _check(_alone(tri), _rays(300, n), _log2(n))


@pytest.mark.parametrize("n", [32, 256, 1500, 2100])
@pytest.mark.parametrize("kind", ["one", "row"])
def test_instances_whose_boxes_tie(kind, n, monkeypatch):
    """Instances spawned at one place or set up in a row, with the clustering builder."""
    monkeypatch.setenv("XR_TLAS_BUILDER", "ploc")
    rng = np.random.default_rng(n)
    scene = box_scene(rng, 6, 2.0)
    inst = [(0, affine(np.eye(3), [8.0 * k if kind == "row" else 0.5, 0, 0])) for k in range(n)]
    _check_world([scene], inst, random_rays(rng, 300, [-4, -4, -4], [60 if kind == "row" else 4, 4, 4]))


def _check_world(scenes, inst, rays):
    world = ob.OracleWorld([ob.OracleScene.from_scene(s) for s in scenes])
    world.set_instances(inst)
    c = world.trace_instanced(rays)
    with xr.Renderer(8, 8) as r:
        r.upload_scenes(scenes)
        r.set_instances(inst)
        g = r.trace_instanced(rays)
        assert r.stats().error_flags == 0
    for x, y in zip(g, c):
        assert np.array_equal(np.asarray(x).view(np.uint32), np.asarray(y).view(np.uint32))


@pytest.mark.parametrize("n", [40, 256, 1500, 2100])
@pytest.mark.parametrize("kind", ["nested", "far"])
def test_instances_that_do_not_cluster(kind, n, monkeypatch):
    """Boxes inside one another, of which a clustering makes a chain, and boxes whose merged
    areas overflow, which it cannot order."""
    monkeypatch.setenv("XR_TLAS_BUILDER", "ploc")
    rng = np.random.default_rng(n)
    scene = box_scene(rng, 6, 2.0)
    if kind == "nested":
        inst = [(0, affine(np.eye(3) * (1.0 + k / 64.0), [0, 0, 0])) for k in rng.permutation(n)]
    else:
        inst = [(0, affine(np.eye(3), list(rng.uniform(-1e20, 1e20, 3) * (k > 3)))) for k in range(n)]
    _check_world([scene], inst, random_rays(rng, 300, -4, 4))


@pytest.mark.parametrize("n", [1380, 1340])
def test_deep_chains_are_built(n):
    """Triangles inside one another cluster one by one: the deepest trees that are built have
    200 levels (these some 197 and 191), and rays that stay outside find them empty."""
    s = (1.0 + np.arange(n) / 64.0)[:, None, None]
    tri = s * np.array([[[-1.0, -1.0, -1.0], [1.0, 1.0, -1.0], [0.0, 0.0, 1.0]]])
    rays = random_rays(np.random.default_rng(n), 300, 30, 40)
    rays[:, 4:7] = np.abs(rays[:, 4:7])
    with xr.Renderer(8, 8) as r:
        r.upload_scene(_alone(tri))
        r.build_bvh()
        p, _, _ = r.trace(rays)
        st = r.stats()
    assert 185 <= st.bvh_depth <= 200 and (st.bvh_depth > 192) == (n == 1380)
    assert st.error_flags == 0 and np.all(p == -1)
