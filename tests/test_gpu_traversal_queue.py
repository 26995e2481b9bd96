"""The traversal's queue of triangle tests and its helper lanes at their edges, against
the oracle bit for bit: ray counts around a warp (the last rays of a launch are shared
out to idle lanes), nodes whose leaves are hit many at a time (more tests per lane than
one round pushes), batches from one test to a whole warp's, refills from one lane to all.
"""
import numpy as np
import pytest

import xvk_ray_gb300 as xr
from oracle import binding as ob

pytestmark = pytest.mark.gpu


def _soup(n, size, seed):
    """n triangles of up to `size` units around the origin: large ones overlap, so that a
    ray meets most leaves of a node; a few of them twice, so that hits tie."""
    rng = np.random.default_rng(seed)
    c = rng.uniform(-1, 1, (n, 1, 3))
    p = (c + rng.uniform(-size, size, (n, 3, 3))).astype(np.float32)
    p[1::37] = p[0::37][: len(p[1::37])]
    v = np.zeros((3 * n, 9), np.float32)
    v[:, :3] = p.reshape(-1, 3)
    v[:, 4] = 1.0
    base = xr.Scene.cornell()
    return xr.Scene(v, np.arange(3 * n, dtype=np.uint32), base.materials[:1].copy(), np.zeros((1, 2), np.uint32),
                    base.camera)


def _rays(n, seed):
    rng = np.random.default_rng(seed)
    r = np.zeros((n, 8), np.float32)
    r[:, :3] = rng.uniform(-2.5, 2.5, (n, 3))
    d = rng.uniform(-0.6, 0.6, (n, 3)) - r[:, :3]
    r[:, 4:7] = d / np.linalg.norm(d, axis=1, keepdims=True)
    r[:, 3], r[:, 7] = 1e-4, 1e4
    r[::5, 7] = 1.5          # some end before the far side
    return r


@pytest.mark.parametrize("n_rays", [1, 2, 31, 32, 33, 1000])
@pytest.mark.parametrize("tris,size", [(9, 1.0), (3000, 0.02), (3000, 0.8)])
def test_few_rays_and_crowded_nodes(n_rays, tris, size):
    scene, rays = _soup(tris, size, tris + n_rays), _rays(n_rays, n_rays)
    osc = ob.OracleScene.from_scene(scene)
    op, ot, obary = osc.trace(rays)
    hit = op >= 0
    with xr.Renderer(8, 8) as r:
        r.upload_scene(scene)
        r.build_bvh()
        for refill, batch in ((0, 0), (1, 1), (32, 32), (8, 5)):
            r.set_tuning(refill_min=refill, postpone_below=batch)
            gp, gt, gb = r.trace(rays)
            assert np.array_equal(gp, op), (refill, batch)
            assert np.array_equal(gt[hit].view(np.uint32), ot[hit].view(np.uint32))
            assert np.array_equal(gb[hit].view(np.uint32), obary[hit].view(np.uint32))
            ga, _, _ = r.trace(rays, any_hit=True)
            assert np.array_equal(ga >= 0, hit), (refill, batch)
        assert r.stats().error_flags == 0


@pytest.mark.parametrize("n_rays", [1, 31, 33, 1000])
@pytest.mark.parametrize("copies", [1, 7, 40])
def test_few_rays_in_an_instanced_world(n_rays, copies):
    """Overlapping instances of crowded soups: lanes that wait for their tests before they
    leave an instance, and for others before they enter one; groups beyond the closest hit
    are dropped."""
    rng = np.random.default_rng(copies)
    scenes = [_soup(200, 0.5, 1), _soup(9, 1.0, 2)]
    inst = []
    for i in range(copies):
        m = np.zeros((3, 4), np.float32)
        m[:, :3] = np.linalg.qr(rng.standard_normal((3, 3)))[0] * rng.uniform(0.4, 1.5)
        m[:, 3] = rng.uniform(-1, 1, 3)
        inst.append((i % 2, m))
    world = ob.OracleWorld([ob.OracleScene.from_scene(s) for s in scenes])
    world.set_instances(inst)
    rays = _rays(n_rays, n_rays)
    c = world.trace_instanced(rays)
    with xr.Renderer(8, 8) as r:
        r.upload_scenes(scenes)
        r.set_instances(inst)
        for refill, batch in ((0, 0), (1, 1), (32, 32)):
            r.set_tuning(refill_min=refill, postpone_below=batch)
            g = r.trace_instanced(rays)
            for name, x, y in zip(("prim", "instance", "t", "bary"), g, c):
                assert np.array_equal(np.asarray(x).view(np.uint32), np.asarray(y).view(np.uint32)), (name, refill, batch)
            assert np.array_equal(r.trace_instanced(rays, any_hit=True)[0] >= 0, c[0] >= 0)
        assert r.stats().error_flags == 0
