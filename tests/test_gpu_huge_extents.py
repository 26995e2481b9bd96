"""Scenes of more than 2^113 grid cells' extent along an axis, whose stored cell is infinite:
the box test leaves that axis out, and hits are the oracle's."""
import numpy as np
import pytest

import xvk_ray_gb300 as xr
from oracle import binding as ob
from tests.helpers import affine
from tests.test_gpu_build_degenerate import _alone

pytestmark = pytest.mark.gpu


def _case(axis, big):
    """A triangle `big` long along one axis and rays that cross it near the origin."""
    tri = np.array([[-big, -1.0, 0.0], [big, -1.0, 0.0], [0.0, 1.0, 0.0]])
    rng = np.random.default_rng(axis)
    n = 2000
    rays = np.zeros((n, 8), np.float32)
    o = np.stack([rng.uniform(-3, 3, n), rng.uniform(-2, 2, n), np.full(n, 5.0)], 1)
    d = np.stack([rng.uniform(-0.1, 0.1, n), rng.uniform(-0.1, 0.1, n), np.full(n, -1.0)], 1)
    roll = lambda a: np.roll(a, axis, axis=-1)
    rays[:, :3], rays[:, 4:7] = roll(o), roll(d)
    rays[:, 3], rays[:, 7] = 1e-4, 1e4
    return _alone(roll(tri)[None]), rays


@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("big", [2.0 ** 118, 2.0 ** 121, 2.0 ** 123])
def test_one_axis_of_huge_extent(axis, big):
    scene, rays = _case(axis, big)
    osc = ob.OracleScene.from_scene(scene)
    c = osc.trace(rays)
    assert 0.2 < (c[0] >= 0).mean() < 0.9
    with xr.Renderer(8, 8) as r:
        r.upload_scene(scene)
        r.build_bvh()
        g = r.trace(rays)
        assert r.stats().error_flags == 0
    hit = c[0] >= 0
    assert np.array_equal(g[0], c[0])
    assert np.array_equal(g[1][hit].view(np.uint32), c[1][hit].view(np.uint32))


@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("big", [2.0 ** 118, 2.0 ** 121, 2.0 ** 123])
def test_an_instance_of_huge_extent(axis, big):
    scene, rays = _case(axis, big)
    world = ob.OracleWorld([ob.OracleScene.from_scene(scene)])
    inst = [(0, affine(np.eye(3), [0, 0, 0])), (0, affine(np.eye(3), [0, 0.5, 0]))]
    world.set_instances(inst)
    c = world.trace_instanced(rays)
    with xr.Renderer(8, 8) as r:
        r.upload_scenes([scene])
        r.set_instances(inst)
        g = r.trace_instanced(rays)
        assert r.stats().error_flags == 0
    for x, y in zip(g, c):
        assert np.array_equal(np.asarray(x).view(np.uint32), np.asarray(y).view(np.uint32))
