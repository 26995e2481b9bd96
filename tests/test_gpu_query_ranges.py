"""Ray queries over intervals that reach behind the origin: a closest hit is the hit of the
smallest t, also where that is negative, in a scene and in a world of instances."""
import numpy as np
import pytest

import xvk_ray_gb300 as xr
from oracle import binding as ob
from tests.helpers import affine, box_scene, random_rays, rotation

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("copies", [1, 3, 40])
@pytest.mark.parametrize("tmin,tmax", [(-30.0, 30.0), (-30.0, -0.5), (-2.0, 1e4)])
def test_closest_hit_behind_the_origin(copies, tmin, tmax):
    rng = np.random.default_rng(copies)
    # at most 256 triangles: the oracle tests every one, without boxes
    scenes = [box_scene(rng, 20, 3.0), box_scene(rng, 12, 2.0, light=False)]
    inst = [(k % 2, affine(rotation([1, 2, 3], 25.0 * k), list(rng.uniform(-6, 6, 3)))) for k in range(copies)]
    rays = random_rays(rng, 4000, -8, 8, tmin, tmax)
    world = ob.OracleWorld([ob.OracleScene.from_scene(s) for s in scenes])
    world.set_instances(inst)
    c = world.trace_instanced(rays)
    one = ob.OracleScene.from_scene(scenes[0]).trace(rays)
    assert ((c[0] >= 0) & (c[2] < 0)).mean() > 0.01
    with xr.Renderer(8, 8) as r:
        r.upload_scenes(scenes)
        r.set_instances(inst)
        g = r.trace_instanced(rays)
        ga = r.trace_instanced(rays, any_hit=True)
    for name, x, y in zip(("prim", "instance", "t", "bary"), g, c):
        assert np.array_equal(np.asarray(x).view(np.uint32), np.asarray(y).view(np.uint32)), name
    assert np.array_equal(ga[0] >= 0, c[0] >= 0)
    with xr.Renderer(8, 8) as r:
        r.upload_scene(scenes[0])
        r.build_bvh()
        p, t, _ = r.trace(rays)
    hit = one[0] >= 0
    assert np.array_equal(p, one[0]) and np.array_equal(t[hit].view(np.uint32), one[1][hit].view(np.uint32))
