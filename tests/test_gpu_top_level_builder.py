"""The two builders of the top-level BVH on both sides of the lines between them."""
import numpy as np
import pytest

import xvk_ray_gb300 as xr
from oracle import binding as ob
from tests.helpers import affine, box_scene, random_rays, rotation

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [31, 32, 33])
def test_top_level_builders_agree(n):
    """From 32 instances on, a frame with 4096 pixels an instance gets the other top-level
    builder: the same hits on both sides of both lines, and as the oracle's."""
    rng = np.random.default_rng(n)
    scenes = [box_scene(rng, 24, 3.0), box_scene(rng, 12, 2.0, light=False)]
    inst = [(k % len(scenes), affine(rotation([1, 2, 3], 20.0 * k), list(rng.uniform(-6, 6, 3)))) for k in range(n)]
    rays = random_rays(rng, 3000, -8, 8)
    world = ob.OracleWorld([ob.OracleScene.from_scene(s) for s in scenes])
    world.set_instances(inst)
    c = world.trace_instanced(rays)
    for w, h in ((8, 8), (512, 256), (512, 255)):
        with xr.Renderer(w, h) as r:
            r.upload_scenes(scenes)
            r.set_instances(inst)
            g = r.trace_instanced(rays)
            for a, b in zip(g, c):
                assert np.array_equal(np.asarray(a).view(np.uint32), np.asarray(b).view(np.uint32))
