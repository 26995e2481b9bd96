"""The autotuner's candidates: what it tries beside a scene's own defaults."""
import numpy as np
import pytest

import xvk_ray_gb300 as xr
from tests.helpers import affine, camera_sequence

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("instances", [False, True])
def test_candidates_beside_the_defaults(instances):
    """Besides the defaults: two shading block counts, refills of 4, 6, 8, 12, 16 and 20 lanes
    and batches of 8, 16, 24 and 32 tests less the scene's own, two ray bundles, three temporal
    and two spatial block sizes."""
    scene = xr.Scene.cornell()
    with xr.Renderer(64, 64) as r:
        r.set_params(xr.params_default(64, 64))
        r.upload_scene(scene)
        r.build_bvh()
        if instances:
            r.set_instances([(0, affine(np.eye(3), [0, 0, 0]))])
        ubo = camera_sequence(scene, 64, 64, 1, 4)[0]
        t = r.autotune([[ubo]])
        assert r.stats().error_flags == 0
    assert t.configs_tried == 1 + 2 + 5 + 3 + 2 + 3 + 2
