"""Host arrays staged in the pool or, from 32 MB on, in a block of their own: the same hits
as the device entry point gives, at one ray and on both sides of the line."""
import numpy as np
import pytest
import torch

import xvk_ray_gb300 as xr
from tests.helpers import random_rays

pytestmark = pytest.mark.gpu

L = xr._lib
LINE = (32 << 20) // 48   # 32 B of ray and 16 B of results each


@pytest.mark.parametrize("n", [1, LINE, LINE + 1])
def test_host_trace_equals_device_trace(n):
    rays = np.tile(random_rays(np.random.default_rng(5), 4096, -0.9, 0.9), (n // 4096 + 1, 1))[:n].astype(np.float32)
    rays = np.ascontiguousarray(rays)
    with xr.Renderer(8, 8) as r:
        r.upload_scene(xr.Scene.cornell())
        r.build_bvh()
        d = torch.from_numpy(rays).cuda()
        prim = torch.empty(n, dtype=torch.int32, device="cuda")
        t, bary = torch.empty(n, device="cuda"), torch.empty(n, 2, device="cuda")
        torch.cuda.synchronize()
        L.check(L.load().xr_trace_rays_device(r.ctx, d.data_ptr(), n, 0, prim.data_ptr(), t.data_ptr(),
                                              bary.data_ptr()), r.ctx)
        r.sync()
        for _ in range(2):   # the second call finds the pool's block
            hp, ht, hb = r.trace(rays, False)
            assert np.array_equal(hp, prim.cpu().numpy())
            assert np.array_equal(ht.view(np.uint32), t.cpu().numpy().view(np.uint32))
            assert np.array_equal(hb.view(np.uint32), bary.cpu().numpy().view(np.uint32))
