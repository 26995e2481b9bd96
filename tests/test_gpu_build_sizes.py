"""BVH builds at the sizes where the builder changes its way (one-block sort, one-block end
of the clustering, several lanes per cluster, blocks of the sort and the compaction), with
coincident triangles: hits against the oracle bit for bit, every level accounted for."""
import numpy as np
import pytest

import xvk_ray_gb300 as xr
from oracle import binding as ob
from tests.test_gpu_traversal_queue import _rays, _soup

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("builder", ["ploc", "lbvh"])
@pytest.mark.parametrize("n", [2, 4, 64, 65, 129, 1023, 1025, 2047, 2048, 2049, 2561, 65535, 65537, 66561])
def test_build_sizes(n, builder, monkeypatch):
    monkeypatch.setenv("XR_BVH_BUILDER", builder)
    scene, rays = _soup(n, 2.0 / n ** 0.5, n), _rays(500, n)
    with xr.Renderer(8, 8) as r:
        r.upload_scene(scene)
        for _ in range(2):      # a rebuild reuses the pool's memory
            r.build_bvh()
            gp, gt, gb = r.trace(rays)
        st = r.stats()
    op, ot, obary = ob.OracleScene.from_scene(scene).trace(rays)
    hit = op >= 0
    assert st.error_flags == 0 and st.bvh_triangles == n
    assert np.array_equal(gp, op)
    assert np.array_equal(gt[hit].view(np.uint32), ot[hit].view(np.uint32))
    assert np.array_equal(gb[hit].view(np.uint32), obary[hit].view(np.uint32))
