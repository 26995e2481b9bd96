"""The radiance cache's kernels at the edges of their tiles of 128 samples, of one wave of
blocks and of the groups of threads that share a sample."""
import numpy as np
import pytest

import xvk_ray_gb300 as xr

pytestmark = pytest.mark.gpu

L = xr._lib


def _samples(n, seed=3):
    rng = np.random.default_rng(seed)
    s = np.zeros(n, xr.api.CACHE_SAMPLE_DTYPE)
    s["pos"] = rng.uniform(-0.9, 0.9, (n, 3))
    for name in ("normal", "wo"):
        d = rng.standard_normal((n, 3))
        s[name] = d / np.linalg.norm(d, axis=1, keepdims=True)
    s["albedo"] = rng.uniform(0.1, 0.9, (n, 3))
    s["roughness"] = rng.uniform(0.1, 1.0, n)
    s["kind"] = rng.choice([0, 1, 5], n)
    s["target"] = rng.exponential(0.5, (n, 3))
    return s


def _open():
    r = xr.Renderer(8, 8)
    r.cache.reset(11)
    r.cache.set_bounds((-1.0, -1.0, -1.0), 0.5)
    return r


@pytest.mark.parametrize("n", [1, 127, 128, 129, 152 * 3 * 128 + 1])
def test_queries_do_not_depend_on_the_batch(n):
    """A sample's prediction is its own: in any batch, tile and lane the same bits."""
    with _open() as r:
        s = _samples(152 * 3 * 128 + 300)
        whole = r.cache.query(s)
        assert np.isfinite(whole).all() and np.abs(whole).max() > 0
        part = r.cache.query(np.ascontiguousarray(s[-n:]))
        assert np.array_equal(part.view(np.uint32), whole[-n:].view(np.uint32))


@pytest.mark.parametrize("copies", [2, 256, 1024])
def test_gradients_of_repeated_tiles(copies):
    """The mean loss of a power of two of copies of a tile has the tile's gradients: every
    factor scales exactly, and what is left is the order of the sums: at most 8 K-steps of 7
    tiles a block and 152 blocks, 208 roundings of 2^-24 of the sum's absolute terms, which a
    layer's largest gradient exceeds a sixteenth of."""
    with _open() as r:
        s = _samples(128)
        loss1 = r.cache.train(s, apply=False)
        g1 = r.cache.read(L.XR_CACHE_MLP_GRAD)
        loss = r.cache.train(np.tile(s, copies), apply=False)
        g = r.cache.read(L.XR_CACHE_MLP_GRAD)
        assert abs(loss - loss1) <= 1e-4 * abs(loss1)
        for a in range(0, g.size, 4096):
            top = np.abs(g1[a:a + 4096]).max()
            assert top > 0
            assert np.abs(g[a:a + 4096] - g1[a:a + 4096]).max() <= 16 * 208 * 2.0 ** -24 * top
