"""Triangle tests shared by a warp (dyn_traverse): closest and any hits against
the oracle bit for bit at the edges of warps, blocks and block runs, and on
scenes whose leaves overlap so much that a warp holds several windows of 32
pending pairs (up to 24 per ray)."""
import numpy as np
import pytest

from crender_gb300 import api, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width,leaf_max", [(8, 3), (8, 1), (4, 2), (2, 3)])
@pytest.mark.parametrize("ntri,sigma", [(1, 0.5), (24, 0.5), (700, 0.5), (3000, 0.02)])
def test_shared_triangle_tests_match_oracle(ctx, orc, width, leaf_max, ntri, sigma):
    v = scenes.soup(ntri, 41, sigma)
    s = api.Scene(ctx, v, np.zeros(ntri, np.uint32), scenes.material_table([{}])).build(width, 0, leaf_max)
    b = orc.Bvh(v, width=width, leaf_max=leaf_max)
    try:
        for n in (1, 31, 32, 33, 127, 129, 1000):
            rays, srays = scenes.soup_rays(n, 42 + n), scenes.soup_rays(n, 43 + n, shadow=True)
            g, want = s.intersect(rays), b.closest(rays)
            assert np.array_equal(g.view(np.uint32), want.view(np.uint32))
            assert np.array_equal(s.intersect(srays, any_hit=True), b.any(srays))
    finally:
        s.close()


def test_many_block_runs(ctx, orc):
    """More rays than the blocks' runs hold at once, an odd count."""
    v = scenes.soup(5000, 44)
    s = api.Scene(ctx, v, np.zeros(len(v), np.uint32), scenes.material_table([{}])).build()
    b = orc.Bvh(v)
    n = 1_300_001
    try:
        rays, srays = scenes.soup_rays(n, 45), scenes.soup_rays(n, 46, shadow=True)
        g, ga = s.intersect(rays), s.intersect(srays, any_hit=True)
        idx = np.r_[np.random.default_rng(5).choice(n, 20_000, replace=False), n - 1]
        assert np.array_equal(g[idx].view(np.uint32), b.closest(np.ascontiguousarray(rays[idx])).view(np.uint32))
        assert np.array_equal(ga[idx], b.any(np.ascontiguousarray(srays[idx])))
    finally:
        s.close()


@pytest.mark.parametrize("width", [8, 4, 2])
@pytest.mark.parametrize("n", [1, 3, 5, 4095, 4096, 4097, 8192, 8193, 16384, 16385])
def test_few_rays(ctx, orc, width, n):
    """Counts around those at which a warp takes one ray, two, four or one per lane."""
    v = scenes.soup(3000, 47, 0.05)
    s = api.Scene(ctx, v, np.zeros(len(v), np.uint32), scenes.material_table([{}])).build(width, 1)
    b = orc.Bvh(v, width=width, treelet=1)
    try:
        rays, srays = scenes.soup_rays(n, 48), scenes.soup_rays(n, 49, shadow=True)
        assert np.array_equal(s.intersect(rays).view(np.uint32), b.closest(rays).view(np.uint32))
        assert np.array_equal(s.intersect(srays, any_hit=True), b.any(srays))
    finally:
        s.close()
