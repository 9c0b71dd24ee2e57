"""The traversal with one ray per lane asked for by name, at counts of which a call
without a scheme gives each ray several lanes: leaves that overlap so much that
a warp holds several windows of 32 pending pairs (up to 24 per ray)."""
import numpy as np
import pytest

from crender_gb300 import api, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width,leaf_max", [(8, 3), (8, 1), (4, 2), (2, 3)])
@pytest.mark.parametrize("ntri,sigma", [(1, 0.5), (24, 0.5), (700, 0.5), (3000, 0.02)])
def test_lane_traversal_matches_oracle(ctx, orc, width, leaf_max, ntri, sigma):
    v = scenes.soup(ntri, 41, sigma)
    s = api.Scene(ctx, v, np.zeros(ntri, np.uint32), scenes.material_table([{}])).build(width, 0, leaf_max)
    b = orc.Bvh(v, width=width, leaf_max=leaf_max)
    try:
        for n in (1, 31, 32, 33, 127, 129, 1000, 16385):
            rays, srays = scenes.soup_rays(n, 42 + n), scenes.soup_rays(n, 43 + n, shadow=True)
            g = s.intersect(rays, traversal=api.TRAVERSAL_THREAD)
            assert np.array_equal(g.view(np.uint32), b.closest(rays).view(np.uint32))
            assert np.array_equal(s.intersect(srays, any_hit=True, traversal=api.TRAVERSAL_THREAD), b.any(srays))
    finally:
        s.close()
