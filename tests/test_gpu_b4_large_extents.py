"""Axis-parallel rays through scenes of great extent: a zero direction component
is taken as 2^-80 in the box tests, whose products with a node's quantum then
come near the largest float.  The rays go through points of triangles."""
import numpy as np
import pytest

from crender_gb300 import api, scenes

pytestmark = pytest.mark.gpu


def axis_rays(v, n, extent, seed):
    """Rays along the axes through random points of random triangles, zeros of both signs."""
    r = np.random.default_rng(seed)
    t = v.reshape(-1, 3, 3).astype(np.float64)
    k, row = r.integers(0, len(t), n), np.arange(n)
    p = (t[k] * r.dirichlet((1, 1, 1), n)[:, :, None]).sum(1)
    axis, sign = r.integers(0, 3, n), r.choice([-1.0, 1.0], n)
    d = np.where(r.random((n, 3)) < 0.5, np.float32(0.0), np.float32(-0.0))
    d[row, axis] = sign
    p[row, axis] -= 4.0 * extent * sign
    rays = np.zeros(n, scenes.RAY_DTYPE)
    rays["org"], rays["dir"], rays["tmin"], rays["tmax"] = p, d, 1e-5, np.inf
    return rays


@pytest.mark.parametrize("width", [8, 4, 2])
@pytest.mark.parametrize("log2", [30, 38, 39, 40, 41, 42])
def test_axis_parallel_rays_match_oracle(ctx, orc, width, log2):
    extent = 2.0 ** log2
    v = np.ascontiguousarray((scenes.soup(700, 5, 0.1) * np.float32(extent)).astype(np.float32))
    s = api.Scene(ctx, v, np.zeros(len(v), np.uint32), scenes.material_table([{}])).build(width)
    b = orc.Bvh(v, width=width)
    try:
        rays = axis_rays(v, 20_000, extent, log2)
        want = b.closest(rays)
        assert (want.view(np.uint32).reshape(len(rays), -1)[:, 1] != 0xFFFFFFFF).all()
        for n in (1000, 20_000):  # a group of lanes to a ray, a lane to a ray
            assert np.array_equal(s.intersect(rays[:n]).view(np.uint32), want[:n].view(np.uint32))
            assert (s.intersect(rays[:n], any_hit=True) == 1).all()
    finally:
        s.close()
