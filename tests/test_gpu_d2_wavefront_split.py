"""Wavefront form, its split stages asked for by name: small batches take the
fused kernel by default, so what is tested here at small sizes gives `fuse`."""
import numpy as np
import pytest

from crender_gb300 import api
from test_gpu_c_render import _box_variant
from test_gpu_d_wavefront import OFF, _mega, _same

pytestmark = pytest.mark.gpu

TIMEOUT = 4  # CRG_ERR_TIMEOUT


@pytest.mark.parametrize("cap", [1, 3, 7])
@pytest.mark.parametrize("opts", [dict(fuse=1), dict(fuse=1, path_pool=96), dict(fuse=1, path_pool=96, refill=OFF),
                                  dict(fuse=2, path_pool=96), dict(fuse=3, path_pool=96)])
@pytest.mark.parametrize("host_loop", [1, 2])
def test_iteration_cap_in_the_host_driven_loop(ctx, opts, cap, host_loop):
    """The host polls every eighth iteration only, so iterations follow the one that
    reached the cap: they take up nothing, and the same context then renders."""
    sc = _box_variant("materials")
    s = api.Scene(ctx, sc["verts"], sc["mat_idx"], sc["mats"]).build()
    st = api.make_settings(32, 32, 3, max_bounces=8, rr_depth=0, mode=1, seed=6)
    view = [(0, sc["camera"], st)]
    f, g = api.Film(ctx, 32, 32, f64=True), api.Film(ctx, 32, 32, f64=True)
    try:
        stats = []
        for loop in (0, host_loop):  # the graph stops at the cap itself
            assert api.render_batch([s], view, [f], dict(opts, max_iterations=cap, host_loop=loop)) == TIMEOUT
            stats.append(api.batch_stats(ctx))
            f.reset()
        assert stats[0] == stats[1] and stats[0]["iterations"] == cap
        ctx.check(api.render_batch([s], view, [g], dict(opts, host_loop=host_loop)))
        _same(g.download(f64=True), _mega(ctx, s, sc["camera"], st))
    finally:
        f.close()
        g.close()
        s.close()
