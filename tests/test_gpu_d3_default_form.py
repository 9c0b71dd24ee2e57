"""The default form of a batch (no fusion level given) around the pool sizes at which
it changes, by films: every form gives the megakernel's."""
import pytest

from crender_gb300 import api
from test_gpu_c_render import _box_variant
from test_gpu_d_wavefront import _mega, _same

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("host_loop", [0, 1, 2])
@pytest.mark.parametrize("pool", [1 << 17, (1 << 17) + 1, 1 << 19])
def test_refilled_pools_match_megakernel(ctx, pool, host_loop):
    sc = _box_variant("materials")
    s = api.Scene(ctx, sc["verts"], sc["mat_idx"], sc["mats"]).build()
    st = api.make_settings(512, 300, 5, max_bounces=4, rr_depth=0, mode=1, seed=37, aspect=512 / 300)
    f = api.Film(ctx, st.width, st.height, f64=True)
    try:
        ctx.check(api.render_batch([s], [(0, sc["camera"], st)], [f], dict(path_pool=pool, host_loop=host_loop)))
        _same(f.download(f64=True), _mega(ctx, s, sc["camera"], st))
    finally:
        f.close()
        s.close()
