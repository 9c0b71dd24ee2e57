"""Adjoint with material tables around the sizes at which its FP64 sums move from a
copy per warp to one per block (312, before 384) to global memory (1,536)."""
import numpy as np
import pytest

from crender_gb300 import api, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("spp", [3, 9])
@pytest.mark.parametrize("nmat", [312, 313, 384, 385, 1248, 1249, 1536, 1537])
def test_many_materials_match_oracle(ctx, orc, nmat, spp):
    """The oracle adds the same FP64 terms in another order: far below 1e-9."""
    sc = scenes.inverse_box(np.full((34, 3), 0.5), np.full(3, 0.6))
    used, r = len(sc["mats"]), np.random.default_rng(nmat)
    place = np.sort(np.r_[r.choice(nmat - 1, used - 1, replace=False), nmat - 1])  # the last one among them
    mats = np.repeat(sc["mats"][:1], nmat)
    mats[place] = sc["mats"]
    sc = dict(sc, mats=mats, mat_idx=place[sc["mat_idx"]].astype(np.uint32))
    st = api.make_settings(33, 9, spp, max_bounces=6, rr_depth=3, mode=1, seed=83, aspect=33 / 9)
    adj = r.normal(0, 1, 33 * 9 * 3).astype(np.float32)
    s = api.Scene(ctx, sc["verts"], sc["mat_idx"], sc["mats"]).build()
    bufs = [api.DeviceBuffer.from_array(ctx, adj), api.DeviceBuffer.from_array(ctx, np.zeros(3 * nmat)),
            api.DeviceBuffer.from_array(ctx, np.zeros(nmat))]
    try:
        api.backward(s, sc["camera"], st, *bufs)
        g_col, g_em = bufs[1].download(np.zeros(3 * nmat)), bufs[2].download(np.zeros(nmat))
    finally:
        for b in bufs:
            b.free()
        s.close()
    o_col, o_em = orc.adjoint(sc, sc["camera"], st, adj)
    assert np.abs(o_col).max() > 0
    for a, b in ((g_col, np.asarray(o_col).reshape(-1)), (g_em, np.asarray(o_em).reshape(-1))):
        assert np.abs(a - b).max() <= 1e-9 * max(np.abs(b).max(), 1e-12)
