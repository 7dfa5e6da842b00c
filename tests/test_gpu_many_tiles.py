"""Frames of very many tiles: the learned cut's list passes split their tiles into groups, and their
slabs' counts are bounded."""
import numpy as np
import pytest

import helpers as H
from antiradiancecuts_b200 import _lib as L
from antiradiancecuts_b200 import api, learned

pytestmark = pytest.mark.gpu


# 50,177 tiles: the counting pass in two groups; 226,721: fewer slabs than the chip would take
@pytest.mark.parametrize("tiles", [50177, 226721])
def test_learned_lists_of_many_tiles(ctx, tiles):
    """Threshold 1 never refines below the band, so the lists are those of the error-bound cut at
    band * eps, tile by tile."""
    d = H.workload("boxes2_720p_64k", 640, 360, 200)
    # one row of tiles: eight pixels of the image each
    w = 8 * tiles
    pick = (np.arange(w) * 7 + np.arange(w) // 8 * 13) % (640 * 360)
    pos, nrm = (np.ascontiguousarray(d[k].reshape(-1, 4)[pick][None]) for k in ("pos", "nrm"))
    ctx.upload_materials(d["mats"])
    bvh = api.AvplBvh(ctx)
    bvh.build(ctx.upload_avpls(d["avpls"]))
    gb, out = api.GBuffer(pos, nrm), api.Outputs(w, 1, parts=False, fp64=False)
    model = learned.Model(ctx, seed=5, loss=L.ARC_MLP_LOSS_BCE)
    eps, band = float(np.float32(0.2)), 4.0
    room = dict(max_cut_nodes=1024, cut_pool_entries=1024 * tiles)
    cuts = []
    for cut in (api.cut_params(L.ARC_CUT_ERROR_BOUND, error_bound=eps * band, **room),
                api.cut_params(L.ARC_CUT_LEARNED, error_bound=eps, mlp_band=band, model=model.handle.value,
                               mlp_threshold=1.0, **room)):
        api.gather_cut(ctx, bvh, None, gb, d["cam"], api.gather_params(L.ARC_AR_CONE, 30.0, 0.01), cut, out)
        assert ctx.synchronize() == 0
        cuts.append(api.last_cut(ctx))
    assert len(cuts[0]) == tiles
    assert all(np.array_equal(a, b) for a, b in zip(*cuts))
    assert len({len(c) for c in cuts[0]}) > 3
    model.close()
    bvh.close()
