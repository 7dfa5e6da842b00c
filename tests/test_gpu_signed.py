"""AVPLs with negative components (radiance and antiradiance are signed sums in a program that
subtracts one set from another)."""
import numpy as np
import pytest

import helpers as H
from antiradiancecuts_b200 import _lib as L
from antiradiancecuts_b200 import api
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mixed", [False, True])
def test_error_bound_cut_of_signed_avpls_identical(ctx, mixed):
    """The selection's approximate bound must leave the same decisions to the rounded one whatever the
    signs of the sums: every tile's list equals the oracle's, at bounds around those of the upper nodes."""
    w, h, n = 640, 360, 4096
    d = H.workload("boxes2_720p_64k", w, h, n)
    a = d["avpls"].copy()
    r = np.random.default_rng(4)
    if mixed:
        a["incRadiance"][r.random(n) < 0.7] *= -1.0
        a["antiradiance"][r.random(n) < 0.5] *= -1.0
    else:
        a["incRadiance"] *= -1.0
    ctx.upload_materials(d["mats"])
    bvh = api.AvplBvh(ctx)
    bvh.build(ctx.upload_avpls(a))
    tree, gb, out = bvh.host_arrays(), api.GBuffer(d["pos"], d["nrm"]), api.Outputs(w, h)
    bad, total = 0, 0
    for eps in np.geomspace(0.3, 100, 24).astype(np.float32):
        api.gather_cut(ctx, bvh, None, gb, d["cam"], api.gather_params(L.ARC_AR_CONE, 30.0, 0.01),
                       api.cut_params(L.ARC_CUT_ERROR_BOUND, error_bound=float(eps)), out)
        assert ctx.synchronize() == 0
        got = api.last_cut(ctx)
        want, _, over = O.tile_cut(d["pos"], d["nrm"], tree, d["dif"], float(eps), 0.01, 2, 30.0, max_cut=65536)
        assert over == 0
        bad += sum(not np.array_equal(x, y) for x, y in zip(got, want))
        total += sum(map(len, want))
    assert bad == 0 and total > 24 * len(want)
    bvh.close()
