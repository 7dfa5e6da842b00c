"""A tree whose links form a cycle: the walks are bounded, report it and mark the pixels."""
import ctypes as C
import math

import numpy as np
import pytest

from antiradiancecuts_b200 import _lib as L
from antiradiancecuts_b200 import api
from antiradiancecuts_b200.scene import AVPL_DTYPE

pytestmark = pytest.mark.gpu


def test_solid_angle_walk_that_runs_out_marks_every_pixel_it_left(ctx):
    """Two pixels of a warp: one walks into an inner node that is its own child, the other only still has a
    leaf to visit when the walk's budget ends.  Neither may keep a partial sum."""
    a = np.zeros(3, AVPL_DTYPE)
    a["position"] = [(0.9, 0.45, 0.45), (0.1, 0.45, 0.45), (0.2, 0.45, 0.45)]
    a["normal"] = [(-1.0, 0.0, 0.0), (1.0, 0.0, 0.0), (1.0, 0.0, 0.0)]
    a["incRadiance"] = 1.0
    mats = (L.ArcMaterial * 2)()
    mats[1].diffuse = L.f3((0.5, 0.5, 0.5))
    ctx.upload_materials(mats)
    bvh = api.AvplBvh(ctx)
    dv = ctx.upload_avpls(a)
    bvh.build(dv)
    v = bvh.view()
    tree = bvh.host_arrays()
    # the root holds the leaf at x = 0.9 (sorted last) and inner node 1 over the other two
    bounds = tree["bounds"].copy()
    links = bounds.view(np.int32)
    assert bounds[1, 4] < 0.5 and {tree["left"][0], tree["right"][0]} == {-2, 2}
    links[0, 3], links[0, 7] = 2, -2  # the inner node is visited first
    links[1, 3], links[1, 7] = -2, 0  # and is its own child
    L.check(ctx.lib.arc_copy_h2d(ctx.handle, C.c_void_p(v.bounds), bounds.ctypes.data, bounds.nbytes), "copy")
    pos, nrm = np.zeros((1, 2, 4), np.float32), np.zeros((1, 2, 4), np.float32)
    pos[..., :3], nrm[..., 3] = 0.5, 1.0
    nrm[0, 0, 0], nrm[0, 1, 0] = 1.0, -1.0  # pixel 0 sees the leaf alone, pixel 1 the inner node
    out = api.Outputs(2, 1)
    api.gather_cut(ctx, bvh, dv, api.GBuffer(pos, nrm), (0.5, 0.5, 0.5), api.gather_params(L.ARC_AR_NONE),
                   api.cut_params(L.ARC_CUT_SOLID_ANGLE, solid_angle_threshold=1e-6 * math.pi), out)
    assert ctx.synchronize() == L.ARC_DEVERR_BAD_NODE
    assert np.array_equal(out.radiance.cpu().numpy()[0, :, :3], [[1e5, 0.0, 1e5]] * 2)
    bvh.close()
