"""Clustered deferred antiradiance without a caller that reads the clusters (info NULL, and so every
arc_run): against the gather that evaluates every pair, and against the cluster lists."""
import ctypes as C
import math

import numpy as np
import pytest

import helpers as H
from antiradiancecuts_b200 import _lib as L
from antiradiancecuts_b200 import api, scene

pytestmark = pytest.mark.gpu

# Every side adds the same terms with compensated FP32 sums: each within 2^-22 of the exact sum, and two
# of them, rounded once more to float, within twice that.
TOL = 2.0 ** -21


@pytest.fixture(scope="module")
def case(ctx):
    d = H.workload("boxes2_720p_64k", 96, 64, 8192)
    r = H.disk_radius(d["desc"])
    ctx.upload_materials(d["mats"])
    dv, gb, out = api.DeviceAvpls(d["avpls"]), api.GBuffer(d["pos"], d["nrm"]), api.Outputs(96, 64)
    api.gather_bruteforce(ctx, dv.param, gb, d["cam"],
                          api.gather_params(L.ARC_AR_DISK, 30.0, 0.01, r, precision=L.ARC_PREC_KAHAN_STRICT), out)
    assert ctx.synchronize() == 0
    planes = [p.cpu().numpy()[..., :3].astype(np.float64) for p in (out.radiance, out.antiradiance)]
    assert (planes[1] > 0).mean() > 0.05
    return d, dv, gb, r, planes


def test_clustered_without_info_equals_every_pair(ctx, case):
    d, dv, gb, r, (_, want) = case
    prm, cp = api.gather_params(L.ARC_AR_DISK, 30.0, 0.0, r), L.ArcClusterParams(0.1, math.radians(30.0))
    for info in (None, L.ArcClusterInfo()):
        out = api.Outputs(96, 64)
        L.check(ctx.lib.arc_antiradiance_clustered(ctx.handle, C.byref(dv.param), C.byref(gb.view()), L.f3(d["cam"]),
                                                   C.byref(cp), C.byref(prm), C.byref(out.view()),
                                                   C.byref(info) if info is not None else None), "clustered")
        assert ctx.synchronize() == 0
        assert np.all(np.abs(out.antiradiance.cpu().numpy()[..., :3] - want) <= TOL * want)
        assert np.all(np.abs(out.result64.cpu().numpy() - want) <= TOL * want)


@pytest.mark.parametrize("clustered", [0, 1])
def test_run_with_disk_antiradiance_equals_every_pair(ctx, case, clustered):
    """arc_run without light cuts, the disk radius from its photon radius scale."""
    d, _, gb, r, (rad, ar) = case
    g = api.CudaGather(ctx, gb, d["mats"])
    cfg = api.run_config(useLightCuts=0, ar_kind=L.ARC_AR_DISK, useClusteredDeferred=clustered, dist_clamp=0.01,
                         cluster_theta=math.radians(0.5 * d["desc"].camera_fov_deg))
    out = g.run(d["avpls"], d["cam"], scene.scene_extent(d["desc"]), cfg)
    assert ctx.synchronize() == 0
    assert np.all(np.abs(out.antiradiance.cpu().numpy()[..., :3] - ar) <= TOL * ar)
    # radiance: per-chunk FP32 partials of up to 128 additions on one side
    assert np.all(np.abs(out.result64.cpu().numpy() - (rad - ar)) <= TOL * ar + 256 * 2.0 ** -23 * (rad + ar))
