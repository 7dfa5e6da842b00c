"""Gathers of few AVPLs take the kernel that evaluates every pair: the same sums on both sides of the rule."""
import numpy as np
import pytest

from antiradiancecuts_b200 import _lib as L
from antiradiancecuts_b200 import api
from test_gpu_culled_gather import _inputs

pytestmark = pytest.mark.gpu


# 16 AVPLs at any size, up to 64 in at most 2^23 pairs: the AVPLs with and without one more that adds nothing
# (beside it: 512 x 256 x 64 = 2^23 with and without one more row of pixels)
@pytest.mark.parametrize("w,h,n", [(1, 1, 64), (37, 21, 64), (640, 480, 16), (640, 480, 1), (512, 256, 64),
                                   (512, 257, 64)])
@pytest.mark.parametrize("ar,precision", [(L.ARC_AR_DISK, L.ARC_PREC_KAHAN), (L.ARC_AR_CONE, L.ARC_PREC_FP64),
                                          (L.ARC_AR_NONE, L.ARC_PREC_FP64)])
def test_few_avpls_on_both_sides_of_the_rule(ctx, w, h, n, ar, precision):
    """The two kernels round a term differently: its cosines lie within 4 u of theirs, its inverse square
    distance within 4 u relative, and a sum of n adds n u: |sum - exact| <= (16 + n) u times the sum of the terms with
    cosines of 1, u = 2^-24 or 2^-53, on either side.  Disk antiradiance: the same terms, compensated.  The
    float planes are rounded once more."""
    pos, nrm, a = _inputs(w, h, n + 1, seed=w + n, flat=True)
    a["incRadiance"][n] = a["antiradiance"][n] = 0.0
    mats = (L.ArcMaterial * 3)()
    for i in range(3):
        mats[i].diffuse = L.f3((0.9, 0.5 / (i + 1), 0.25))
    ctx.upload_materials(mats)
    gb, planes = api.GBuffer(pos, nrm), []
    for k in (n, n + 1):
        out = api.Outputs(w, h)
        api.gather_bruteforce(ctx, ctx.upload_avpls(a[:k]), gb, (0.5, 0.5, -1.0),
                              api.gather_params(ar, 40.0, 0.02, 0.2, precision=precision), out)
        assert ctx.synchronize() == 0
        planes.append([t.cpu().numpy()[..., :3].astype(np.float64) for t in (out.radiance, out.antiradiance,
                                                                                out.result64)])
    want, got = planes
    assert (want[0] > 0).any() or n < 2 or not (nrm[..., 3] > 0).any()
    most = np.zeros((h, w, 1))
    for k in range(n):
        d2 = ((pos[..., :3].astype(np.float64) - a["position"][k].astype(np.float64)) ** 2).sum(-1, keepdims=True)
        most += float(max(a["incRadiance"][k].max(), a["antiradiance"][k].max())) / np.maximum(d2, 0.02 ** 2)
    u = 2.0 ** -24 if precision == L.ARC_PREC_KAHAN else 2.0 ** -53
    tol = 2 * (16 + n) * u * (0.9 / np.pi) * most
    ar_tol = 2.0 ** -22 * want[1] if ar == L.ARC_AR_DISK else tol + 2.0 ** -23 * want[1]
    assert np.all(np.abs(got[0] - want[0]) <= tol + 2.0 ** -23 * want[0])
    assert np.all(np.abs(got[1] - want[1]) <= ar_tol)
    assert np.all(np.abs(got[2] - want[2]) <= tol + ar_tol + 2.0 ** -50 * (want[0] + want[1]))
