"""The culled gather (records tested against a tile's bounds before the pair loops): the same pixels
gathered in tiles whose bounds are too wide to drop any record, at the edges of tiles, chunks and
segments, over pixels and AVPLs of arbitrary orientation."""
import numpy as np
import pytest

from antiradiancecuts_b200 import _lib as L
from antiradiancecuts_b200 import api
from antiradiancecuts_b200.scene import AVPL_DTYPE

pytestmark = pytest.mark.gpu

# Both gathers add the same FP32 terms (all >= 0) and differ in their order alone: a chunk's partial is
# at most 128 sequential FP32 additions of each half, so each sum lies within 128 x 2^-24 of the exact
# sum of its terms and two of them within twice that (the partials are added in FP64).  All-FP64: at
# most one addition per AVPL.
TOL = {L.ARC_PREC_KAHAN: lambda n: 2 * 128 * 2.0 ** -24, L.ARC_PREC_FP64: lambda n: 2 * (n + 8) * 2.0 ** -53}


def _inputs(w, h, n, seed, flat):
    """Random pixels (flat: one axis-aligned wall per 24 columns, as in a room) and AVPLs on and off
    the walls; some without radiance, without antiradiance, without a direction, with a long one."""
    r = np.random.default_rng(seed)
    unit = lambda v: v / np.linalg.norm(v, axis=-1, keepdims=True)  # noqa: E731
    pos = np.zeros((h, w, 4), np.float32)
    nrm = np.zeros((h, w, 4), np.float32)
    pos[..., :3], pos[..., 3] = r.random((h, w, 3)), 1.0
    nrm[..., :3] = unit(r.normal(size=(h, w, 3)))
    if flat:
        for x in range(w):
            axis, side = (x // 24) % 3, (x // 72) % 2
            pos[:, x, axis] = side
            nrm[:, x, :3] = 0.0
            nrm[:, x, axis] = 1.0 - 2.0 * side
    nrm[..., 3] = r.integers(0, 3, (h, w))  # material 0: no surface
    a = np.zeros(n, AVPL_DTYPE)
    a["position"] = r.random((n, 3))
    a["normal"] = unit(r.normal(size=(n, 3)))
    wall = r.random(n) < 0.6
    axis, side = r.integers(0, 3, n), r.integers(0, 2, n)
    a["position"][wall, axis[wall]] = side[wall]
    a["normal"][wall] = 0.0
    a["normal"][wall, axis[wall]] = 1.0 - 2.0 * side[wall]
    a["incDirection"] = unit(r.normal(size=(n, 3))) * np.where(r.random((n, 1)) < 0.1, 1.5, 1.0)
    a["incRadiance"], a["antiradiance"] = r.random((n, 3)), r.random((n, 3))
    a["incRadiance"][r.random(n) < 0.2] = 0.0
    a["antiradiance"][r.random(n) < 0.4] = 0.0
    a["incDirection"][r.random(n) < 0.05] = 0.0
    a["materialIndex"] = r.integers(0, 3, n)
    return pos, nrm, a


def _gather(ctx, pos, nrm, a, ar, precision, clamp):
    mats = (L.ArcMaterial * 3)()
    for i in range(1, 3):
        mats[i].diffuse = L.f3((0.9, 0.5 / i, 0.25))
    mats[0].diffuse = L.f3((0.3, 0.3, 0.3))
    ctx.upload_materials(mats)
    dv = ctx.upload_avpls(a)
    h, w = pos.shape[:2]
    out = api.Outputs(w, h)
    api.gather_bruteforce(ctx, dv, api.GBuffer(pos, nrm), (0.5, 0.5, -1.0),
                          api.gather_params(ar, 40.0, clamp, precision=precision), out)
    assert ctx.synchronize() == 0
    return [t.cpu().numpy()[..., :3].astype(np.float64) for t in (out.radiance, out.antiradiance, out.result64)]


def _among_outliers(pos, nrm):
    """The pixels with two columns of far, opposite pixels in every 16-column tile."""
    h, w = pos.shape[:2]
    cols = np.arange(w)
    at = cols // 14 * 16 + cols % 14
    wide = (w + 13) // 14 * 16
    p, n = np.zeros((h, wide, 4), np.float32), np.zeros((h, wide, 4), np.float32)
    p[:, at], n[:, at] = pos, nrm
    for col, s in ((14, -1.0), (15, 1.0)):
        p[:, col::16, :3], n[:, col::16, :3], n[:, col::16, 3] = 99.0 * s, s / np.sqrt(3.0), 1.0
    return p, n, at


@pytest.mark.parametrize("ar", [L.ARC_AR_NONE, L.ARC_AR_CONE])
@pytest.mark.parametrize("size", [(1, 1, 1), (15, 17, 2), (16, 32, 255), (33, 31, 256), (80, 33, 257), (100, 70, 1537),
                                  (16, 16, 20011)])
def test_culled_records_add_nothing(ctx, size, ar):
    for flat, clamp in ((False, 0.02), (True, 0.02), (True, 0.0)):
        pos, nrm, a = _inputs(*size, seed=sum(size) + flat, flat=flat)
        wide_pos, wide_nrm, at = _among_outliers(pos, nrm)
        for precision, tol in TOL.items():
            want = [v[:, at] for v in _gather(ctx, wide_pos, wide_nrm, a, ar, precision, clamp)]
            got = _gather(ctx, pos, nrm, a, ar, precision, clamp)
            scale = want[0] + want[1]
            assert (want[0] > 0).any() or size[2] < 3
            # (the float planes are rounded once more)
            assert np.all(np.abs(got[0] - want[0]) <= (tol(size[2]) + 2.0 ** -23) * want[0])
            assert np.all(np.abs(got[1] - want[1]) <= (tol(size[2]) + 2.0 ** -23) * want[1])
            assert np.all(np.abs(got[2] - want[2]) <= tol(size[2]) * (1 + 1e-6) * scale)


def test_records_without_finite_radiance_are_not_dropped(ctx):
    pos, nrm, a = _inputs(40, 40, 600, seed=3, flat=True)
    a["incRadiance"][17] = np.inf
    a["antiradiance"][400] = np.nan
    for precision in (L.ARC_PREC_KAHAN, L.ARC_PREC_FP64):
        want = _gather(ctx, pos, nrm, a, L.ARC_AR_CONE, L.ARC_PREC_NAIVE, 0.02)
        got = _gather(ctx, pos, nrm, a, L.ARC_AR_CONE, precision, 0.02)
        assert np.array_equal(np.isfinite(got[2]), np.isfinite(want[2]))


@pytest.mark.parametrize("size", [(1, 1, 1), (16, 16, 1023), (17, 33, 1024), (40, 31, 1025), (70, 50, 5003),
                                  (800, 800, 301)])
def test_culled_disk_antiradiance_equals_every_pair(ctx, size):
    """Each disk term is A or nothing, added in AVPL order with a compensated sum by both kernels: the
    same sums, rounded once to float."""
    for flat, radius in ((False, 0.2), (True, 0.03), (True, 0.2)):
        pos, nrm, a = _inputs(*size, seed=sum(size) + flat, flat=flat)
        mats = (L.ArcMaterial * 3)()
        for i in range(3):
            mats[i].diffuse = L.f3((0.9, 0.5 / (i + 1), 0.25))
        ctx.upload_materials(mats)
        dv, gb = ctx.upload_avpls(a), api.GBuffer(pos, nrm)
        outs = []
        for precision in (L.ARC_PREC_KAHAN_STRICT, L.ARC_PREC_KAHAN):
            out = api.Outputs(size[0], size[1])
            api.gather_bruteforce(ctx, dv, gb, (0.5, 0.5, -1.0),
                                  api.gather_params(L.ARC_AR_DISK, 40.0, 0.02, radius, precision=precision), out)
            assert ctx.synchronize() == 0
            outs.append([t.cpu().numpy()[..., :3].astype(np.float64) for t in (out.antiradiance, out.radiance,
                                                                                out.result, out.result64)])
        want, got = outs
        assert (want[0] > 0).any() or size[2] < 2
        assert np.all(np.abs(got[0] - want[0]) <= 2.0 ** -22 * want[0])
        # the result is the FP64 difference of the gather's own radiance and antiradiance
        assert np.all(np.abs(got[3] - (got[1] - got[0])) <= 2.0 ** -23 * (got[1] + got[0]))
        assert np.array_equal(got[2], got[3].astype(np.float32))
