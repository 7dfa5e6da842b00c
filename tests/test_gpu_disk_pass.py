"""The culled disk antiradiance far from the origin, against the gather that
evaluates every pair with the same terms (per-term Kahan)."""
import numpy as np
import pytest

from antiradiancecuts_b200 import _lib as L
from antiradiancecuts_b200 import api
from antiradiancecuts_b200.scene import AVPL_DTYPE

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("far", [0.0, 1e3, 1e4, 1e5])
def test_disk_antiradiance_far_from_the_origin(ctx, far):
    """A wall of pixels 0.003 apart, hit by rays within a disk of 0.01: the rounding of a coordinate is
    not small against the radius there, but the differences of positions that decide are exact."""
    r = np.random.default_rng(11)
    w, h, n, radius = 96, 64, 6000, 0.01
    at = np.array([far, 0.7 * far, far / 3])
    y, x = np.mgrid[0:h, 0:w]
    pos, nrm = np.zeros((h, w, 4), np.float32), np.zeros((h, w, 4), np.float32)
    pos[..., :3] = at + np.stack([0.003 * x, 0.003 * y, 0.0 * x], -1)
    nrm[..., 2:] = 1.0
    a = np.zeros(n, AVPL_DTYPE)
    d = r.normal(size=(n, 3))
    d[:, 2] = -np.abs(d[:, 2]) - 0.2
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    aim = pos[r.integers(0, h, n), r.integers(0, w, n), :3] + np.append(r.normal(size=(n, 2)) * 0.005, np.zeros((n, 1)), 1)
    a["position"] = aim - d * r.uniform(0.05, 1.0, (n, 1))
    a["normal"] = (0.0, 0.0, 1.0)
    a["incDirection"] = d
    a["antiradiance"] = r.random((n, 3))
    mats = (L.ArcMaterial * 2)()
    mats[1].diffuse = L.f3((0.9, 0.5, 0.25))
    ctx.upload_materials(mats)
    dv, gb = ctx.upload_avpls(a), api.GBuffer(pos, nrm)
    outs = []
    for precision in (L.ARC_PREC_KAHAN_STRICT, L.ARC_PREC_KAHAN):
        out = api.Outputs(w, h)
        api.gather_bruteforce(ctx, dv, gb, (0.0, 0.0, 1.0),
                              api.gather_params(L.ARC_AR_DISK, 40.0, 0.0, radius, precision=precision), out)
        assert ctx.synchronize() == 0
        outs.append(out.antiradiance.cpu().numpy()[..., :3].astype(np.float64))
    want, got = outs
    assert (want > 0).mean() > 0.5
    assert np.all(np.abs(got - want) <= 2.0 ** -22 * want)
