"""The exact gather of frames in which few pixels of a tile have a surface."""
import numpy as np
import pytest

from antiradiancecuts_b200 import _lib as L
from antiradiancecuts_b200 import api
from test_gpu_culled_gather import TOL, _inputs

pytestmark = pytest.mark.gpu


def _gather(ctx, pos, nrm, a, ar, precision, shape=-1):
    mats = (L.ArcMaterial * 3)()
    for i in range(3):
        mats[i].diffuse = L.f3((0.9, 0.5 / (i + 1), 0.25))
    ctx.upload_materials(mats)
    dv = ctx.upload_avpls(a)
    h, w = pos.shape[:2]
    out = api.Outputs(w, h)
    for plane in (out.radiance, out.antiradiance, out.result, out.result64):
        plane.fill_(7.0)  # every pixel has to be written
    api.gather_bruteforce(ctx, dv, api.GBuffer(pos, nrm), (0.5, 0.5, -1.0),
                          api.gather_params(ar, 40.0, 0.02, precision=precision, tile_config=shape), out)
    assert ctx.synchronize() == 0
    return [t.cpu().numpy()[..., :3].astype(np.float64) for t in (out.radiance, out.antiradiance, out.result64)]


@pytest.mark.parametrize("ar", [L.ARC_AR_NONE, L.ARC_AR_CONE])
@pytest.mark.parametrize("coverage", [0.003, 0.05, 0.15, 0.3, 0.6])
def test_sparse_surfaces_gather_as_dense_ones(ctx, coverage, ar):
    """Scattered surface pixels (one row of tiles full, one column of tiles empty) give the sums that the
    same pixels give side by side; several segments, tile shapes of 1, 2 and 4 pixels per thread."""
    w, h, n = 133, 101, 1537
    pos, nrm, a = _inputs(w, h, n, seed=int(1000 * coverage), flat=True)
    r = np.random.default_rng(9)
    keep = r.random((h, w)) < coverage
    keep[32:64] = True
    keep[:, 48:64] = False
    nrm[..., 3] = np.where(keep, np.maximum(nrm[..., 3], 1.0), 0.0)
    ys, xs = np.nonzero(keep)
    pad = -len(ys) % 64
    dense = [np.concatenate([v[ys, xs], v[ys[:1], xs[:1]].repeat(pad, 0)]).reshape(-1, 64, 4) for v in (pos, nrm)]
    for precision, shape in ((L.ARC_PREC_KAHAN, 0), (L.ARC_PREC_KAHAN, 6), (L.ARC_PREC_KAHAN, -1), (L.ARC_PREC_KAHAN, 3),
                             (L.ARC_PREC_FP64, -1)):
        tol = TOL[precision](n)
        want = [v.reshape(-1, 3)[: len(ys)] for v in _gather(ctx, *dense, a, ar, precision)]
        got = _gather(ctx, pos, nrm, a, ar, precision, shape)
        assert all((v[~keep] == 0).all() for v in got)
        got = [v[ys, xs] for v in got]
        assert (want[0] > 0).any()
        assert np.all(np.abs(got[0] - want[0]) <= (tol + 2.0 ** -23) * want[0])
        assert np.all(np.abs(got[1] - want[1]) <= (tol + 2.0 ** -23) * want[1])
        assert np.all(np.abs(got[2] - want[2]) <= tol * (1 + 1e-6) * (want[0] + want[1]))
