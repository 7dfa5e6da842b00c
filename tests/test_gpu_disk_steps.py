"""The culled disk antiradiance in segments of several steps of AVPLs, in both tile sizes."""
import numpy as np
import pytest

from antiradiancecuts_b200 import _lib as L
from antiradiancecuts_b200 import api
from test_gpu_culled_gather import _inputs

pytestmark = pytest.mark.gpu


# steps of 512 AVPLs; 16 x 16 tiles: 16 steps in 4 segments, 47 in 9; 32 x 32: 12 steps in 4 segments, 40 in 4
@pytest.mark.parametrize("size", [(512, 512, 8192), (333, 300, 24000), (1024, 1024, 6000), (1023, 1000, 20480)])
def test_culled_disk_antiradiance_over_several_steps(ctx, size):
    """Segments of several steps: lists that collect survivors over steps (small radius) and lists that
    fill with every step (large radius), against the gather that evaluates every pair.  Both add the
    same terms; per-term compensation leaves each sum within 2^-22 of exact."""
    for flat, radius in ((True, 0.01), (False, 0.5)):
        pos, nrm, a = _inputs(*size, seed=sum(size) + flat, flat=flat)
        # neighbouring pixels near each other, as in an image
        gy, gx = np.mgrid[0:size[1], 0:size[0]]
        pos[..., 0] = gx / size[0]
        pos[..., 1] = gy / size[1]
        if flat:
            pos[..., 2] = 0.0
            nrm[..., :3] = (0.0, 0.0, 1.0)
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
            outs.append(out.antiradiance.cpu().numpy()[..., :3].astype(np.float64))
        want, got = outs
        assert (want > 0).any()
        assert np.all(np.abs(got - want) <= 2.0 ** -22 * want)
