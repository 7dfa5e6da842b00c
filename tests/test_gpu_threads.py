"""Contexts in different threads share no mutable state."""
import threading

import pytest

from antiradiancecuts_b200 import _lib as L
from antiradiancecuts_b200 import api
from test_gpu_culled_gather import _inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [L.ARC_PREC_KAHAN, L.ARC_PREC_KAHAN_STRICT])
def test_contexts_with_different_tile_shapes_share_no_limit(precision):
    """Six threads, each with its own context, run every tile shape (the autotuner, in one call each time):
    no launch may fail because another thread's shape needs less shared memory."""
    pos, nrm, a = _inputs(16, 16, 64, seed=5, flat=True)
    failed, start = [], threading.Barrier(6)

    def work():
        c = api.Context(0)
        c.upload_materials((L.ArcMaterial * 3)())
        dv, gb, out = c.upload_avpls(a), api.GBuffer(pos, nrm), api.Outputs(16, 16)
        prm = api.gather_params(L.ARC_AR_CONE, 40.0, 0.02, precision=precision)
        start.wait()
        try:
            for _ in range(100):
                api.autotune_bruteforce(c, dv, gb, (0.5, 0.5, -1.0), prm, out)
        except L.ArcError as e:
            failed.append(str(e))
        c.synchronize()
        c.close()

    threads = [threading.Thread(target=work) for _ in range(6)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed
