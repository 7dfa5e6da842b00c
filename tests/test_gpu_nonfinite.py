"""Values that are not finite: they show wherever the same arithmetic without culling shows them."""
import numpy as np
import pytest

from antiradiancecuts_b200 import _lib as L
from test_gpu_culled_gather import _gather, _inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [L.ARC_PREC_KAHAN, L.ARC_PREC_FP64])
@pytest.mark.parametrize("field,index,value", [("incRadiance", 17, np.inf), ("antiradiance", 400, np.nan),
                                               ("antiradiance", 401, np.inf)])
def test_one_record_without_a_finite_value_shows_everywhere(ctx, precision, field, index, value):
    """0 times such a value is not 0, also outside the record's cone."""
    pos, nrm, a = _inputs(40, 40, 600, seed=3, flat=True)
    a[field][index] = value
    want = _gather(ctx, pos, nrm, a, L.ARC_AR_CONE, L.ARC_PREC_NAIVE, 0.02)
    got = _gather(ctx, pos, nrm, a, L.ARC_AR_CONE, precision, 0.02)
    assert not np.isfinite(want[2]).all()
    for g, v in zip(got, want):
        assert np.array_equal(np.isfinite(g), np.isfinite(v))
