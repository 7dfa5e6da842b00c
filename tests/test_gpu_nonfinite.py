"""Values that are not finite: they show wherever the same arithmetic without culling shows them."""
import numpy as np
import pytest

import helpers as H
from antiradiancecuts_b200 import _lib as L
from oracle import oracle as O
from test_gpu_culled_gather import _gather, _inputs
from test_gpu_lbvh import FLOAT_KEYS, INT_KEYS, _build

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


def test_lbvh_with_radiance_that_is_not_a_number(ctx):
    """A representative's random number is compared with i1 / (i1 + i2), which is not a number when the
    sibling's radiance is none: the left child stays, also when its own radiance is 0."""
    d = H.workload("room_256_4k", 8, 8, 4096)
    a = d["avpls"].copy()
    r = np.random.default_rng(2)
    a["incRadiance"][r.random(len(a)) < 0.5] = 0.0
    a["incRadiance"][r.integers(0, len(a), 40)] = np.nan
    a["antiradiance"][r.integers(0, len(a), 40)] = np.nan
    bvh, _ = _build(ctx, a, d["mats"])
    gpu, ref = bvh.host_arrays(), O.build_tree(a, d["dif"])
    for k in INT_KEYS + FLOAT_KEYS:
        assert np.array_equal(gpu[k], ref[k], equal_nan=gpu[k].dtype.kind == "f"), k
