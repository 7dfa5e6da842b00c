"""Kernels that split their work by size, at the sizes where the split changes: tree blocks and sort
passes, the learned cut's list groups, rows of the network's training kernel, and ragged frames of the
solid-angle cut."""
import ctypes as C
import math

import numpy as np
import pytest

import helpers as H
from antiradiancecuts_b200 import _lib as L
from antiradiancecuts_b200 import api, learned
from oracle import mlp_oracle as M
from oracle import oracle as O
from test_gpu_lbvh import _build, _compare

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [127, 128, 129, 257, 16385, 65537, 524288, 524289])
def test_lbvh_at_block_and_sort_edges(ctx, n):
    """128 leaves per block; 4, 8 or 16 keys per thread of a sort pass.  Bit for bit, also when all
    Morton codes are equal (every block is a chain of index bits)."""
    d = H.workload("variant500_1080p_1m", 8, 8, n)
    a = d["avpls"].copy()
    for same in (False, True) if n < 65536 else (False,):
        if same:
            a["position"] = a["position"][0]
        bvh, _ = _build(ctx, a, d["mats"])
        _compare(bvh.host_arrays(), O.build_tree(a, d["dif"]), n)


# tiles: 1; 8,192 and 8,193 (one and two groups); 33,669 (four groups, more tiles in each)
@pytest.mark.parametrize("w,h", [(5, 3), (1024, 512), (21848, 24), (2088, 1025)])
def test_learned_lists_at_group_edges(ctx, w, h):
    """Threshold 1 never refines below the band, so the lists are those of the error-bound cut at
    band * eps, tile by tile."""
    d = H.workload("boxes2_720p_64k", w, h, 700)
    ctx.upload_materials(d["mats"])
    bvh = api.AvplBvh(ctx)
    bvh.build(ctx.upload_avpls(d["avpls"]))
    gb = api.GBuffer(d["pos"], d["nrm"])
    model = learned.Model(ctx, seed=5, loss=L.ARC_MLP_LOSS_BCE)
    eps, band = float(np.float32(0.05)), 4.0
    cuts = []
    for cut in (api.cut_params(L.ARC_CUT_ERROR_BOUND, error_bound=eps * band),
                api.cut_params(L.ARC_CUT_LEARNED, error_bound=eps, mlp_band=band, model=model.handle.value,
                               mlp_threshold=1.0)):
        api.gather_cut(ctx, bvh, None, gb, d["cam"], api.gather_params(L.ARC_AR_CONE, 30.0, 0.01), cut,
                       api.Outputs(w, h))
        assert ctx.synchronize() == 0
        cuts.append(api.last_cut(ctx))
    assert len(cuts[0]) == (w + 7) // 8 * ((h + 7) // 8)
    assert all(np.array_equal(a, b) for a, b in zip(*cuts))
    assert sum(len(c) for c in cuts[0]) > 0
    model.close()


# the last: 1,185 tiles of 128 rows, from which a multiprocessor takes two blocks where it has 148
@pytest.mark.parametrize("act", [L.ARC_MLP_ACT_GELU, L.ARC_MLP_ACT_RELU])
@pytest.mark.parametrize("rows", [1, 127, 129, 18945, 151553])
def test_gradients_of_equal_rows_add_up(ctx, rows, act):
    """R equal rows give R times one row's gradients and loss.  Every parameter sums equal FP32 terms:
    at most 1,024 rows of a block after one another (16 at a time) and 296 blocks, each addition within
    2^-23 of the sum; 2,048 additions bound both sides."""
    import torch

    h = C.c_void_p()
    L.check(ctx.lib.arc_mlp_create(ctx.handle, 7, C.byref(h)), "create")
    L.check(ctx.lib.arc_mlp_set_activation(h, act), "set_activation")
    row = torch.randn(1, 16, device="cuda", generator=torch.Generator(device="cuda").manual_seed(3))
    got = []
    for r in (128, rows):
        x = row.to(torch.bfloat16).expand(r, 16).contiguous()
        lab, wts = torch.ones(r, device="cuda"), torch.ones(r, device="cuda")
        g, loss = np.zeros(M.NUM_PARAMS, np.float32), C.c_float()
        L.check(ctx.lib.arc_mlp_gradients(h, C.c_void_p(x.data_ptr()), C.c_void_p(lab.data_ptr()),
                                          C.c_void_p(wts.data_ptr()), r, 1.0,
                                          g.ctypes.data_as(C.POINTER(C.c_float)), C.byref(loss)), "gradients")
        got.append(np.append(g.astype(np.float64), loss.value) / r)
    ctx.lib.arc_mlp_destroy(h)
    assert np.abs(got[0]).max() > 0
    assert np.all(np.abs(got[1] - got[0]) <= 2048 * 2.0 ** -23 * np.abs(got[0]))


@pytest.mark.parametrize("specular", [False, True])
@pytest.mark.parametrize("w,h", [(1, 1), (9, 7), (33, 17), (64, 40)])
def test_solid_angle_cut_at_ragged_sizes(ctx, w, h, specular):
    """Both forms of the walk (an exponent of 8 makes up to 8 roundings of its base's error: within the
    1e-5 of the cut's other comparisons)."""
    d = H.workload("boxes2_720p_64k", w, h, 4096)
    mats, spe, ex = d["mats"], d["spe"].copy(), d["ex"].copy()
    if specular:
        spe[:], ex[:] = 0.25, 8.0
        for m in mats:
            m.specular, m.exponent = L.f3((0.25, 0.25, 0.25)), 8.0
    bvh, dv = _build(ctx, d["avpls"], mats)
    out = api.Outputs(w, h)
    api.gather_cut(ctx, bvh, dv, api.GBuffer(d["pos"], d["nrm"]), d["cam"],
                   api.gather_params(L.ARC_AR_NONE, dist_clamp=0.01),
                   api.cut_params(L.ARC_CUT_SOLID_ANGLE, solid_angle_threshold=math.pi / 10), out)
    assert ctx.synchronize() == 0
    want, err = O.cut_solid_angle(d["pos"], d["nrm"], np.arange(w * h), bvh.host_arrays(), d["dif"], spe, ex, d["cam"],
                                  math.pi / 10, 0.01)
    assert err.sum() == 0 and np.abs(want).max() > 0
    assert H.rel_rmse(out.radiance.cpu().numpy()[..., :3], want) < 1e-5
