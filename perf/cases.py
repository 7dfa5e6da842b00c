"""What the framework is asked to do in earnest, as cases that can be timed and compared.

A case is one call (or one frame's calls) of the public API over the synthetic scenes of
antiradiancecuts_b200.scene: the exact gather, the cut gathers, the tree build, the learned cut's
network, a batch of views, a progressive frame.  listed() gives the cases, draw() more of the same
ranges; prepare() makes what a program holds before the call, run() is the call, work() what it
cannot do without, exact() its result in 64-bit torch arithmetic where that is affordable.
"""
import ctypes as C
import math

import numpy as np
import torch

from antiradiancecuts_b200 import _lib as L
from antiradiancecuts_b200 import api, learned, scene

ONE_OVER_PI = float(np.float32(0.318309886))
FLOP_PER_PAIR = 43  # radiance and cone antiradiance of one (pixel, AVPL) pair
MLP_FLOP_FORWARD = 2 * (16 * 64 + 64 * 64 + 64 * 64 + 64)

PRESETS = {
    "room": (L.ARC_SCENE_ROOM, 1, 0),
    "boxes2": (L.ARC_SCENE_ROOM_2BOXES, 2, 2),
    "boxes16": (L.ARC_SCENE_ROOM_RANDOM, 3, 16),
    "variant": (L.ARC_SCENE_TRAIN_VARIANT, 500, 0),
}


def listed():
    return [
        # one interactive preview frame: host AVPLs up, plain gather, 256 x 256 (latency counts)
        {"name": "run_room_256_4k", "kind": "run", "scene": "room", "width": 256, "height": 256, "avpls": 4096,
         "light_cuts": False, "ar": "cone", "clustered": False},
        # the reference's default configuration: solid-angle light cut, brute-force disk antiradiance
        {"name": "run_default_512_32k", "kind": "run", "scene": "boxes2", "width": 512, "height": 512, "avpls": 32768,
         "light_cuts": True, "ar": "disk", "clustered": False},
        # the same with clustered deferred antiradiance at 720p
        {"name": "run_clustered_720p_64k", "kind": "run", "scene": "boxes2", "width": 1280, "height": 720,
         "avpls": 65536, "light_cuts": True, "ar": "disk", "clustered": True},
        # a ground-truth frame: the exact gather of the precision configuration, the largest case
        {"name": "gather_1080p_256k", "kind": "gather", "scene": "boxes16", "width": 1920, "height": 1080,
         "avpls": 262144, "bounces": 5, "cone_deg": 60.0, "clamp": 0.005, "precision": "kahan"},
        # the all-FP64 image that errors are measured against, at a ragged size
        {"name": "image_fp64_637x359_16k", "kind": "gather", "scene": "variant", "width": 637, "height": 359,
         "avpls": 16381, "bounces": 3, "cone_deg": 30.0, "clamp": 0.01, "precision": "fp64"},
        # one frame of progressive rendering: AVPLs traced on the GPU, tree, error-bound cut, accumulation
        {"name": "progressive_720p_64k", "kind": "progressive", "scene": "boxes2", "width": 1280, "height": 720,
         "avpls": 65536},
        # a small learned-cut frame, where the launches of the tree levels count
        {"name": "learned_512_16k", "kind": "learned", "scene": "variant", "width": 512, "height": 512,
         "avpls": 16384},
        # the flagship frame: tree, learned cut and evaluation at 1080p with a million AVPLs
        {"name": "learned_1080p_1m", "kind": "learned", "scene": "variant", "width": 1920, "height": 1080,
         "avpls": 1048576},
        # the tree alone over a ragged million of AVPLs
        {"name": "lbvh_1000003", "kind": "lbvh", "scene": "variant", "avpls": 1000003, "normals": False},
        # several views with their own AVPL sets rendered as one batch
        {"name": "batch_8_views", "kind": "batch", "scene": "boxes2", "views": 8},
        # the network over a scene's worth of labelled rows (evaluating a trained model)
        {"name": "forward_1m_rows", "kind": "forward", "rows": 1048573, "act": "relu"},
        # forward and backward over one training batch
        {"name": "gradients_8192_rows", "kind": "gradients", "rows": 8192, "act": "relu"},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["run", "run", "gather", "fp64", "progressive", "learned", "learned", "lbvh", "batch", "forward",
                       "gradients"])
    room = rng.choice(["room", "boxes2", "boxes16", "variant"])
    if kind == "run":
        ar = rng.choice(["cone", "disk"])
        return {"kind": "run", "scene": room, "width": _log(rng, 64, 1280), "height": _log(rng, 64, 720),
                "avpls": _log(rng, 1024, 65536), "light_cuts": ar == "disk", "ar": ar,
                "clustered": ar == "disk" and rng.random() < 0.5}
    if kind in ("gather", "fp64"):
        w, h = _log(rng, 96, 1920), _log(rng, 64, 1080)
        # at most a quarter of the largest listed case in FP32, a small fraction of it in FP64
        most = min(1 << 20, int((1.3e11 if kind == "gather" else 4e9) / (w * h)))
        return {"kind": "gather", "scene": room, "width": w, "height": h, "avpls": _log(rng, 1000, max(2000, most)),
                "bounces": rng.choice([3, 5]), "cone_deg": rng.choice([20.0, 30.0, 60.0]),
                "clamp": rng.choice([0.0, 0.005, 0.01]), "precision": "kahan" if kind == "gather" else "fp64"}
    if kind in ("progressive", "learned"):
        return {"kind": kind, "scene": room, "width": _log(rng, 160, 1920), "height": _log(rng, 120, 1080),
                "avpls": _log(rng, 2000, 400000)}
    if kind == "lbvh":
        return {"kind": "lbvh", "scene": room, "avpls": _log(rng, 1000, 3000000), "normals": rng.random() < 0.3}
    if kind == "batch":
        return {"kind": "batch", "scene": room, "views": rng.randint(2, 10), "view_seed": rng.randint(1, 10000)}
    act = rng.choice(["relu", "gelu"])
    if kind == "forward":
        return {"kind": "forward", "rows": _log(rng, 1000, 4000000), "act": act}
    return {"kind": "gradients", "rows": _log(rng, 256, 500000), "act": act}


# One context per process, with the tree and batch renderer that a program keeps between frames.
_kept = {}


def _ctx():
    if "ctx" not in _kept:
        _kept["ctx"] = api.Context(0)
        _kept["bvh"] = api.AvplBvh(_kept["ctx"])
    torch.cuda.set_stream(_kept["ctx"].stream)
    return _kept["ctx"]


def _model(ctx):
    if "model" not in _kept:
        _kept["model"] = learned.load_default_model(ctx)
    return _kept["model"]


def _desc(case):
    return scene.scene_desc(*PRESETS[case["scene"]])


def _camera(desc):
    p = desc.camera_position
    return (p.x, p.y, p.z)


def _device_avpls(ctx, desc, case, seed, bounces=3):
    return scene.trace_avpls_device(ctx, desc, 1 + seed, case["avpls"], bounces)[0]


class _Memory:
    """Device memory of the library as a CUDA array, so that torch can view it."""

    def __init__(self, ptr, shape, typestr):
        addr = ptr if isinstance(ptr, int) else C.cast(ptr, C.c_void_p).value
        self.__cuda_array_interface__ = {"shape": shape, "typestr": typestr, "data": (addr, False), "version": 3}


def _view(ptr, typestr, *shape):
    return torch.as_tensor(_Memory(ptr, shape, typestr), device="cuda:0")


def prepare(case, seed):
    ctx = _ctx()
    kind = case["kind"]
    s = {"kind": kind, "case": case, "ctx": ctx}
    if kind in ("forward", "gradients"):
        g = torch.Generator(device="cuda").manual_seed(seed)
        act = L.ARC_MLP_ACT_RELU if case["act"] == "relu" else L.ARC_MLP_ACT_GELU
        s["params"] = _model(ctx).params()
        s["model"] = learned.Model(ctx, s["params"], act=act)
        n = case["rows"]
        # the features' ranges: logarithms over 8, ratios, cosines, flags
        x = torch.randn((n, 16), device="cuda", generator=g) * 0.5
        x[:, 3:12] = x[:, 3:12].abs().clamp(max=1.0)
        x[:, 8:10] = (x[:, 8:10] > 0.4).float()
        s["x"] = x.to(torch.bfloat16)
        if kind == "forward":
            s["logits"] = torch.empty(n, device="cuda")
        else:
            s["labels"] = (torch.rand(n, device="cuda", generator=g) < 0.3).float()
            s["weights"] = 1.0 + s["labels"]
            s["weight_sum"] = float(s["weights"].sum().item())
            s["grads"] = np.zeros(learned.NUM_PARAMS, np.float32)
        return s
    desc = _desc(case)
    s["desc"], s["cam"] = desc, _camera(desc)
    mats = scene.materials(desc)[0]
    if kind == "lbvh":
        ctx.upload_materials(mats)
        s["avpls"], s["bvh"] = _device_avpls(ctx, desc, case, seed), _kept["bvh"]
        return s
    if kind == "batch":
        ctx.upload_materials(mats)
        if "batch" not in _kept:
            _kept["batch"] = api.Batch(ctx)
        s["batch"], items = _kept["batch"], []
        for i, v in enumerate(scene.batch_views(desc, case.get("view_seed", 4), case["views"])):
            d = scene.scene_desc(*PRESETS[case["scene"]])
            d.camera_position, d.camera_target = v.camera_position, v.camera_target
            av = scene.trace_avpls_device(ctx, d, v.avpl_seed + 7919 * (1 + seed), v.num_avpls)[0]
            items.append((av, scene.gbuffer_device(ctx, d, v.width, v.height), _camera(d),
                          api.Outputs(v.width, v.height, fp64=False)))
        s["items"] = items
        s["views"] = api.Batch.views([(a.param, gb, cam, out) for a, gb, cam, out in items])
        s["lbvh"] = api.lbvh_params()
        s["prm"] = api.gather_params(L.ARC_AR_CONE, 30.0, 0.01)
        s["cut"] = api.cut_params(L.ARC_CUT_ERROR_BOUND, error_bound=0.01)
        return s
    w, h = case["width"], case["height"]
    s["gb"] = scene.gbuffer_device(ctx, desc, w, h)
    if kind == "run":
        s["avpls"] = scene.trace_avpls(desc, 1 + seed, case["avpls"])[0]
        s["extent"] = scene.scene_extent(desc)
        s["out"] = api.Outputs(w, h, fp64=False)
        s["gather"] = api.CudaGather(ctx, s["gb"], mats, s["out"])
        s["config"] = api.run_config(useLightCuts=int(case["light_cuts"]), cut_kind=L.ARC_CUT_SOLID_ANGLE,
                                     ar_kind=L.ARC_AR_DISK if case["ar"] == "disk" else L.ARC_AR_CONE,
                                     dist_clamp=0.01, useClusteredDeferred=int(case["clustered"]),
                                     cluster_theta=math.radians(0.5 * desc.camera_fov_deg))
        return s
    ctx.upload_materials(mats)
    if kind == "gather":
        fp64 = case["precision"] == "fp64"
        s["avpls"] = _device_avpls(ctx, desc, case, seed, case["bounces"])
        s["out"] = api.Outputs(w, h, fp64=fp64)
        s["prm"] = api.gather_params(L.ARC_AR_CONE, case["cone_deg"], case["clamp"],
                                     precision=L.ARC_PREC_FP64 if fp64 else L.ARC_PREC_KAHAN)
        return s
    s["prm"] = api.gather_params(L.ARC_AR_CONE, 30.0, 0.01)
    s["out"], s["bvh"] = api.Outputs(w, h, fp64=False), _kept["bvh"]
    if kind == "learned":
        s["avpls"] = _device_avpls(ctx, desc, case, seed)
        s["cut"] = learned.cut_params(_model(ctx))
    else:
        s["seed"] = 1 + seed
        s["cut"] = api.cut_params(L.ARC_CUT_ERROR_BOUND, error_bound=0.01)
        s["sum"], s["shown"] = api.Accumulator(ctx, w, h), api.Outputs(w, h, fp64=False)
    return s


def _planes(out):
    return [out.result, out.radiance, out.antiradiance]


def run(s):
    kind, ctx = s["kind"], s["ctx"]
    if kind == "run":
        return _planes(s["gather"].run(s["avpls"], s["cam"], s["extent"], s["config"]))
    if kind == "gather":
        api.gather_bruteforce(ctx, s["avpls"].param, s["gb"], s["cam"], s["prm"], s["out"])
        out = _planes(s["out"])
        return out if s["out"].result64 is None else out + [s["out"].result64]
    if kind == "learned":
        s["bvh"].build(s["avpls"].param)
        api.gather_cut(ctx, s["bvh"], None, s["gb"], s["cam"], s["prm"], s["cut"], s["out"])
        return _planes(s["out"])
    if kind == "progressive":
        avpls, paths = scene.trace_avpls_device(ctx, s["desc"], s["seed"], s["case"]["avpls"])
        s["bvh"].build(avpls.param)
        api.gather_cut(ctx, s["bvh"], None, s["gb"], s["cam"], s["prm"], s["cut"], s["out"])
        s["sum"].add(s["out"], paths)
        return [_planes(s["sum"].normalize(s["shown"])), paths]
    if kind == "batch":
        s["batch"].render(s["views"], s["lbvh"], s["prm"], s["cut"])
        return [_planes(out) for _, _, _, out in s["items"]]
    if kind == "forward":
        s["model"].forward(s["x"], s["logits"])
        return s["logits"]
    if kind == "gradients":
        loss = C.c_float(0.0)
        L.check(ctx.lib.arc_mlp_gradients(s["model"].handle, C.c_void_p(s["x"].data_ptr()),
                                          C.c_void_p(s["labels"].data_ptr()), C.c_void_p(s["weights"].data_ptr()),
                                          s["x"].shape[0], s["weight_sum"],
                                          s["grads"].ctypes.data_as(C.POINTER(C.c_float)), C.byref(loss)),
                "arc_mlp_gradients")
        return [s["grads"], np.float32(loss.value)]
    s["bvh"].build(s["avpls"].param, consider_normals=s["case"]["normals"])
    v = s["bvh"].view()
    n, nd = v.num_leaves, v.node_data
    t = 2 * n - 1
    bounds = _view(v.bounds, "<f4", n - 1, 16)  # columns 3 and 7 hold the children (left, right below)
    return {"morton": _view(v.morton, "<i4", n), "sorted_index": _view(v.sorted_index, "<i4", n),
            "left": _view(v.left, "<i4", n - 1), "right": _view(v.right, "<i4", n - 1),
            "parents": _view(v.parents, "<i4", t), "range": _view(v.range, "<i4", n - 1, 2),
            "box_min": bounds[:, 0:3], "box_max": bounds[:, 4:7], "cones": bounds[:, 8:16],
            "records": _view(v.records, "<f4", t, 16), "dirstat": _view(v.dirstat, "<f4", t, 4),
            "size": _view(nd.size, "<i4", t), "material": _view(nd.materialIndex, "<i4", t),
            "random": _view(nd.randomNumbers, "<f4", t), "position": _view(nd.position, "<f4", t, 3),
            "normal": _view(nd.normal, "<f4", t, 3), "radiance": _view(nd.incRadiance, "<f4", t, 3),
            "direction": _view(nd.incDirection, "<f4", t, 3)}


def work(case):
    kind = case["kind"]
    if kind == "forward":
        return {"bytes": 36 * case["rows"], "flops": MLP_FLOP_FORWARD * case["rows"]}
    if kind == "gradients":
        return {"bytes": 40 * case["rows"] + 4 * learned.NUM_PARAMS, "flops": 3 * MLP_FLOP_FORWARD * case["rows"]}
    if kind == "lbvh":  # inputs read, every array of the tree written
        return {"bytes": (68 + 8 + 2 * (64 + 16 + 60 + 4) + 64 + 8 + 8) * case["avpls"], "flops": 0}
    if kind == "batch":
        views = scene.batch_views(_desc(case), case.get("view_seed", 4), case["views"])
        parts = [_frame(v.width, v.height, v.num_avpls, 1.0) for v in views]
        return {"bytes": sum(p["bytes"] for p in parts), "flops": sum(p["flops"] for p in parts)}
    # the rooms fill a square field of view of the preset camera; beside it lies background
    surface = min(1.0, 0.964 * case["height"] / case["width"])
    if kind == "gather" or (kind == "run" and not case["light_cuts"]):
        px = case["width"] * case["height"]
        return {"bytes": 68 * case["avpls"] + 80 * px, "flops": FLOP_PER_PAIR * surface * px * case["avpls"]}
    return _frame(case["width"], case["height"], case["avpls"], surface)


def _frame(width, height, avpls, surface):
    """A cut frame: the tree, and a cut of about 20 sqrt(N) nodes (20,000 at a million AVPLs)."""
    px = width * height
    return {"bytes": 68 * avpls + 400 * avpls + 80 * px,
            "flops": FLOP_PER_PAIR * surface * px * min(avpls, 20 * math.sqrt(avpls))}


def exact(case, seed):
    kind = case["kind"]
    if kind in ("forward", "gradients"):
        return _exact_mlp(case, seed)
    if kind not in ("gather", "run") or case["width"] * case["height"] * case["avpls"] > 3e10:
        return None
    s = prepare(case, seed)
    if kind == "gather":
        a, cone, clamp = s["avpls"].to_host(), case["cone_deg"], case["clamp"]
    else:
        a, cone, clamp = s["avpls"], 30.0, 0.01
    radius = s["extent"] * s["config"].photonRadiusScale / 100.0 if kind == "run" else 0.0
    rad, ar = _exact_gather(s, a, case.get("ar", "cone"), math.radians(cone), clamp, radius)
    one = torch.ones_like(rad[..., :1])
    full = [torch.cat([v, one], -1) for v in (rad - ar, rad, ar)]
    if kind == "run" and case["light_cuts"]:  # the light cut is an approximation of its own
        return [None, None, full[2]]
    return full + ([rad - ar] if case.get("precision") == "fp64" else [])


def _exact_gather(s, avpls, ar_kind, half_angle, clamp, radius):
    """Radiance and antiradiance [H, W, 3] over every AVPL in FP64 (Lambertian surfaces)."""
    dev = "cuda:0"
    f64 = lambda v: torch.as_tensor(np.ascontiguousarray(v), device=dev).double()  # noqa: E731
    diffuse = f64(scene.materials(s["desc"])[1]) * ONE_OVER_PI
    p, n, w = f64(avpls["position"]), f64(avpls["normal"]), f64(avpls["incDirection"])
    n = n / n.norm(dim=1, keepdim=True)
    light = (w == 0).all(1)
    mat = torch.as_tensor(np.ascontiguousarray(avpls["materialIndex"]), device=dev).long()
    rho = torch.where(light[:, None], torch.ones_like(p), diffuse[mat])
    ld, ad = f64(avpls["incRadiance"]) * rho, f64(avpls["antiradiance"])
    wl = w.norm(dim=1)
    wu = torch.where(light[:, None], torch.zeros_like(w), w / wl.clamp(min=1e-30)[:, None])
    h, wd = s["gb"].pos.shape[:2]
    gp, gn = s["gb"].pos.reshape(-1, 4).double(), s["gb"].nrm.reshape(-1, 4).double()
    live = torch.nonzero(gn[:, 3] > 0).reshape(-1)
    rad = torch.zeros((h * wd, 3), dtype=torch.float64, device=dev)
    ar = torch.zeros_like(rad)
    cos_thr, step = max(math.cos(half_angle), 0.001), max(1, (1 << 25) // len(p))
    for i in range(0, len(live), step):
        px = live[i:i + step]
        q, m = gp[px, :3], gn[px, :3]
        m = m / m.norm(dim=1, keepdim=True)
        l2 = torch.zeros((len(px), len(p)), dtype=torch.float64, device=dev)
        nd, nad, wdot = torch.zeros_like(l2), torch.zeros_like(l2), torch.zeros_like(l2)
        for k in range(3):
            d = p[None, :, k] - q[:, k, None]
            l2 += d * d
            nd += m[:, k, None] * d
            nad += n[None, :, k] * d
            wdot += w[None, :, k] * d
        l2.clamp_(min=1e-30)
        r = l2.rsqrt()
        inv = 1.0 / l2.clamp(min=clamp * clamp) if clamp > 0 else 1.0 / l2
        g = (nd * r).clamp(min=0) * (-nad * r).clamp(min=0) * inv
        rad[px] = diffuse[gn[px, 3].long()] * (g @ ld)
        if ar_kind == "cone":
            ga = torch.where((-wdot * r > cos_thr) & (nd * r > 0.001), nd * r * inv, torch.zeros_like(l2))
        else:
            wn = m @ w.T
            t = -nd / wn
            h2 = torch.zeros_like(l2)
            for k in range(3):
                h2 += (p[None, :, k] - q[:, k, None] + t * wu[None, :, k]) ** 2
            hit = (wn < 0) & (t > 0) & (h2 < radius * radius) & (nad > 0)
            ga = hit.double() / (math.pi * radius * radius)
        ar[px] = diffuse[gn[px, 3].long()] * (ga @ ad)
    return rad.reshape(h, wd, 3), ar.reshape(h, wd, 3)


def _exact_mlp(case, seed):
    s = prepare(case, seed)
    flat = torch.tensor(s["params"], dtype=torch.float64, device="cuda:0", requires_grad=True)
    sizes, at, layers = [(16, 64), (64, 64), (64, 64), (64, 1)], 0, []
    for i, o in sizes:
        layers.append((flat[at:at + i * o].reshape(o, i), flat[at + i * o:at + i * o + o]))
        at += i * o + o
    act = torch.relu if case["act"] == "relu" else lambda z: z * torch.sigmoid(1.702 * z)
    parts, loss, rows = [], 0.0, s["x"].shape[0]
    for i in range(0, rows, 1 << 18):
        h = s["x"][i:i + (1 << 18)].double()
        for wt, b in layers[:-1]:
            h = act(h @ wt.T + b)
        y = (h @ layers[-1][0].T + layers[-1][1]).reshape(-1)
        parts.append(y.detach())
        if case["kind"] == "gradients":
            lab, wgt = s["labels"][i:i + (1 << 18)].double(), s["weights"][i:i + (1 << 18)].double()
            bce = torch.nn.functional.binary_cross_entropy_with_logits(y, lab, reduction="none")
            part = (wgt * bce).sum() / s["weight_sum"]
            part.backward(retain_graph=True)
            loss += float(part.item())
    if case["kind"] == "forward":
        return torch.cat(parts)
    return [flat.grad.detach(), np.float64(loss)]
