"""What users of this package have it do, as cases that can be timed.

A case is a plain dict.  `listed()` gives the fixed ones, `draw(rng)` one more of the same ranges,
`prepare(case, seed)` what a user's program holds before the call, `run(state)` one pass through the public
entry points, `work(case)` the bytes and operations a pass cannot do without, `tolerance(case)` how far two
correct implementations may differ.

Five kinds of case:
  op3d       the one-stage operator (MultiScale3DDeformableAttnFunction*): forward, or forward + backward
  two_stage  the same operator through the two Functions of the two-stage API, forward + backward
  msda       plain 2-D multi-scale deformable attention (temporal self-attention, detection decoder)
  dist       depth distribution from the depth network's logits
  encoder    the modules of modules.py on the frames of a six-camera rig: the spatial cross-attention stack,
             or the full encoder layer with its temporal self-attention
"""
import math
import os
import sys

import torch

sys.path.insert(0, os.path.join(os.getcwd(), "3d-deformable-attention_b200"))

import dfa3d_b200 as M  # noqa: E402
from dfa3d_b200 import modules  # noqa: E402
from dfa3d_b200.dist_producer import depth_distribution  # noqa: E402

BASE = "116x200 58x100 29x50 15x25"      # 928 x 1600 images at strides 8 / 16 / 32 / 64
SMALL = "23x40"                          # 736 x 1280 images at stride 32


def _op(kind, **kw):
    c = dict(kind=kind, B=1, levels=BASE, D=64, Q=1000, P=8, H=8, C=32, dtype="fp32", train=True, local=False)
    c.update(kw)
    return c


def _enc(**kw):
    c = dict(kind="encoder", module="stack", layers=6, bev_h=200, bev_w=200, levels=BASE, D=118, P=8, Z=4, E=256,
             H=8, ffn=512, train=False)
    c.update(kw)
    return c


def listed():
    return [
        # 900 object queries of the detection decoder look into one 200 x 200 BEV map: the smallest call that a
        # served frame makes, once per decoder layer; launches and host work are all there is to it
        _op("msda", name="decoder_infer", levels="200x200", Q=900, P=4, train=False, local=True),
        # a small problem stepped forward and backward (unit-test and debugging sized): latency again
        _op("op3d", name="op_small_train", levels="32x32 16x16", D=16, Q=512, P=4),
        # one feature level, 6 cameras: the operator as the small detector configuration trains it
        _op("op3d", name="op_single_level_train", B=6, levels=SMALL, Q=6000),
        # the base detector configuration and the default workload of bench.py: 15.4 M sampled points
        _op("op3d", name="op_base_train", B=6, Q=10000),
        # the same shapes served with bf16 features and depth distributions
        _op("op3d", name="op_base_bf16_infer", B=6, Q=10000, dtype="bf16", train=False, local=True),
        # mixed-precision training at sizes that divide nothing: odd levels, 3 x 5 points, half storage
        _op("op3d", name="op_half_odd_train", B=3, levels="57x101 29x51 15x25", D=59, Q=3777, P=5, C=16,
            dtype="fp16", local=True),
        # depth scores and attention as two Functions with the (B,Q,H,L,P,4) tensor between them
        _op("two_stage", name="two_stage_train", B=2, levels="58x100 29x50", D=80, Q=5000, P=4, local=True),
        # temporal self-attention of a 200 x 200 BEV over the previous and the current map: 4 points per item
        _op("msda", name="bev_self_attention_train", B=2, levels="200x200", Q=40000, P=4, local=True),
        # depth network's logits of 6 cameras to the operator's distribution at all four levels, and back
        dict(kind="dist", name="depth_dist_train", B=6, levels=BASE, D=64, map_h=58, map_w=100, dtype="fp32",
             activation="softmax"),
        # the cross-attention stack on one frame at the base configuration, served
        _enc(name="encoder_stack_infer"),
        # one spatial cross-attention layer (attention, norm, feed-forward, norm) of the base configuration, trained
        _enc(name="cross_attention_layer_train", layers=1, train=True),
        # the full encoder layer (temporal self-attention first) of the small configuration, trained
        _enc(name="encoder_layer_small_train", module="layer", layers=1, bev_h=150, bev_w=150, levels=SMALL,
             D=64, train=True),
    ]


# ------------------------------------------------------------------------------------------------
def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_levels(rng, n, h_lo=12, h_hi=116):
    h = _log_int(rng, h_lo, h_hi)
    w = int(round(h * rng.uniform(1.5, 1.9)))
    out = []
    for _ in range(n):
        out.append("%dx%d" % (max(2, h), max(2, w)))
        h, w = (h + 1) // 2, (w + 1) // 2
    return " ".join(out)


def draw(rng):
    kind = rng.choice(("op3d", "op3d", "op3d", "two_stage", "msda", "msda", "dist", "encoder"))
    if kind == "dist":
        n = rng.randint(1, 4)
        levels = _draw_levels(rng, n, 16)
        h, w = (int(x) for x in levels.split()[rng.randrange(n)].split("x"))
        return dict(kind="dist", B=rng.randint(1, 6), levels=levels, D=rng.randint(32, 118), map_h=h, map_w=w,
                    dtype=rng.choice(("fp32", "fp32", "bf16")), activation=rng.choice(("softmax", "softmax", "sigmoid")))
    if kind == "encoder":
        layer = rng.random() < 0.5
        side = _log_int(rng, 40, 160)
        P = rng.choice((4, 8))
        return _enc(module="layer" if layer else "stack", layers=1 if layer else rng.randint(1, 3), bev_h=side,
                    bev_w=max(40, side + rng.randint(-10, 10)), levels=_draw_levels(rng, rng.choice((1, 1, 2, 4)), 23),
                    D=rng.randint(48, 118), P=P, Z=4, train=rng.random() < 0.5)
    train = rng.random() < 0.65
    if kind == "msda":
        if rng.random() < 0.5:                       # decoder: few queries; one BEV map or several image levels
            return _op("msda", B=rng.randint(1, 4), levels=rng.choice(("200x200", "150x150", _draw_levels(rng, 4))),
                       Q=_log_int(rng, 100, 1500), P=4, train=train, local=rng.random() < 0.7)
        side = _log_int(rng, 40, 200)                # BEV self-attention: one query per cell
        return _op("msda", B=2 * rng.randint(1, 2), levels="%dx%d" % (side, side), Q=side * side,
                   P=rng.choice((4, 4, 8)), train=train, local=True)
    L = rng.randint(1, 4)
    c = _op(kind, B=rng.randint(1, 6), levels=_draw_levels(rng, L), D=rng.randint(16, 118), Q=_log_int(rng, 200, 10000),
            P=rng.choice((2, 4, 4, 5, 8, 8)), H=rng.choice((4, 8, 8)), C=rng.choice((16, 32, 32, 64)),
            train=train or kind == "two_stage", local=rng.random() < 0.5)
    if kind == "op3d":
        c["dtype"] = rng.choice(("fp32", "fp32", "bf16", "fp16"))
    while c["B"] * c["Q"] * c["H"] * L * c["P"] * max(c["C"], 32) > 6 * 10000 * 8 * 32 * 32:
        c["Q"] = c["Q"] // 2 + 1
    return c


# ------------------------------------------------------------------------------------------------
_DTYPE = {"fp32": torch.float32, "bf16": torch.bfloat16, "fp16": torch.float16}


def _levels(case):
    return [tuple(int(x) for x in l.split("x")) for l in case["levels"].split()]


def _level_tensors(levels, D=None):
    shapes = torch.tensor([[h, w] + ([D] if D else []) for h, w in levels], dtype=torch.int64)
    hw = shapes[:, 0] * shapes[:, 1]
    return shapes.cuda(), torch.cat([hw.new_zeros(1), hw.cumsum(0)[:-1]]).cuda()


def _locations(case, levels, g, dims):
    """Uniform over a frame a little larger than the image (one point in seven falls outside), or -- local --
    around one reference point per query with offsets of a few pixels and bins, neighbouring queries beside each
    other, as the attention modules produce them."""
    B, Q, H, L, P = case["B"], case["Q"], case["H"], len(levels), case["P"]
    r = torch.rand(B, Q, H, L, P, dims, generator=g, device="cuda")
    if not case["local"]:
        r[..., :2] = r[..., :2] * 1.0846 - 0.0423
        return r
    side = max(1, int(round(Q ** 0.5)))
    q = torch.arange(Q, device="cuda")
    rows = -(-Q // side)
    ref = torch.stack([((q % side).float() + 0.5) / side, ((q // side).float() + 0.5) / rows], -1)
    ref = ref + 0.02 * torch.randn(B, Q, 2, generator=g, device="cuda")
    if dims == 3:
        ref = torch.cat([ref, 0.05 + 0.8 * torch.rand(B, Q, 1, generator=g, device="cuda")], -1)
    size = torch.tensor([[w, h, case["D"]] for h, w in levels], dtype=torch.float32, device="cuda")[:, :dims]
    off = (r - 0.5) * torch.tensor([12.0, 12.0, 4.0], device="cuda")[:dims] / size[:, None, :]
    return (ref[:, :, None, None, None, :] + off).contiguous()


def _prepare_op(case, g):
    levels = _levels(case)
    B, Q, H, C, D, L, P = case["B"], case["Q"], case["H"], case["C"], case["D"], len(levels), case["P"]
    N = sum(h * w for h, w in levels)
    dt = _DTYPE[case["dtype"]]
    s = dict(case=case)
    s["value"] = torch.randn(B, N, H, C, generator=g, device="cuda").to(dt)
    s["attn"] = torch.randn(B, Q, H, L * P, generator=g, device="cuda").softmax(-1).view(B, Q, H, L, P)
    s["grad_out"] = torch.randn(B, Q, H * C, generator=g, device="cuda")
    s["shapes2"], s["lsi"] = _level_tensors(levels)
    if case["kind"] == "msda":
        s["loc"] = _locations(case, levels, g, 2)
    else:
        s["shapes3"], _ = _level_tensors(levels, D)
        s["loc"] = _locations(case, levels, g, 3)
        dist = torch.randn(B, N, D, generator=g, device="cuda").softmax(-1)
        if case["kind"] == "two_stage":              # that API takes the distribution repeated over the heads
            dist = dist[:, :, None].repeat(1, 1, H, 1)
        s["dist"] = dist.to(dt)
    if case["train"]:
        if case["dtype"] == "fp16":
            s["grad_out"] = s["grad_out"].half()
        s["leaves"] = [s[k].requires_grad_(True) for k in ("value", "dist", "loc", "attn") if k in s]
    return s


def _rig(case, g):
    """A ring of six cameras around the vehicle: their projection matrices at a padded 928 x 1600 image, each yaw
    a little off, as calibration files give them."""
    cams, h, w = 6, 928.0, 1600.0
    jitter = (torch.rand(cams, generator=g, device="cuda") * 0.1 - 0.05).tolist()
    mats = []
    for c in range(cams):
        yaw = 2 * math.pi * c / cams + jitter[c]
        fwd = torch.tensor([math.cos(yaw), math.sin(yaw), 0.0])
        right = torch.tensor([math.sin(yaw), -math.cos(yaw), 0.0])
        down = torch.tensor([0.0, 0.0, -1.0])
        rot = torch.stack([right, down, fwd])
        pos = 0.8 * fwd + torch.tensor([0.0, 0.0, -0.3])
        ext = torch.eye(4)
        ext[:3, :3] = rot
        ext[:3, 3] = -rot @ pos
        k = torch.eye(4)
        k[0, 0] = k[1, 1] = 1260.0
        k[0, 2], k[1, 2] = w / 2, h / 2
        mats.append(k @ ext)
    return torch.stack(mats)[None].cuda(), (h, w)


def _prepare_encoder(case, g):
    # projection products on the tf32 tensor cores, as bench.py runs the encoder stack
    torch.backends.cuda.matmul.allow_tf32 = True
    levels = _levels(case)
    N, E, Q = sum(h * w for h, w in levels), case["E"], case["bev_h"] * case["bev_w"]
    kw = dict(embed_dims=E, ffn_dims=case["ffn"], num_cams=6, num_heads=case["H"], num_levels=len(levels),
              num_points=case["P"], dropout=0.0)
    if case["module"] == "layer":
        net = modules.BEVFormerEncoderLayer(bev_h=case["bev_h"], bev_w=case["bev_w"], **kw)
    else:
        net = modules.SCAEncoderStack(num_layers=case["layers"], **kw)
    net = net.cuda()
    with torch.no_grad():                            # trained-like weights: offsets and attention depend on the query
        for n, p in net.named_parameters():
            if n.endswith("weight") and p.dim() == 2 and any(k in n for k in ("sampling_offsets", "attention_weights")):
                p.copy_(0.02 * torch.randn(p.shape, generator=g, device="cuda"))
            elif p.dim() == 2:
                p.copy_(torch.randn(p.shape, generator=g, device="cuda") / math.sqrt(p.shape[1]))
            elif "ffn" in n:
                p.copy_(0.02 * torch.randn(p.shape, generator=g, device="cuda"))
    lidar2img, img = _rig(case, g)
    ref3d = modules.bev_reference_points(case["bev_h"], case["bev_w"], num_points_in_pillar=case["Z"])
    ref_cam, mask = modules.point_sampling(ref3d, (-51.2, -51.2, -5.0, 51.2, 51.2, 3.0), lidar2img, img, (2.0, 58.0, 0.5))
    shapes, lsi = _level_tensors(levels)
    s = dict(case=case, net=net)
    s["query"] = torch.randn(1, Q, E, generator=g, device="cuda")
    s["grad_out"] = torch.randn(1, Q, E, generator=g, device="cuda")
    s["value"] = torch.randn(6, N, 1, E, generator=g, device="cuda")
    s["dist"] = torch.randn(6, N, 1, case["D"], generator=g, device="cuda").softmax(-1)
    s["kw"] = dict(value_dpt_dist=s["dist"], reference_points_cam=ref_cam, bev_mask=mask, spatial_shapes=shapes,
                   level_start_index=lsi)
    if case["module"] == "layer":
        s["kw"]["prev_bev"] = torch.randn(2, Q, E, generator=g, device="cuda")
    if case["train"]:
        net.train()
        s["params"] = list(net.parameters())
        s["leaves"] = [s["query"].requires_grad_(True), s["value"].requires_grad_(True), s["dist"].requires_grad_(True)]
    else:
        net.eval()
    return s


def prepare(case, seed):
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    if case["kind"] == "dist":
        levels = _levels(case)
        N = sum(h * w for h, w in levels)
        s = dict(case=case, N=N)
        s["logits"] = torch.randn(case["B"], case["D"], case["map_h"], case["map_w"], generator=g,
                                  device="cuda").requires_grad_(True)
        s["grad_out"] = torch.randn(case["B"], N, case["D"], generator=g, device="cuda").to(_DTYPE[case["dtype"]])
        s["shapes2"], s["lsi"] = _level_tensors(levels)
        return s
    if case["kind"] == "encoder":
        return _prepare_encoder(case, g)
    return _prepare_op(case, g)


# ------------------------------------------------------------------------------------------------
def _run_op3d(s):
    case = s["case"]
    fn = M.MultiScale3DDeformableAttnFunction_fp16 if case["dtype"] == "fp16" else \
        M.MultiScale3DDeformableAttnFunction if case["dtype"] == "bf16" else M.MultiScale3DDeformableAttnFunction_fp32
    if not case["train"]:
        with torch.no_grad():
            return fn.apply(s["value"], s["dist"], s["shapes3"], s["lsi"], s["loc"], s["attn"], 64, False)[0]
    out, ds = fn.apply(s["value"], s["dist"], s["shapes3"], s["lsi"], s["loc"], s["attn"], 64)
    return (out, ds) + torch.autograd.grad(out, s["leaves"], s["grad_out"])


def _run_two_stage(s):
    ds = M.MultiScaleDepthScoreSampleFunction_fp32.apply(s["dist"], s["shapes3"], s["lsi"], s["loc"], 64)
    out = M.WeightedMultiScaleDeformableAttnFunction_fp32.apply(
        s["value"], s["shapes2"], s["lsi"], s["loc"][..., :2].contiguous(), s["attn"], ds, 64)
    return (out, ds) + torch.autograd.grad(out, s["leaves"], s["grad_out"])


def _run_msda(s):
    fn = M.MultiScaleDeformableAttnFunction_fp32
    if not s["case"]["train"]:
        with torch.no_grad():
            return fn.apply(s["value"], s["shapes2"], s["lsi"], s["loc"], s["attn"], 64)
    out = fn.apply(s["value"], s["shapes2"], s["lsi"], s["loc"], s["attn"], 64)
    return (out,) + torch.autograd.grad(out, s["leaves"], s["grad_out"])


def _run_dist(s):
    case = s["case"]
    d = depth_distribution(s["logits"], s["shapes2"], s["lsi"], s["N"], case["activation"], _DTYPE[case["dtype"]])
    return (d,) + torch.autograd.grad(d, (s["logits"],), s["grad_out"])


def _run_encoder(s):
    case = s["case"]
    call = (lambda: s["net"](s["query"], value=s["value"], **s["kw"]))
    if not case["train"]:
        with torch.no_grad():
            return call()
    out = call()
    return (out,) + torch.autograd.grad(out, s["leaves"] + s["params"], s["grad_out"])


_RUN = {"op3d": _run_op3d, "two_stage": _run_two_stage, "msda": _run_msda, "dist": _run_dist, "encoder": _run_encoder}


def run(state):
    return _RUN[state["case"]["kind"]](state)


# ------------------------------------------------------------------------------------------------
def _op_work(case):
    levels = _levels(case)
    N = sum(h * w for h, w in levels)
    e = 4 if case["dtype"] == "fp32" else 2
    rows = case["B"] * case["Q"] * case["H"]
    pts = rows * len(levels) * case["P"]
    value, out = case["B"] * N * case["H"] * case["C"], rows * case["C"]
    small = pts * 4 * (3 if case["kind"] == "msda" else 4)            # location and attention weight of a point
    dist = 0 if case["kind"] == "msda" else case["B"] * N * case["D"] * (case["H"] if case["kind"] == "two_stage" else 1)
    eo = 2 if case["dtype"] == "fp16" and case["train"] else 4
    score = pts * 4 * eo if case["train"] and case["kind"] != "msda" else 0
    # of the features and the distribution only what the points can touch has to be read
    read = min(value, pts * 4 * case["C"]) + min(dist, pts * 8)
    b = read * e + small + out * eo + score
    f = pts * (4 * case["C"] * 2 + 40)
    if case["train"]:
        b += out * eo + (read + value + dist) * e + small
        f += pts * (4 * case["C"] * 4 + 80)
    return b, f


def work(case):
    if case["kind"] == "dist":
        n = sum(h * w for h, w in _levels(case))
        e = 4 if case["dtype"] == "fp32" else 2
        maps, dist = case["B"] * case["map_h"] * case["map_w"] * case["D"], case["B"] * n * case["D"]
        return {"bytes": 8 * maps + 2 * dist * e, "flops": 6 * maps + dist}
    if case["kind"] != "encoder":
        b, f = _op_work(case)
        return {"bytes": b, "flops": f}
    levels = _levels(case)
    N, E, Q = sum(h * w for h, w in levels), case["E"], case["bev_h"] * case["bev_w"]
    seen = 1.6 * Q                                   # (camera, query) pairs of the rig, nearly
    pts = seen * case["H"] * len(levels) * case["P"]
    per_query = case["H"] * len(levels) * case["P"] * 4
    gemm = 2 * E * (6 * N * E + seen * per_query + Q * (E + 2 * case["ffn"]))
    inputs = 4 * (6 * N * (E + case["D"]) + Q * E + 6 * Q * case["Z"] * 3) + 6 * Q * case["Z"]
    weights = 4 * (E * (2 * E + per_query + 2 * case["ffn"]))
    f = case["layers"] * (gemm + pts * (4 * (E // case["H"]) * 2 + 60))
    b = inputs + case["layers"] * weights + 4 * Q * E
    if case["module"] == "layer":                    # temporal self-attention over two maps, 4 points per item
        f += 2 * Q * E * (2 * E + E + 2 * 2 * case["H"] * 4 * 3) + 2 * Q * case["H"] * 4 * (4 * (E // case["H"]) * 2)
        b += 4 * 2 * Q * E + 4 * (2 * E * E + 2 * E * 2 * case["H"] * 4 * 3)
    if case["train"]:
        f *= 3
        b += 4 * (Q * E + 6 * N * (E + case["D"]) + Q * E) + case["layers"] * weights
    return {"bytes": b, "flops": f}


def tolerance(case):
    if case["kind"] == "encoder":
        return {"rel": 1e-2}                         # tf32 products
    if case["dtype"] == "fp32":
        return {"rel": 2e-5}                         # 32-bit sums in another order
    if case["kind"] == "op3d" and case["dtype"] == "bf16" and not case["train"]:
        return {"rel": 2e-5}                         # bf16 storage only: products, sums and results are 32-bit
    return {"rel": 1e-2}                             # results rounded to the 16-bit storage type
