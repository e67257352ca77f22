"""Launches that fill the device: items that several of a warp share keep the lanes that their points need, and a CTA walks
several groups of items, so that a warp's tables are used again.  Every form of the operator -- one-stage, two-stage, plain
2-D, from offsets, cameras of different numbers of queries, queries by index -- against the CPU oracle, with every storage
type; first that the sizes used here reach what they are for."""
import numpy as np
import pytest
import torch

from dfa3d_b200 import workloads as wl
from helpers import BWD, FWD, assert_close, oracle_all
from test_walk import walk  # noqa: F401 (fixture)

DEV = "cuda"
B, H = 3, 3
LEVELS = ((12, 20), (6, 9), (4, 5))
STORAGE = {"fp32": (torch.float32, torch.float32), "bf16": (torch.bfloat16, torch.bfloat16),
           "fp16": (torch.float16, torch.float16), "fp32_bf16": (torch.float32, torch.bfloat16),
           "bf16_fp32": (torch.bfloat16, torch.float32)}
# (levels, points a level, channels); CTA-sized batches of items: two of them a CTA where 4 or 5 CTAs are resident on an SM
# (880), where 6 are (1100)
FEW = [(1, 3, 64), (1, 4, 16), (1, 4, 32), (1, 5, 16), (1, 7, 64), (2, 4, 32), (3, 4, 32), (2, 8, 64)]
BATCHES = (880, 1100)
# one item a warp: two groups a CTA in the backward (680 to 910 groups at 4 resident), two to five in the forward
MANY = [(1, 17, 8), (1, 20, 16), (1, 32, 32), (1, 32, 64), (2, 20, 64), (3, 6, 32)]
GROUPS = (800, 2880)
FULL = 36000                                          # groups from which every launch takes the full walk


def queries(LP, batches):
    return -(-batches * 8 * (32 // (4 if LP <= 4 else 8 if LP <= 8 else 16)) // (B * H))


def test_sizes_reach_the_lanes_and_walks_they_are_for(walk):
    for L, P, C in FEW:
        for v in (4, 8):
            for batches in BATCHES:
                LP, items = L * P, B * H * queries(L * P, batches)
                least = 4 if LP <= 4 else 8 if LP <= 8 else 16
                assert all(walk.lanes(LP, C, v, items, bwd, bins, 148) == least for bwd in (0, 1) for bins in (0, 1))
        took = lambda n, resident: walk.forward(-(-n // B), B, 2, resident, 148, 6, 8)
        assert took(880, 4) == took(880, 5) == took(1100, 6) == 2
        assert walk.backward(-(-880 // B), B, 2, 4, 148) == 2
    assert walk.backward(-(-800 // B), B, 4, 4, 148) == 2
    assert all(1 < walk.forward(-(-n // B), B, 8, r, 148, 2, 8) < 8 for n, r in ((800, 4), (800, 5), (2880, 4), (2880, 5), (2880, 6)))
    assert walk.forward(FULL // B, B, 8, 5, 148, 2, 8) == 8 and walk.backward(FULL // B, B, 4, 4, 148) == 4


def problem(L, P, C, Q, storage, seed):
    w = wl.WORKLOADS["tiny"].with_(B=B, H=H, C=C, D=6, Q=Q, levels=LEVELS[:L], P=P, seed=seed, oob=True,
                                   value_dtype="fp32" if storage == "fp32" else "fp16" if storage == "fp16" else "bf16")
    d = wl.make_inputs(w, head_repeat=True)
    t = {k: v.to(DEV) for k, v in d.items()}
    vt, dt = STORAGE[storage]
    t["value"], t["dist"] = t["value"].to(vt), t["dist"].to(dt)
    return d, t


def cameras_of_different_sizes(Q):
    counts = torch.tensor([Q, Q // 3, Q - 1])
    offsets = torch.cat([torch.zeros(1, dtype=torch.int64), counts.cumsum(0)]).int().to(DEV)
    rows = lambda x: torch.cat([x[b, :int(n)] for b, n in enumerate(counts)]).contiguous()
    return offsets, rows


def zeros(t):
    return [torch.zeros(t[k].shape, device=DEV) for k in ("value", "dist")]


def nans(*like):
    return [torch.full_like(x, float("nan")) for x in like]


def check(names, got, want, tol=BWD):
    for name, g, w in zip(names, got, want):
        assert_close(name, g, w, **tol)


def check_from_locations(d, t, Q):
    from dfa3d_b200 import ext
    ref = oracle_all(d, np.float32)
    args = [t[k] for k in ("value", "dist", "shapes", "lsi", "loc", "attn")]
    out, ds = ext.dfa3d_fused_forward(*args, 64)
    check(("out", "depth_score"), (out, ds), (ref["out"], ref["ds"]), FWD)
    assert_close("out only", ext.dfa3d_fused_forward(*args, 64, False)[0], ref["out"], **FWD)
    grads = "grad_value", "grad_dist", "grad_loc", "grad_attn"
    got = zeros(t) + nans(t["loc"], t["attn"])
    ext.dfa3d_fused_backward(*args, t["grad_out"], *got, 64)
    check(grads, got, [ref[k] for k in grads])
    # cameras of different numbers of queries: per-query results are the dense ones
    offsets, rows = cameras_of_different_sizes(Q)
    some = [*args[:4], rows(t["loc"]), rows(t["attn"])]
    r_out, r_ds = ext.dfa3d_fused_forward_ragged(*some, offsets, Q)
    assert torch.equal(r_out, rows(out)) and torch.equal(r_ds, rows(ds))
    r_got = zeros(t) + nans(*some[4:])
    ext.dfa3d_fused_backward_ragged(*some, offsets, Q, rows(t["grad_out"]), *r_got)
    assert torch.equal(r_got[2], rows(got[2])) and torch.equal(r_got[3], rows(got[3]))
    d1 = dict(d, **{k: d[k][1:2, :Q // 3] if k in ("loc", "attn", "grad_out") else d[k][1:2] for k in
                    ("value", "dist", "loc", "attn", "grad_out")})
    one = oracle_all(d1, np.float32)
    check(("ragged grad_value", "ragged grad_dist"), (r_got[0][1:2], r_got[1][1:2]), (one["grad_value"], one["grad_dist"]))


def check_two_stage_and_2d(d, t, plain):
    import dfa3d_oracle as O
    from dfa3d_b200 import ext
    n = {k: v.numpy() for k, v in d.items()}
    shapes2, loc2 = t["shapes"][:, :2].contiguous(), t["loc"][..., :2].contiguous()
    n2 = n["shapes"][:, :2].copy(), n["lsi"], n["loc"][..., :2].copy(), n["attn"]
    ds = O.ms_depth_score_sample_forward(n["dist"], n["shapes"], n["lsi"], n["loc"])
    args = [t["value"], shapes2, t["lsi"], loc2, t["attn"]]
    dsd = torch.from_numpy(ds).to(DEV)
    assert_close("two-stage out", ext.wms_deform_attn_forward(*args, dsd, 64), O.wms_deform_attn_forward(n["value"], *n2, ds), **FWD)
    got = zeros(t)[:1] + nans(loc2, t["attn"], dsd)
    ext.wms_deform_attn_backward(*args, dsd, t["grad_out"], *got, 64)
    check(("two-stage grad_value", "grad_loc", "grad_attn", "grad_ds"), got,
          O.wms_deform_attn_backward(n["value"], *n2, ds, n["grad_out"]))
    if not plain:
        return
    assert_close("2-D out", ext.ms_deform_attn_forward(*args, 64), O.ms_deform_attn_forward(n["value"], *n2), **FWD)
    got = zeros(t)[:1] + nans(loc2, t["attn"])
    ext.ms_deform_attn_backward(*args, t["grad_out"], *got, 64)
    check(("2-D grad_value", "grad_loc", "grad_attn"), got, O.ms_deform_attn_backward(n["value"], *n2, n["grad_out"]))


def check_from_offsets(d, t, Q):
    import dfa3d_oracle as O
    from dfa3d_b200 import ext
    _, _, _, L, P, _ = d["loc"].shape
    g = torch.Generator().manual_seed(Q)
    Z = 2 if P % 2 == 0 else 1
    raw = [torch.rand(B, Q, Z, 3, generator=g) * 1.2 - 0.1, torch.randn(B, Q, H, L, P, 2, generator=g) * 1.5,
           torch.randn(B, Q, H, L, P, generator=g), torch.randn(B, Q, H, L * P, generator=g)]
    n = [d[k].numpy() for k in ("value", "dist", "shapes", "lsi")] + [x.numpy() for x in raw]
    fixed, raw = [t[k] for k in ("value", "dist", "shapes", "lsi")], [x.to(DEV) for x in raw]
    out = ext.dfa3d_attn3d_forward(*fixed, *raw)
    assert_close("from offsets", out, O.attn3d_forward(*n), **FWD)
    got = zeros(t) + nans(*raw[1:])
    ext.dfa3d_attn3d_backward(*fixed, *raw, t["grad_out"], *got)
    check(("grad_value", "grad_dist", "grad_off_uv", "grad_off_d", "grad_logits"), got, O.attn3d_backward(*n, d["grad_out"].numpy()))
    offsets, rows = cameras_of_different_sizes(Q)
    some = [rows(x) for x in raw]
    assert torch.equal(ext.dfa3d_attn3d_forward_ragged(*fixed, *some, offsets, Q), rows(out))
    r_got = zeros(t) + nans(*some[1:])
    ext.dfa3d_attn3d_backward_ragged(*fixed, *some, offsets, Q, rows(t["grad_out"]), *r_got)
    for r, dense in zip(r_got[2:], got[2:]):
        assert torch.equal(r, rows(dense))


@pytest.mark.gpu
@pytest.mark.parametrize("batches", BATCHES)
@pytest.mark.parametrize("storage", sorted(STORAGE))
@pytest.mark.parametrize("L,P,C", FEW)
def test_items_that_share_a_warp(lib_built, L, P, C, storage, batches):
    Q = queries(L * P, batches)
    d, t = problem(L, P, C, Q, storage, seed=10 * P + L)
    check_from_locations(d, t, Q)
    check_from_offsets(d, t, Q)
    if not storage.startswith("fp32_"):
        check_two_stage_and_2d(d, t, storage == "fp32")


@pytest.mark.gpu
@pytest.mark.parametrize("groups", GROUPS)
@pytest.mark.parametrize("storage", sorted(STORAGE))
@pytest.mark.parametrize("L,P,C", MANY)
def test_an_item_a_warp(lib_built, L, P, C, storage, groups):
    Q = -(-groups * 8 // (B * H))
    d, t = problem(L, P, C, Q, storage, seed=10 * P + L)
    check_from_locations(d, t, Q)
    check_from_offsets(d, t, Q)
    if not storage.startswith("fp32_"):
        check_two_stage_and_2d(d, t, storage == "fp32")


@pytest.mark.gpu
@pytest.mark.parametrize("L,P,C,storage", [(1, 17, 16, "fp32"), (1, 32, 16, "bf16"), (1, 20, 32, "fp16"), (1, 32, 32, "bf16_fp32")])
def test_the_full_walk(lib_built, L, P, C, storage):
    Q = -(-FULL * 8 // (B * H))
    d, t = problem(L, P, C, Q, storage, seed=P)
    check_from_locations(d, t, Q)
    check_from_offsets(d, t, Q)


@pytest.mark.gpu
@pytest.mark.parametrize("L,P", [(1, 4), (1, 8), (2, 16)])
def test_queries_by_index(lib_built, L, P):
    """The spatial cross-attention without gradients reads a query's row through the plan's index; with them it copies rows."""
    from dfa3d_b200 import modules
    torch.manual_seed(P)
    E, heads, D, cams, Q, Z = 64, 2, 6, 3, (queries(L * P, 880) if L * P <= 16 else 2200) * B * H // 6, 4
    shapes = torch.tensor(LEVELS[:L], device=DEV)
    lsi = torch.cat([shapes.new_zeros(1), shapes.prod(1).cumsum(0)[:-1]])
    N = int(shapes.prod(1).sum())
    net = modules.SpatialCrossAttention_DFA3D(E, cams, 0.0, modules.MSDeformableAttention3D_DFA3D(E, heads, L, P), bev_h=1,
                                              bev_w=Q, num_head=heads).to(DEV)
    with torch.no_grad():
        for p in net.parameters():
            p.copy_(torch.randn_like(p) * 0.1)
    mask = torch.rand(cams, 1, Q, Z, device=DEV) < 0.7
    kw = dict(value=torch.randn(cams, N, 1, E, device=DEV), value_dpt_dist=torch.rand(cams, N, 1, D, device=DEV),
              reference_points_cam=torch.rand(cams, 1, Q, Z, 3, device=DEV), bev_mask=mask, spatial_shapes=shapes,
              level_start_index=lsi)
    query = torch.randn(1, Q, E, device=DEV)
    want = net(query, **kw).detach()
    with torch.no_grad():
        got = net(query, **kw)
    assert float((got - want).abs().max()) <= 1e-5 * float(want.abs().max())


@pytest.mark.gpu
@pytest.mark.parametrize("L,P", [(1, 4), (1, 8), (2, 8)])
def test_2d_from_offsets(lib_built, monkeypatch, L, P):
    """The decoder's attention, whose kernel forms the locations, against its operations one after the other."""
    from dfa3d_b200 import modules
    E, heads, bs, Q = 64, 2, 3, queries(L * P, 880) * B * H // 6
    g = torch.Generator().manual_seed(P)
    shapes = torch.tensor(LEVELS[:L], device=DEV)
    lsi = torch.cat([shapes.new_zeros(1), shapes.prod(1).cumsum(0)[:-1]])
    query, grad = (torch.randn(Q, bs, E, generator=g).to(DEV) for _ in range(2))
    bev = torch.randn(int(shapes.prod(1).sum()), bs, E, generator=g).to(DEV)
    refp = torch.rand(bs, Q, L, 2, generator=g).to(DEV)
    net = modules.CustomMSDeformableAttention(E, heads, L, P, dropout=0.0).to(DEV)
    with torch.no_grad():
        net.attention_weights.weight.normal_(0, 0.05)
        net.sampling_offsets.bias.add_(torch.rand(net.sampling_offsets.bias.shape, generator=g).to(DEV))

    def run():
        v = bev.clone().requires_grad_(True)
        out = net(query, value=v, reference_points=refp, spatial_shapes=shapes, level_start_index=lsi)
        return (out.detach(), *torch.autograd.grad(out, [v, net.attention_weights.weight, net.sampling_offsets.weight], grad))

    got = run()
    monkeypatch.setattr(modules, "_attention_2d", lambda *a: None)
    # sums of some hundred terms (value) and of 9 000 (weights), in another order
    for name, a, b, tol in zip(("out", "grad_value", "grad_logit_weight", "grad_offset_weight"), got, run(), (1e-5, 1e-5, 1e-4, 1e-4)):
        assert float((a - b).abs().max()) <= tol * float(b.abs().max()), name
