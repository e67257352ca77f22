"""A query's result does not depend on what else its launch holds: many cameras at once, one of them alone and a few of its
queries give the same bits, in the sizes where the kernels that put several items into a warp give an item more lanes in the
smaller launch.  Dense and ragged, with and without scores, all storage types; plain 2-D; from offsets."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"
CAMS, Q, H, D = 6, 500, 8, 16
LEVELS = {1: ((23, 40),), 2: ((23, 40), (12, 20))}


def _problem(L, P, C, dtype):
    g = torch.Generator(device=DEV).manual_seed(10 * P + C)
    levels = torch.tensor([[h, w, D] for h, w in LEVELS[L]], device=DEV)
    hw = levels[:, 0] * levels[:, 1]
    lsi = torch.cat([hw.new_zeros(1), hw.cumsum(0)[:-1]])
    N = int(hw.sum())
    r = lambda *s: torch.randn(*s, generator=g, device=DEV)
    return dict(value=r(CAMS, N, H, C).to(dtype), dist=r(CAMS, N, D).softmax(-1).to(dtype), shapes=levels, lsi=lsi,
                loc=torch.rand(CAMS, Q, H, L, P, 3, generator=g, device=DEV) * 1.1 - 0.05,
                attn=r(CAMS, Q, H, L * P).softmax(-1).view(CAMS, Q, H, L, P), grad_out=r(CAMS, Q, H * C))


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("L,P,C", [(1, 1, 16), (1, 3, 32), (1, 4, 16), (1, 4, 32), (1, 4, 64), (2, 1, 64), (1, 5, 32), (1, 8, 16),
                                   (2, 4, 32), (1, 7, 64)])
def test_cameras_together_and_alone(lib_built, L, P, C, dtype):
    from dfa3d_b200 import ext
    d = _problem(L, P, C, dtype)
    fixed = d["shapes"], d["lsi"]
    shapes2 = d["shapes"][:, :2].contiguous()
    out, ds = ext.dfa3d_fused_forward(d["value"], d["dist"], *fixed, d["loc"], d["attn"], 64)
    bare = ext.dfa3d_fused_forward(d["value"], d["dist"], *fixed, d["loc"], d["attn"], 64, False)[0]
    loc2 = d["loc"][..., :2].contiguous()
    two = ext.wms_deform_attn_forward(d["value"], shapes2, d["lsi"], loc2, d["attn"], ds, 64)
    gl, ga = torch.empty_like(d["loc"]), torch.empty_like(d["attn"])
    gv, gd = (torch.zeros(d[k].shape, device=DEV) for k in ("value", "dist"))
    ext.dfa3d_fused_backward(d["value"], d["dist"], *fixed, d["loc"], d["attn"], d["grad_out"], gv, gd, gl, ga, 64)
    offsets = torch.arange(CAMS + 1, device=DEV, dtype=torch.int32) * Q
    rows = lambda x: x.reshape(-1, *x.shape[2:])
    ragged = ext.dfa3d_fused_forward_ragged(d["value"], d["dist"], *fixed, rows(d["loc"]), rows(d["attn"]), offsets, Q)
    assert torch.equal(ragged[0], rows(out)) and torch.equal(ragged[1], rows(ds)) and torch.equal(bare, out)
    for b, n in ((0, Q), (4, Q), (5, 33)):
        one = {k: d[k][b:b + 1] if k in ("value", "dist") else d[k][b:b + 1, :n].contiguous()
               for k in ("value", "dist", "loc", "attn", "grad_out")}
        o, s = ext.dfa3d_fused_forward(one["value"], one["dist"], *fixed, one["loc"], one["attn"], 64)
        assert torch.equal(o, out[b:b + 1, :n]) and torch.equal(s, ds[b:b + 1, :n])
        assert torch.equal(o, ext.dfa3d_fused_forward(one["value"], one["dist"], *fixed, one["loc"], one["attn"], 64, False)[0])
        assert torch.equal(two[b:b + 1, :n], ext.wms_deform_attn_forward(
            one["value"], shapes2, d["lsi"], one["loc"][..., :2].contiguous(), one["attn"], s, 64))
        gl1, ga1 = torch.empty_like(one["loc"]), torch.empty_like(one["attn"])
        ext.dfa3d_fused_backward(one["value"], one["dist"], *fixed, one["loc"], one["attn"], one["grad_out"], gv[b:b + 1],
                                 gd[b:b + 1], gl1, ga1, 64)
        assert torch.equal(gl1, gl[b:b + 1, :n]) and torch.equal(ga1, ga[b:b + 1, :n])


@pytest.mark.parametrize("P,C", [(4, 16), (4, 32), (8, 32), (3, 64)])
def test_plain_2d(lib_built, P, C):
    from dfa3d_b200 import ext
    d = _problem(1, P, C, torch.float32)
    shapes2, loc = d["shapes"][:, :2].contiguous(), d["loc"][..., :2].contiguous()
    out = ext.ms_deform_attn_forward(d["value"], shapes2, d["lsi"], loc, d["attn"], 64)
    for b, n in ((1, Q), (3, 33)):
        got = ext.ms_deform_attn_forward(d["value"][b:b + 1], shapes2, d["lsi"], loc[b:b + 1, :n].contiguous(),
                                         d["attn"][b:b + 1, :n].contiguous(), 64)
        assert torch.equal(got, out[b:b + 1, :n])


@pytest.mark.parametrize("P,C", [(4, 16), (4, 32), (8, 32)])
def test_from_offsets(lib_built, P, C):
    from dfa3d_b200 import ext
    d = _problem(1, P, C, torch.float32)
    g = torch.Generator(device=DEV).manual_seed(7)
    r = lambda *s: torch.randn(*s, generator=g, device=DEV)
    a = [torch.rand(CAMS, Q, 2, 3, generator=g, device=DEV), r(CAMS, Q, H, 1, P, 2), r(CAMS, Q, H, 1, P), r(CAMS, Q, H, P)]
    out = ext.dfa3d_attn3d_forward(d["value"], d["dist"], d["shapes"], d["lsi"], *a)
    for b, n in ((1, Q), (3, 33)):
        got = ext.dfa3d_attn3d_forward(d["value"][b:b + 1], d["dist"][b:b + 1], d["shapes"], d["lsi"],
                                       *(x[b:b + 1, :n].contiguous() for x in a))
        assert torch.equal(got, out[b:b + 1, :n])
