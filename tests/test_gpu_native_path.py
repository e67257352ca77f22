"""The native host path of the autograd Functions gives what the Python Functions give: same results, same
gradients, same refusals; and it leaves every case that is not plain to them."""
import pytest
import torch

from dfa3d_b200 import functions as F
from dfa3d_b200 import workloads as wl
from helpers import BWD, assert_close

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _python(cls):
    """The same Function without the native path (which only the exact class takes)."""
    return type("Python" + cls.__name__, (cls,), {})


def _inputs(name, half=False):
    d = {k: v.to(DEV) for k, v in wl.make_inputs(wl.WORKLOADS[name]).items()}
    if half:
        d["value"], d["dist"], d["grad_out"] = d["value"].half(), d["dist"].half(), d["grad_out"].half()
    return d


def _args(d, kind):
    shapes2 = d["shapes"][:, :2].contiguous()
    loc2 = d["loc"][..., :2].contiguous()
    B, Q = d["loc"].shape[:2]
    q_off = (torch.arange(B + 1, dtype=torch.int32) * Q).to(DEV)
    score = torch.rand(*d["attn"].shape, 4, generator=torch.Generator().manual_seed(3)).to(DEV)
    flat = lambda t: t.flatten(0, 1).contiguous()
    ref, uv, od = d["loc"][:, :, 0, 0, :1].contiguous(), loc2 * 3, d["loc"][..., 2:].contiguous()
    logits = d["attn"].flatten(3).log()
    return {
        "fused": (d["value"], d["dist"], d["shapes"], d["lsi"], d["loc"], d["attn"], 64),
        "wms": (d["value"], shapes2, d["lsi"], loc2, d["attn"], score, 64),
        "msda": (d["value"], shapes2, d["lsi"], loc2, d["attn"], 64),
        "depth": (d["dist"], d["shapes"], d["lsi"], d["loc"], 64),
        "attn3d": (d["value"], d["dist"], d["shapes"], d["lsi"], ref, uv, od, logits),
        "ragged": (d["value"], d["dist"], d["shapes"], d["lsi"], flat(d["loc"]), flat(d["attn"]), q_off, Q),
        "attn3d_ragged": (d["value"], d["dist"], d["shapes"], d["lsi"], flat(ref), flat(uv), flat(od), flat(logits),
                          q_off, Q),
    }[kind]


CASES = [("fused", F.MultiScale3DDeformableAttnFunction_fp32, False), ("fused", F.MultiScale3DDeformableAttnFunction, True),
         ("fused", F.MultiScale3DDeformableAttnFunction_fp16, True), ("wms", F.WeightedMultiScaleDeformableAttnFunction, False),
         ("wms", F.WeightedMultiScaleDeformableAttnFunction_fp16, True), ("msda", F.MultiScaleDeformableAttnFunction_fp32, False),
         ("msda", F.MultiScaleDeformableAttnFunction_fp16, True), ("depth", F.MultiScaleDepthScoreSampleFunction, False),
         ("attn3d", F.DeformableAttn3DFromOffsetsFunction_fp32, False),
         ("ragged", F.MultiScale3DDeformableAttnRaggedFunction_fp32, False),
         ("attn3d_ragged", F.DeformableAttn3DFromOffsetsRaggedFunction, False)]


@pytest.mark.parametrize("kind,cls,half", CASES, ids=lambda v: getattr(v, "__name__", str(v)))
@pytest.mark.parametrize("name", ["tiny", "cfg0"])
def test_native_path_equals_the_python_function(lib_built, kind, cls, half, name):
    d = _inputs(name, half)
    got = []
    for fn in (cls, _python(cls)):
        args = [a.detach().clone().requires_grad_(a.is_floating_point()) if torch.is_tensor(a) else a
                for a in _args(d, kind)]
        out = fn.apply(*args)
        outs = out if isinstance(out, tuple) else (out,)
        leaves = [a for a in args if torch.is_tensor(a) and a.requires_grad and not (kind.startswith("attn3d") and a is args[4])]
        g = torch.randn(outs[0].shape, generator=torch.Generator().manual_seed(5)).to(DEV, outs[0].dtype)
        grads = torch.autograd.grad(outs[0], leaves, g)
        with torch.no_grad():
            bare = fn.apply(*args)
        bare = bare if isinstance(bare, tuple) else (bare,)
        assert not bare[0].requires_grad and all(torch.equal(a, b) for a, b in zip(bare, outs))
        got.append((outs, grads))
    (o0, g0), (o1, g1) = got
    assert type(o0[0].grad_fn).__name__ != type(o1[0].grad_fn).__name__          # two different implementations
    for a, b in zip(o0, o1):
        assert a.dtype == b.dtype and torch.equal(a, b)
    for i, (a, b) in enumerate(zip(g0, g1)):
        assert a.dtype == b.dtype and a.shape == b.shape
        tol = dict(rtol=2e-3, atol=1e-3 * float(b.abs().max())) if a.dtype == torch.float16 else BWD
        assert_close(f"grad {i}", a.float(), b.float(), **tol)


def test_native_path_refuses_what_the_python_function_refuses(lib_built):
    d = _inputs("tiny")
    fn = F.MultiScale3DDeformableAttnFunction
    args = list(_args(d, "fused"))
    args[0] = args[0].requires_grad_(True)
    out, score = fn.apply(*args)
    with pytest.raises(NotImplementedError):                                      # gradient into depth_score
        (out.sum() + score.sum()).backward()
    out, score = fn.apply(*args)
    (g,) = torch.autograd.grad(out.pow(2).sum(), args[0], create_graph=True)
    with pytest.raises(RuntimeError, match="once_differentiable"):
        g.sum().backward()
    out, score = fn.apply(*args[:7], False)
    assert score is None
    with pytest.raises(RuntimeError, match="contiguous"):                         # left to the Python checks
        fn.apply(args[0].transpose(0, 1), *args[1:])
    with torch.autocast("cuda", dtype=torch.float16):
        out = F.MultiScale3DDeformableAttnFunction_fp32.apply(args[0].half(), args[1].half(), *args[2:])[0]
    assert out.dtype == torch.float32
    out = fn.apply(*[a.double() if torch.is_tensor(a) and a.is_floating_point() else a for a in args])[0]
    assert out.dtype == torch.float64
