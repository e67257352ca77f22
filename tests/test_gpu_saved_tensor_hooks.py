"""Saved-tensor hooks see what a forward keeps.  A hook that hands back equal tensors -- moved, in another layout -- changes
nothing; one that hands back another type or size is refused before a kernel reads by its address."""
import pytest
import torch

from dfa3d_b200 import functions as F
from dfa3d_b200 import layer_ops
from dfa3d_b200 import workloads as wl
from dfa3d_b200.dist_producer import depth_distribution

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _call(kind):
    """A function of no arguments that runs the forward, and its leaves."""
    torch.manual_seed(0)
    d = {k: v.to(DEV) for k, v in wl.make_inputs(wl.WORKLOADS["tiny"]).items()}
    value, dist, loc, attn = (d[k].requires_grad_(True) for k in ("value", "dist", "loc", "attn"))
    shapes2, loc2 = d["shapes"][:, :2].contiguous(), d["loc"][..., :2].detach().contiguous().requires_grad_(True)
    layers = [layer_ops.Linear(32, 32).to(DEV) for _ in range(2)]
    params = [p for m in layers for p in m.parameters()]
    norm, x = layer_ops.AddLayerNorm(32).to(DEV), torch.randn(9, 32, device=DEV, requires_grad=True)
    logits = torch.randn(1, 16, 4, 5, device=DEV, requires_grad=True)
    table = torch.tensor([[4, 5]], device=DEV), torch.zeros(1, dtype=torch.int64, device=DEV)
    return {
        "fused": (lambda: F.MultiScale3DDeformableAttnFunction_fp32.apply(value, dist, d["shapes"], d["lsi"], loc, attn, 64)[0],
                  [value, dist, loc, attn]),
        "depth": (lambda: F.MultiScaleDepthScoreSampleFunction.apply(dist[:, :, None].repeat(1, 1, attn.shape[2], 1),
                                                                     d["shapes"], d["lsi"], loc, 64), [dist, loc]),
        "msda": (lambda: F.MultiScaleDeformableAttnFunction_fp32.apply(value, shapes2, d["lsi"], loc2, attn, 64),
                 [value, loc2, attn]),
        "linear": (lambda: layers[0](x), [x] + params[:2]),
        "linear_relu": (lambda: layer_ops.linear_relu(x, layers[0], torch.nn.ReLU()), [x] + params[:2]),
        "joint": (lambda: layer_ops.joint_linear(x, *layers), [x] + params),
        "norm": (lambda: norm(x, x * 2), [x, norm.weight, norm.bias]),
        "dist": (lambda: depth_distribution(logits, *table, 20), [logits]),
    }[kind]


KINDS = ["fused", "depth", "msda", "linear", "linear_relu", "joint", "norm", "dist"]


def _other_layout(t):
    return t.transpose(0, -1).contiguous().transpose(0, -1) if t.dim() > 1 else t.clone()


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("hook", ["cpu", "layout"])
def test_equal_tensors_give_equal_gradients(lib_built, kind, hook):
    call, leaves = _call(kind)
    out = call()
    go = torch.randn(out.shape, generator=torch.Generator().manual_seed(1)).to(DEV)
    want = torch.autograd.grad(out, leaves, go)
    pack, unpack = (lambda t: t.cpu(), lambda t: t.to(DEV)) if hook == "cpu" else (lambda t: t.clone(), _other_layout)
    with torch.autograd.graph.saved_tensors_hooks(pack, unpack):
        out = call()
    for a, b in zip(torch.autograd.grad(out, leaves, go), want):
        torch.testing.assert_close(a, b, rtol=1e-4, atol=1e-5)         # reductions in another order


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("hook", ["type", "size"])
def test_other_tensors_are_refused(lib_built, kind, hook):
    call, leaves = _call(kind)
    pack = (lambda t: t.half() if t.is_floating_point() else t) if hook == "type" else (lambda t: t.flatten()[:1].clone())
    with torch.autograd.graph.saved_tensors_hooks(pack, lambda t: t):
        out = call()
    with pytest.raises(RuntimeError, match="saved-tensor hook"):
        torch.autograd.grad(out, leaves, torch.ones_like(out))
