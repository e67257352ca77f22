"""Under torch.jit.trace a call is recorded as an operation of the graph: the traced function computes anew from the inputs
it is given."""
import pytest
import torch

from dfa3d_b200 import functions as F
from dfa3d_b200 import layer_ops
from dfa3d_b200 import workloads as wl

pytestmark = [pytest.mark.gpu, pytest.mark.filterwarnings("ignore::torch.jit.TracerWarning", "ignore::DeprecationWarning")]
DEV = "cuda"


def test_traced_operator_follows_its_inputs(lib_built):
    d = {k: v.to(DEV) for k, v in wl.make_inputs(wl.WORKLOADS["tiny"]).items()}

    def call(value, attn):
        return F.MultiScale3DDeformableAttnFunction_fp32.apply(value, d["dist"], d["shapes"], d["lsi"], d["loc"], attn, 64,
                                                               False)[0]

    with torch.no_grad():
        traced = torch.jit.trace(call, (d["value"], d["attn"]), check_trace=False)
        value, attn = torch.randn_like(d["value"]), torch.rand_like(d["attn"])
        want = call(value, attn)
        spoil = [torch.full_like(want, float("nan")) for _ in range(8)]   # what freed blocks hand to an empty tensor
        del spoil
        assert torch.equal(traced(value, attn), want)


def test_traced_layer_operations_follow_their_inputs(lib_built):
    torch.manual_seed(0)
    linears = [layer_ops.Linear(32, 32).to(DEV) for _ in range(3)]
    norm, relu = layer_ops.AddLayerNorm(32).to(DEV), torch.nn.ReLU()
    for p in torch.nn.ModuleList([*linears, norm]).parameters():
        p.requires_grad_(False)                                           # a trace takes constants without a gradient only

    def call(x):
        parts = layer_ops.joint_linear(x, *linears)
        x = parts[..., :32] if parts is not None else linears[0](x)
        return norm(layer_ops.linear_relu(x, linears[1], relu), linears[2](x))

    with torch.no_grad():
        traced = torch.jit.trace(call, (torch.randn(7, 32, device=DEV),), check_trace=False)
        x = torch.randn(7, 32, device=DEV)
        want = call(x)
        spoil = [torch.full((7, n), float("nan"), device=DEV) for n in (32, 96) for _ in range(8)]
        del spoil
        torch.testing.assert_close(traced(x), want, rtol=1e-5, atol=1e-5)
