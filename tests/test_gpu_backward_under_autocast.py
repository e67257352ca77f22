"""backward() called inside an autocast region, of a forward outside it: the layers' gradients are the float32 ones.  Row
counts on both sides of the split of the weight gradient."""
import pytest
import torch

from dfa3d_b200 import layer_ops

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("rows", [33, 16384 + 5])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("kind", ["linear", "linear_relu", "joint"])
def test_gradients_stay_float32(lib_built, rows, dtype, kind):
    torch.manual_seed(rows)
    layers = [layer_ops.Linear(24, 32).to(DEV) for _ in range(2)]
    x, go = torch.randn(rows, 24, device=DEV, requires_grad=True), torch.randn(rows, 64, device=DEV)
    leaves = [x] + [p for m in layers for p in m.parameters()]

    def grads(autocast):
        if kind == "joint":
            y = layer_ops.joint_linear(x, *layers)
        elif kind == "linear":
            y = torch.cat([m(x) for m in layers], -1)
        else:
            y = torch.cat([layer_ops.linear_relu(x, m, torch.nn.ReLU()) for m in layers], -1)
        with torch.autocast("cuda", dtype=dtype, enabled=autocast):
            return torch.autograd.grad(y, leaves, go)

    for a, b in zip(grads(True), grads(False)):
        assert a.dtype == torch.float32
        # the same products; only the column sums' order varies from run to run
        assert float((a - b).abs().max()) <= 1e-5 * float(b.abs().max())
