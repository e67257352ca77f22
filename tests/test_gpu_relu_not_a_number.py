"""linear_relu and its backward treat NaN and infinities as relu(linear(x)) does: NaN stays NaN and lets its gradient pass."""
import pytest
import torch
import torch.nn as nn
import torch.nn.functional as F

from dfa3d_b200 import layer_ops

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("rows", [5, 70, 16400])
@pytest.mark.parametrize("bad", [float("nan"), float("inf"), -float("inf")])
def test_values_that_are_no_numbers(lib_built, rows, bad):
    torch.manual_seed(rows)
    lin = layer_ops.Linear(24, 32).to(DEV)
    x = torch.randn(rows, 24, device=DEV)
    x[1, 3] = bad
    x.requires_grad_(True)
    go = torch.randn(rows, 32, device=DEV)
    got = layer_ops.linear_relu(x, lin, nn.ReLU())
    want = F.relu(F.linear(x, lin.weight, lin.bias))
    pairs = [(got, want)] + list(zip(torch.autograd.grad(got, [x, lin.weight, lin.bias], go),
                                     torch.autograd.grad(want, [x, lin.weight, lin.bias], go)))
    for a, b in pairs:
        torch.testing.assert_close(a, b, rtol=1e-4, atol=1e-4 * rows ** 0.5, equal_nan=True)
