"""Contiguous tensors that start off a 16-byte boundary, as slices and views of larger buffers do, where only an address
that a kernel reads in wider words asks for more."""
import pytest
import torch
import torch.nn as nn
import torch.nn.functional as F

from dfa3d_b200 import layer_ops, modules

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _shifted(t, floats):
    """The same values `floats` elements behind a 16-byte boundary."""
    buf = torch.empty(t.numel() + floats, device=t.device)
    assert buf.data_ptr() % 16 == 0
    return buf[floats:].view(t.shape).copy_(t)


@pytest.mark.parametrize("floats", [1, 2, 3])
def test_attention_2d_takes_unaligned_reference_points(lib_built, floats):
    torch.manual_seed(floats)
    net = modules.CustomMSDeformableAttention(64, 4, 1, 4, dropout=0.0, batch_first=True).to(DEV)
    nn.init.normal_(net.sampling_offsets.weight, 0, 0.05)
    query, value = torch.randn(1, 37, 64, device=DEV), torch.randn(1, 80, 64, device=DEV)
    ref = torch.rand(1, 37, 1, 2, device=DEV)
    kw = dict(value=value, spatial_shapes=torch.tensor([[8, 10]], device=DEV),
              level_start_index=torch.zeros(1, dtype=torch.int64, device=DEV))
    want = net(query, reference_points=ref, **kw)
    got = net(query, reference_points=_shifted(ref, floats), **kw)
    torch.testing.assert_close(got, want, rtol=1e-5, atol=1e-5)


@pytest.mark.parametrize("floats", [1, 2, 3])
@pytest.mark.parametrize("rows", [64, 16384, 16389])       # one product; 16 slices of it; 16 slices and rows left over
def test_linear_takes_unaligned_input(lib_built, floats, rows):
    torch.manual_seed(rows + floats)
    lin = layer_ops.Linear(24, 32).to(DEV)
    x = _shifted(torch.randn(rows, 24, device=DEV), floats).requires_grad_(True)
    go = torch.randn(rows, 32, device=DEV)
    got = torch.autograd.grad(lin(x), [x, lin.weight, lin.bias], go)
    want = torch.autograd.grad(F.linear(x, lin.weight, lin.bias), [x, lin.weight, lin.bias], go)
    for a, b in zip(got, want):
        torch.testing.assert_close(a, b, rtol=1e-4, atol=1e-4 * rows ** 0.5)


@pytest.mark.parametrize("floats", [1, 2, 3])
def test_linear_relu_takes_unaligned_gradient(lib_built, floats):
    torch.manual_seed(floats)
    lin = layer_ops.Linear(24, 32).to(DEV)
    x = torch.randn(65, 24, device=DEV, requires_grad=True)
    go = _shifted(torch.randn(65, 32, device=DEV), floats)
    got = torch.autograd.grad(layer_ops.linear_relu(x, lin, nn.ReLU()), [x, lin.weight, lin.bias], go)
    want = torch.autograd.grad(F.relu(F.linear(x, lin.weight, lin.bias)), [x, lin.weight, lin.bias], go)
    for a, b in zip(got, want):
        torch.testing.assert_close(a, b, rtol=1e-4, atol=1e-4)
