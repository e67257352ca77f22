"""The layer operations of the native host path against the separate steps they stand for: joint and ReLU Linear layers
(also with rows that no slice of the weight gradient covers), norms without a backward, and 2-D attention from offsets and
logits at every size its kernels exist for."""
import pytest
import torch
import torch.nn as nn
import torch.nn.functional as F

from dfa3d_b200 import functions, layer_ops, modules
from dfa3d_b200.layer_ops import Linear

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _close(got, want, rtol=2e-4):
    for a, b in zip(got, want):
        assert a.shape == b.shape
        scale = float(b.abs().max()) + 1e-30
        assert float((a - b).abs().max()) <= rtol * scale


def _grads(out, leaves, seed=3):
    g = torch.randn(out.shape, generator=torch.Generator().manual_seed(seed)).to(DEV)
    return torch.autograd.grad(out, leaves, g)


@pytest.mark.parametrize("rows", [1, 33, 16384, 16399])      # around the split of the weight gradient: 0 and 15 rows over
@pytest.mark.parametrize("outs", [(8, 4), (64, 32, 32)])
def test_joint_linear_equals_the_layers_one_by_one(lib_built, rows, outs):
    torch.manual_seed(rows)
    layers = [Linear(40, o).to(DEV) for o in outs]
    x = torch.randn(rows, 40, device=DEV, requires_grad=True)
    leaves = [x] + [p for m in layers for p in (m.weight, m.bias)]
    got = layer_ops.joint_linear(x, *layers)
    want = torch.cat([F.linear(x.double(), m.weight.double(), m.bias.double()) for m in layers], -1)
    _close([got], [want.float()])
    _close(_grads(got, leaves), [t.float() for t in _grads(want, leaves)])
    layers[0].register_forward_hook(lambda *a: None)          # a hook wants its layer to be called
    assert layer_ops.joint_linear(x, *layers) is None
    with torch.autocast("cuda"):
        assert layer_ops.joint_linear(x, *[Linear(40, 8).to(DEV) for _ in range(2)]) is None


@pytest.mark.parametrize("rows", [7, 16401])
def test_linear_relu_equals_linear_then_relu(lib_built, rows):
    torch.manual_seed(rows)
    lin = Linear(24, 260).to(DEV)
    x = torch.randn(2, rows, 24, device=DEV, requires_grad=True)
    leaves = [x, lin.weight, lin.bias]
    got = layer_ops.linear_relu(x, lin, nn.ReLU())
    want = F.relu(F.linear(x.double(), lin.weight.double(), lin.bias.double()))
    _close([got], [want.float()])
    _close(_grads(got, leaves), [t.float() for t in _grads(want, leaves)])


@pytest.mark.parametrize("with_residual", [True, False])
def test_norm_without_backward_equals_the_one_with(lib_built, with_residual):
    torch.manual_seed(0)
    norm = layer_ops.AddLayerNorm(132).to(DEV)
    x, r = torch.randn(2, 55, 132, device=DEV)
    want = norm(x, r if with_residual else None)
    with torch.no_grad():
        got = norm(x, r if with_residual else None)
    assert want.requires_grad and not got.requires_grad and torch.equal(got, want)


@pytest.mark.parametrize("maps,L,P,C", [(2, 1, 4, 32), (1, 1, 4, 16), (1, 4, 4, 32), (2, 2, 4, 16), (2, 1, 2, 64), (1, 2, 4, 64),
                                        (4, 1, 4, 32), (1, 1, 16, 32)])
def test_attention_2d_from_offsets_equals_the_steps(lib_built, maps, L, P, C):
    """Softmax map by map, location assembly, operator, mean over the maps -- one step after the other -- against the
    kernels that do all of it; some points outside the maps; an item count that does not fill the last warp."""
    g = torch.Generator().manual_seed(maps * 100 + L * 10 + P)
    bs, Q, H = 2, 37, 3
    levels = [(9, 7), (5, 4), (3, 3), (2, 2)][:L]
    shapes = torch.tensor(levels)
    hw = shapes.prod(1)
    lsi = torch.cat([hw.new_zeros(1), hw.cumsum(0)[:-1]]).to(DEV)
    N = int(hw.sum())
    shapes = shapes.to(DEV)
    value = torch.randn(bs * maps, N, H * C, generator=g).to(DEV).requires_grad_(True)
    joint = torch.randn(bs, Q, H * maps * L * P * 3, generator=g).to(DEV).requires_grad_(True)
    ref = torch.rand(bs * maps, Q, L, 2, generator=g).to(DEV)
    got = functions.MultiScaleDeformableAttnFunction_fp32.from_offsets(value, shapes, lsi, ref, joint, maps, H, P)
    assert got is not NotImplemented
    n = H * maps * L * P
    att = modules.TemporalSelfAttention(H * C, H, L, P, num_bev_queue=maps)
    want = att._attention_in_steps(value.view(bs * maps, N, H, C), joint[..., :2 * n], joint[..., 2 * n:], ref, shapes, lsi)
    _close([got], [want], 1e-5)
    _close(_grads(got, [value, joint]), _grads(want, [value, joint]), 2e-5)
    bare = functions.MultiScaleDeformableAttnFunction_fp32.from_offsets(value.detach(), shapes, lsi, ref, joint.detach(),
                                                                        maps, H, P)
    assert torch.equal(bare, got)


def test_attention_2d_from_offsets_leaves_other_sizes_alone(lib_built):
    fused = functions.MultiScaleDeformableAttnFunction_fp32.from_offsets
    shapes, lsi = torch.tensor([[4, 4]], device=DEV), torch.zeros(1, dtype=torch.int64, device=DEV)
    for P, C in ((3, 32), (32, 32), (4, 24)):
        out = fused(torch.zeros(1, 16, C, device=DEV), shapes, lsi, torch.zeros(1, 5, 1, 2, device=DEV),
                    torch.zeros(1, 5, P * 3, device=DEV), 1, 1, P)
        assert out is NotImplemented


@pytest.mark.parametrize("bs,step,accepted", [(3, 4, False), (3, 2, True), (3, 64, True), (2, 3, False), (1, 0, False)])
def test_attention_2d_refuses_a_batch_that_im2col_step_does_not_divide(lib_built, bs, step, accepted):
    """The step has no use here but the reference's check on it; the joint form makes it like the separate one."""
    att = modules.TemporalSelfAttention(64, 4, 1, 4, im2col_step=step, dropout=0.0).to(DEV)
    query, value = torch.randn(bs, 12, 64, device=DEV), torch.randn(2 * bs, 12, 64, device=DEV)
    kw = dict(value=value, reference_points=torch.rand(2 * bs, 12, 1, 2, device=DEV),
              spatial_shapes=torch.tensor([[3, 4]], device=DEV), level_start_index=torch.zeros(1, dtype=torch.int64, device=DEV))
    if accepted:
        assert att(query, **kw).shape == query.shape
    else:
        with pytest.raises(RuntimeError, match="must divide im2col_step"):
            att(query, **kw)
