"""Blocks of an encoder layer that a user replaces, and hooks on them: a replacement is called as it is, every hook runs."""
import pytest
import torch
import torch.nn as nn

from dfa3d_b200 import modules
from dfa3d_b200.layer_ops import Linear
from test_gpu_modules import DEV, _inputs

pytestmark = pytest.mark.gpu
KEYS = ("value", "value_dpt_dist", "reference_points_cam", "bev_mask", "spatial_shapes", "level_start_index")


def _layer():
    torch.manual_seed(2)
    return modules.BEVFormerEncoderLayer(embed_dims=32, ffn_dims=64, num_cams=3, num_heads=2, num_levels=2, num_points=8,
                                         bev_h=5, bev_w=10, dropout=0.0).to(DEV)


class _Adapter(nn.Module):
    def __init__(self, inner):
        super().__init__()
        self.inner = inner

    def forward(self, x):
        return self.inner(x) * 0.5


def _ffn(kind, ffn):
    if kind == "identity":
        return nn.Identity()
    if kind == "adapter":
        return _Adapter(ffn)
    if kind == "short":
        return nn.Sequential(Linear(32, 32), nn.ReLU())
    if kind == "other activation":
        return nn.Sequential(ffn[0], nn.GELU(), ffn[3])
    if kind == "longer":
        return nn.Sequential(*ffn, nn.Tanh())
    return nn.Sequential(nn.Linear(32, 32), nn.Tanh(), nn.Linear(32, 32), nn.Tanh(), nn.Tanh(), nn.Tanh())


@pytest.mark.parametrize("kind", ["identity", "adapter", "short", "other activation", "longer", "other layers"])
@pytest.mark.parametrize("grad", [True, False])
def test_replaced_feed_forward_is_called(lib_built, kind, grad):
    layer, d = _layer(), _inputs(6)
    layer.ffn = _ffn(kind, layer.ffn).to(DEV)
    seen = []
    layer.norm1.register_forward_hook(lambda m, a, y: seen.append(y))
    with torch.set_grad_enabled(grad):
        got = layer(d["query"], **{k: d[k] for k in KEYS})
        want = layer.norm2(layer.ffn(seen[0]), seen[0])
    torch.testing.assert_close(got, want, rtol=1e-5, atol=1e-5)


@pytest.mark.parametrize("grad", [True, False])
def test_hooks_for_all_modules_see_every_call(lib_built, grad):
    layer, d = _layer(), _inputs(7)
    want = sorted(n for n, m in layer.named_modules() if n)
    names, got = {m: n for n, m in layer.named_modules() if n}, []
    handles = [nn.modules.module.register_module_forward_hook(lambda m, a, y: got.append(names.get(m))),
               nn.modules.module.register_module_forward_pre_hook(lambda m, a: None)]
    try:
        with torch.set_grad_enabled(grad):
            layer(d["query"], **{k: d[k] for k in KEYS})
    finally:
        for h in handles:
            h.remove()
    assert sorted(n for n in got if n) == want


def test_a_forward_set_on_an_instance_is_called(lib_built):
    layer, d = _layer(), _inputs(8)
    called = []
    for name in ("ffn.0", "ffn.1", "ffn", "cross_attn.deformable_attention", "self_attn.sampling_offsets",
                 "cross_attn.deformable_attention.attention_weights"):
        m = layer.get_submodule(name)
        m.forward = lambda *a, _f=m.forward, _n=name, **kw: (called.append(_n), _f(*a, **kw))[1]
    with torch.no_grad():
        layer(d["query"], **{k: d[k] for k in KEYS})
    assert sorted(called) == sorted(["ffn.0", "ffn.1", "ffn", "cross_attn.deformable_attention", "self_attn.sampling_offsets",
                                     "cross_attn.deformable_attention.attention_weights"])


class _OtherCrossAttention(nn.Module):
    """A user's block with the layer's inputs and no more."""

    def forward(self, query, value, value_dpt_dist, reference_points_cam, bev_mask, spatial_shapes, level_start_index,
                return_residual):
        return query * 0.5, query


def test_replaced_cross_attention_gets_what_the_caller_gave(lib_built):
    layer, d = _layer(), _inputs(9)
    layer.cross_attn = _OtherCrossAttention()
    with torch.no_grad():
        assert layer(d["query"], **{k: d[k] for k in KEYS}).shape == d["query"].shape
