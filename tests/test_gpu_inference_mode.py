"""Serving under torch.inference_mode(), whose tensors have no version counter and cannot be saved for a backward: the
encoder modules give what they give under no_grad, and what they keep from such a pass serves a training pass after it."""
import pytest
import torch

from dfa3d_b200 import modules
from test_gpu_modules import DEV, _inputs

pytestmark = pytest.mark.gpu


def _keywords(d):
    return {k: d[k] for k in ("value", "value_dpt_dist", "reference_points_cam", "bev_mask", "spatial_shapes",
                              "level_start_index")}


def _stack():
    torch.manual_seed(0)
    return modules.SCAEncoderStack(num_layers=2, embed_dims=32, ffn_dims=64, num_cams=3, num_heads=2, num_levels=2,
                                   num_points=8, dropout=0.0).to(DEV)


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16])
def test_reference_points_made_inside_inference_mode(lib_built, dtype):
    stack, d = _stack(), _inputs(3)
    d["reference_points_cam"] = d["reference_points_cam"].to(dtype)
    with torch.no_grad():
        want = stack(d["query"], **_keywords(d))
    with torch.inference_mode():
        d["reference_points_cam"] = d["reference_points_cam"] + 0        # as point_sampling makes them: an inference tensor
        got = stack(d["query"], **_keywords(d))
    assert torch.equal(got, want)


def test_reference_points_are_read_in_every_pass(lib_built):
    """A plan that the caller keeps holds nothing of the reference points, however they are written."""
    from dfa3d_b200.rebatch import RebatchPlan
    stack, d = _stack(), _inputs(4)
    kw = dict(_keywords(d), rebatch_plan=RebatchPlan(d["bev_mask"]))
    with torch.no_grad():
        stack(d["query"], **kw)
        d["reference_points_cam"].data.mul_(0.5)                         # no version counter moves
        got = stack(d["query"], **kw)
        want = stack(d["query"], **dict(kw, reference_points_cam=d["reference_points_cam"].clone()))
    assert torch.equal(got, want)


def _full_layer():
    torch.manual_seed(1)
    return modules.BEVFormerEncoderLayer(embed_dims=32, ffn_dims=64, num_cams=3, num_heads=2, num_levels=2, num_points=8,
                                         bev_h=5, bev_w=10, dropout=0.0).to(DEV)


def test_layer_trains_after_it_has_served(lib_built):
    layer, d = _full_layer(), _inputs(5)
    with torch.inference_mode():
        served = layer(d["query"], **_keywords(d)).clone()
    out = layer(d["query"].requires_grad_(True), **_keywords(d))
    assert torch.equal(out, served)
    out.sum().backward()
    assert all(torch.isfinite(p.grad).all() for p in layer.parameters())


def test_layer_saved_after_a_pass_runs_where_it_is_loaded(lib_built, tmp_path):
    layer, d = _full_layer(), _inputs(6)
    with torch.no_grad():
        want = layer(d["query"], **_keywords(d))
        torch.save(layer, tmp_path / "layer.pt")
        loaded = torch.load(tmp_path / "layer.pt", map_location="cpu", weights_only=False).to(DEV)
        assert torch.equal(loaded(d["query"], **_keywords(d)), want)
        layer.bev_h, layer.bev_w = 10, 5                                     # another size of the same layer
        other = layer(d["query"], **_keywords(d))
        layer.bev_h, layer.bev_w = 5, 10
        assert torch.equal(layer(d["query"], **_keywords(d)), want) and not torch.equal(other, want)
