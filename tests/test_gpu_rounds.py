"""CTAs that walk several groups of items, and items that get more lanes in a small launch: launches of a few groups, of some
waves of CTAs and of sizes in between, item counts that do not fill the last group, with one item and with several items
per warp, and cameras of different numbers of queries.  Checked against the CPU oracle."""
import numpy as np
import pytest
import torch

from dfa3d_b200 import workloads as wl
from helpers import BWD, FWD, assert_close, oracle_all

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("Q", [7, 211, 803, 2401])
@pytest.mark.parametrize("P,C", [(17, 8), (3, 16), (2, 64), (4, 32), (7, 64), (8, 32)])
def test_every_item_is_walked(lib_built, P, C, Q):
    from dfa3d_b200 import ext
    w = wl.WORKLOADS["tiny"].with_(B=5, H=7, C=C, D=6, Q=Q, levels=((6, 9),), P=P, seed=Q + P)
    d = wl.make_inputs(w, head_repeat=True)
    ref = oracle_all(d, np.float32)
    t = {k: v.to(DEV) for k, v in d.items()}
    args = (t["value"], t["dist"], t["shapes"], t["lsi"], t["loc"], t["attn"])
    out, ds = ext.dfa3d_fused_forward(*args, 64)
    assert_close("out", out, ref["out"], **FWD)
    assert_close("depth_score", ds, ref["ds"], **FWD)
    gv = torch.zeros_like(t["value"]); gd = torch.zeros_like(t["dist"])
    gl = torch.full_like(t["loc"], float("nan")); ga = torch.full_like(t["attn"], float("nan"))
    ext.dfa3d_fused_backward(*args, t["grad_out"], gv, gd, gl, ga, 64)
    for k, x in (("grad_value", gv), ("grad_dist", gd), ("grad_loc", gl), ("grad_attn", ga)):
        assert_close(k, x, ref[k], **BWD)
    counts = torch.tensor([Q, 0, Q // 3, 1, Q - 1])
    offsets = torch.cat([torch.zeros(1, dtype=torch.int64), counts.cumsum(0)]).int().to(DEV)
    rows = lambda x: torch.cat([x[b, :int(n)] for b, n in enumerate(counts)]).contiguous()
    got = ext.dfa3d_fused_forward_ragged(*args[:4], rows(t["loc"]), rows(t["attn"]), offsets, Q)[0]
    assert_close("ragged out", got, rows(torch.from_numpy(ref["out"])), **FWD)
