"""Kernels in which a warp takes several items of up to 16 points: point counts below, at and between the lane counts
4, 8 and 16, last warps that are partly filled, every storage type and width, small launches (whose items have 16 lanes) and
fp32 ones of two batches per warp, with and without depth scores, one- and two-stage, per-camera query counts.  Checked
against the CPU oracle.  (test_gpu_full_launches.py: the other lane counts.)"""
import numpy as np
import pytest
import torch

from dfa3d_b200 import workloads as wl
from helpers import BWD, FWD, assert_close, oracle_all

pytestmark = pytest.mark.gpu
DEV = "cuda"
LEVELS = ((6, 9), (4, 5), (3, 2), (1, 3), (2, 2))
STORAGE = {"fp32": (torch.float32, torch.float32), "bf16": (torch.bfloat16, torch.bfloat16),
           "fp16": (torch.float16, torch.float16), "fp32_bf16": (torch.float32, torch.bfloat16),
           "bf16_fp32": (torch.bfloat16, torch.float32)}


@pytest.mark.parametrize("Q", [37, 9001])            # 9001 x 3 cameras x 3 heads of 8 lanes: two batches per warp in some kernels
@pytest.mark.parametrize("storage", sorted(STORAGE))
@pytest.mark.parametrize("L,P,C", [(1, 1, 16), (1, 2, 64), (1, 3, 32), (1, 4, 32), (1, 5, 16), (2, 3, 32), (1, 7, 64),
                                   (2, 4, 32), (3, 3, 64), (2, 5, 32), (3, 4, 16), (5, 3, 32), (4, 4, 64)])
def test_every_point_count_matches_oracle(lib_built, L, P, C, storage, Q):
    from dfa3d_b200 import ext
    if Q > 100 and (storage.endswith("2_bf16") or storage == "bf16_fp32" or C == 64):
        Q = 301
    vt, dt = STORAGE[storage]
    w = wl.WORKLOADS["tiny"].with_(B=3, H=3, C=C, D=6, Q=Q, levels=LEVELS[:L], P=P, seed=L * 100 + P,
                                   value_dtype="fp32" if storage == "fp32" else "fp16" if storage == "fp16" else "bf16")
    d = wl.make_inputs(w, head_repeat=True)
    ref = oracle_all(d, np.float32)
    t = {k: v.to(DEV) for k, v in d.items()}
    value, dist, loc, attn = t["value"].to(vt), t["dist"].to(dt), t["loc"], t["attn"]
    args = (value, dist, t["shapes"], t["lsi"], loc, attn)
    out, ds = ext.dfa3d_fused_forward(*args, 64)
    assert_close("out", out, ref["out"], **FWD)
    assert_close("depth_score", ds, ref["ds"], **FWD)
    assert_close("out only", ext.dfa3d_fused_forward(*args, 64, False)[0], ref["out"], **FWD)
    shapes2, loc2 = t["shapes"][:, :2].contiguous(), loc[..., :2].contiguous()
    two = ext.wms_deform_attn_forward(value, shapes2, t["lsi"], loc2, attn, ds, 64)
    assert_close("two-stage out", two, ref["out"], **FWD)
    gv = torch.zeros_like(t["value"]); gd = torch.zeros_like(t["dist"])
    gl = torch.empty_like(loc); ga = torch.empty_like(attn)
    ext.dfa3d_fused_backward(*args, t["grad_out"], gv, gd, gl, ga, 64)
    for k, x in (("grad_value", gv), ("grad_dist", gd), ("grad_loc", gl), ("grad_attn", ga)):
        assert_close(k, x, ref[k], **BWD)
    # the same items as rows of cameras that have different numbers of queries
    counts = torch.tensor([Q, 0, Q // 2])
    offsets = torch.cat([torch.zeros(1, dtype=torch.int64), counts.cumsum(0)]).int().to(DEV)
    rows = lambda x: torch.cat([x[b, :int(n)] for b, n in enumerate(counts)]).contiguous()
    got = ext.dfa3d_fused_forward_ragged(value, dist, t["shapes"], t["lsi"], rows(loc), rows(attn), offsets, Q)[0]
    assert_close("ragged out", got, rows(torch.from_numpy(ref["out"])), **FWD)
