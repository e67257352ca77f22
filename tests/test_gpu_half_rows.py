"""Forward of bf16 and fp16 rows: every width its kernels exist for, items of 32 points, of two batches of them and of a
number that is no multiple, points outside the image, a last CTA that is partly filled.  Checked against the CPU oracle on
the rounded inputs."""
import numpy as np
import pytest
import torch

from dfa3d_b200 import workloads as wl
from helpers import FWD, assert_close, oracle_all

pytestmark = pytest.mark.gpu
DEV = "cuda"
LEVELS = ((6, 9), (4, 5), (3, 2), (1, 3), (2, 2))


@pytest.mark.parametrize("storage", ["bf16", "fp16"])
@pytest.mark.parametrize("L,P", [(4, 8), (2, 32), (5, 7)])
@pytest.mark.parametrize("C", [16, 32, 64, 128, 256])
def test_forward_matches_oracle(lib_built, C, L, P, storage):
    from dfa3d_b200 import ext
    w = wl.WORKLOADS["tiny"].with_(B=2, H=3, C=C, D=6, Q=41, levels=LEVELS[:L], P=P, seed=C + L, oob=True,
                                   value_dtype=storage)
    d = wl.make_inputs(w, head_repeat=True)
    ref = oracle_all(d, np.float32)
    dtype = torch.bfloat16 if storage == "bf16" else torch.float16
    t = {k: v.to(DEV) for k, v in d.items()}
    args = (t["value"].to(dtype), t["dist"].to(dtype), t["shapes"], t["lsi"], t["loc"], t["attn"], 64)
    out, ds = ext.dfa3d_fused_forward(*args)
    assert_close("out", out, ref["out"], **FWD)
    assert_close("depth_score", ds, ref["ds"], **FWD)
    assert_close("out only", ext.dfa3d_fused_forward(*args, False)[0], ref["out"], **FWD)
