"""Conversion of up to two buffers between fp32 and a 16-bit type: bit-equal to torch's, at every remainder of eight, with
one buffer or two, for values that round, overflow, vanish or are not numbers; and where the operator uses it."""
import pytest
import torch

from dfa3d_b200 import _lib, functions, workloads as wl

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _values(n, seed):
    x = torch.randn(n, generator=torch.Generator().manual_seed(seed)) * 10 ** (torch.arange(n) % 12 - 6).float()
    for i, v in enumerate((float("inf"), -float("inf"), float("nan"), 70000.0, 1e-8, -0.0)):
        if i < n:
            x[i] = v
    return x.to(DEV)


@pytest.mark.parametrize("dtype,code", [(torch.float16, _lib.DTYPE_F16), (torch.bfloat16, _lib.DTYPE_BF16)])
@pytest.mark.parametrize("n0,n1", [(1, 0), (7, 9), (8, 15), (16, 3), (0, 5), (4099, 2050), (3000001, 12)])
def test_convert_two_is_bit_equal(lib_built, dtype, code, n0, n1):
    st = torch.cuda.current_stream().cuda_stream
    wide = [_values(max(n, 1), n)[:n] for n in (n0, n1)]
    narrow = [torch.zeros(max(n, 1), dtype=dtype, device=DEV)[:n] for n in (n0, n1)]
    back = [torch.zeros(max(n, 1), device=DEV)[:n] for n in (n0, n1)]
    ptr = lambda t: t.data_ptr() if t.numel() else None
    _lib.call_plain("dfa3d_convert_two", code, 0, ptr(narrow[0]), ptr(wide[0]), n0, ptr(narrow[1]), ptr(wide[1]), n1, st)
    _lib.call_plain("dfa3d_convert_two", code, 1, ptr(narrow[0]), ptr(back[0]), n0, ptr(narrow[1]), ptr(back[1]), n1, st)
    for w, n, b in zip(wide, narrow, back):
        assert torch.equal(n.nan_to_num(7.0), w.to(dtype).nan_to_num(7.0)) and torch.equal(n.isnan(), w.isnan())
        assert torch.equal(b.nan_to_num(7.0), n.float().nan_to_num(7.0))


@pytest.mark.parametrize("value_grad,dist_grad", [(True, True), (True, False), (False, True)])
def test_gradients_arrive_in_their_inputs_types(lib_built, value_grad, dist_grad):
    d = {k: v.to(DEV) for k, v in wl.make_inputs(wl.WORKLOADS["odd"]).items()}
    value, dist = d["value"].half().requires_grad_(value_grad), d["dist"].half().requires_grad_(dist_grad)
    attn = d["attn"].requires_grad_(True)
    out, ds = functions.MultiScale3DDeformableAttnFunction_fp16.apply(value, dist, d["shapes"], d["lsi"], d["loc"], attn, 64)
    assert out.dtype == ds.dtype == torch.float16
    leaves = [t for t in (value, dist, attn) if t.requires_grad]
    for grad_out in (d["grad_out"].half(), d["grad_out"].half().transpose(0, 1).contiguous().transpose(0, 1)):
        for t, g in zip(leaves, torch.autograd.grad(out, leaves, grad_out, retain_graph=True)):
            assert g.dtype == t.dtype and g.shape == t.shape and bool(g.isfinite().all())
