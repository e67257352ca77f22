"""Layer operations exist twice, natively and as the Python Functions that autocast, double precision and unusual layouts go
to.  Both give the same results and gradients, on both sides of every rule that they share."""
import pytest
import torch

from dfa3d_b200 import _lib, layer_ops
from dfa3d_b200.dist_producer import DepthDistributionFunction
from dfa3d_b200.layer_ops import AddLayerNormFunction, LinearFunction
from dfa3d_b200.rebatch import CombineCamerasFunction, GatherQueriesFunction, RebatchPlan
from test_gpu_native_path import _python

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _randn(*shape, seed):
    return torch.randn(*shape, generator=torch.Generator().manual_seed(seed)).to(DEV)


def _arguments(kind, size):
    """Function, its arguments; tensors of floating point are leaves."""
    if kind == "linear":
        return LinearFunction, [_randn(size, 40, seed=1), _randn(64, 40, seed=2), _randn(64, seed=3)]
    if kind == "norm":
        return AddLayerNormFunction, [_randn(size, 132, seed=1), _randn(size, 132, seed=2), _randn(132, seed=3),
                                      _randn(132, seed=4), 1e-5]
    if kind == "norm without residual":
        return AddLayerNormFunction, [_randn(size, 132, seed=1), None, _randn(132, seed=3), _randn(132, seed=4), 1e-5]
    if kind == "dist":
        levels = torch.tensor([[8, 2 * size], [4, size]])
        lsi = torch.tensor([0, 16 * size])
        return DepthDistributionFunction, [_randn(2, 19, 4, size, seed=1), levels.to(DEV), lsi.to(DEV), 20 * size]
    mask = torch.rand(3, 2, size, 4, generator=torch.Generator().manual_seed(5)) < 0.2
    plan = RebatchPlan(mask.to(DEV))
    if kind == "gather":
        return GatherQueriesFunction, [_randn(2, size, 33, seed=1), plan]
    return CombineCamerasFunction, [_randn(2 * plan.rows, 64, seed=1), plan]


@pytest.mark.parametrize("kind,size", [("linear", 7), ("linear", 16383), ("linear", 16384), ("linear", 16399), ("norm", 1),
                                       ("norm", 77), ("norm without residual", 77), ("dist", 7), ("dist", 33), ("gather", 1),
                                       ("gather", 401), ("combine", 401)])
def test_native_layer_operation_equals_the_python_function(lib_built, kind, size):
    fn, args = _arguments(kind, size)
    results = []
    for f in (fn, _python(fn)):
        a = [t.clone().requires_grad_(True) if torch.is_tensor(t) and t.is_floating_point() else t for t in args]
        out = f.apply(*a)
        leaves = [t for t in a if torch.is_tensor(t) and t.requires_grad]
        results.append((out, torch.autograd.grad(out, leaves, _randn(*out.shape, seed=9))))
    (o0, g0), (o1, g1) = results
    assert type(o0.grad_fn).__name__ != type(o1.grad_fn).__name__          # two different implementations
    assert torch.equal(o0, o1)                                             # the same kernels and products
    for a, b in zip(g0, g1):
        # sums over `size` rows of float32 in another order: 2^-24 times the square root of their number, and a factor of 8
        tol = 8 * 2.0 ** -24 * max(size, 16) ** 0.5
        assert a.dtype == b.dtype and a.shape == b.shape
        assert float((a - b).abs().max()) <= tol * float(b.abs().max())


def test_both_split_the_weight_gradient_alike(lib_built):
    native = _lib.native()
    assert (native.split_rows, native.splits) == (layer_ops._SPLIT_ROWS, layer_ops._SPLITS)
