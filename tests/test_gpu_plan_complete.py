"""A re-batching plan that its constructor has returned is complete: for other streams, for a CUDA graph that is captured
with it, and for copies of it."""
import copy
import io

import pytest
import torch

from dfa3d_b200.rebatch import CombineCamerasFunction, GatherQueriesFunction, RebatchPlan, gather_per_camera

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _mask(seed):
    return (torch.rand(3, 2, 401, 4, generator=torch.Generator().manual_seed(seed)) < 0.2).to(DEV)


def _expected(mask):
    return 1.0 / mask.any(-1).sum(0).clamp(min=1).float()


def test_plan_of_another_stream(lib_built):
    mask = _mask(0)
    want = _expected(mask)
    RebatchPlan(mask)                                              # memory and kernels are there
    torch.cuda.synchronize()
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        torch.cuda._sleep(20_000_000)                              # some 10 ms
        plan = RebatchPlan(mask)
    got = plan.inv_count.clone()                                   # on the default stream
    counts = plan.counts.clone()
    torch.cuda.synchronize()
    assert torch.equal(got, want) and counts.tolist() == mask[:, 0].any(-1).sum(-1).tolist()


def test_plan_in_a_captured_graph(lib_built):
    src = torch.randn(2, 401, 64, device=DEV)

    def work(plan):
        return CombineCamerasFunction.apply(GatherQueriesFunction.apply(src, plan), plan)

    work(RebatchPlan(_mask(1)))                                    # warm-up on another frame's plan
    plan = RebatchPlan(_mask(2))
    graph = torch.cuda.CUDAGraph()
    with torch.no_grad(), torch.cuda.graph(graph):
        out = work(plan)
    src.mul_(2)
    graph.replay()
    assert torch.equal(out, work(plan))


def test_plan_can_be_copied_and_saved(lib_built):
    plan, src = RebatchPlan(_mask(3)), torch.randn(3, 2, 401, 4, 3, device=DEV)
    buf = io.BytesIO()
    torch.save(plan, buf)
    buf.seek(0)
    for other in (copy.deepcopy(plan), torch.load(buf, weights_only=False)):
        assert (other.rows, other.max_queries) == (plan.rows, plan.max_queries)
        assert torch.equal(gather_per_camera(src, other), gather_per_camera(src, plan))
