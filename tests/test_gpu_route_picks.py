"""Routing by one warp: at the edges of what it takes (experts, kept experts), with NaNs (not its case), and over a plane of its own. GPU only (-m gpu)."""
import numpy as np
import pytest

from tests import oracle_lib as ol
from tests.test_gpu_moe import cuda, make_bank

pytestmark = pytest.mark.gpu


def same(got, want):
    """The same bits, and a NaN (0 / 0: its payload is the processor's) where there is one."""
    nan = np.isnan(want)
    return np.array_equal(np.isnan(got), nan) and np.array_equal(got[~nan].view(np.uint32), want[~nan].view(np.uint32))


@pytest.mark.parametrize("experts,top", [(1, 1), (3, 3), (31, 8), (33, 32), (40, 33), (255, 8), (256, 32), (257, 8), (1023, 5), (1024, 32), (1025, 8)])
@pytest.mark.parametrize("scoring", [0, 1])
def test_bits_at_the_edges(rq_ctx, oracle, experts, top, scoring):
    import torch

    rng = np.random.default_rng(experts + top)
    scores = rng.normal(size=(experts, 6)).astype(np.float32)
    scores[:, 1] = np.float32(rng.integers(-2, 3, size=experts))  # ties
    scores[:, 2] = np.where(rng.random(experts) < 0.5, np.float32(0.0), np.float32(-0.0))
    scores[:, 3] = rng.permutation(experts).astype(np.float32) * -1e30
    if scoring == 1:
        scores[rng.integers(0, experts), 4] = np.inf
        scores[rng.integers(0, experts), 5] = -np.inf
    want = oracle.topk(scores, top, scoring, True)
    got = rq_ctx.moe_route(cuda(scores), top, scoring, True).cpu().numpy()
    assert same(got, want)
    plane = cuda(scores)  # scores and weights in one plane
    rq_ctx.lib.rq_moe_route(rq_ctx.handle, plane.data_ptr(), plane.stride(0), plane.stride(1), experts, top, scoring, 1, None, 6, plane.data_ptr(), plane.stride(0), plane.stride(1),
                            torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    assert same(plane.cpu().numpy(), want)
    rq_ctx.check()


def test_a_token_with_a_nan_takes_the_ordered_path(rq_ctx, oracle):
    rng = np.random.default_rng(5)
    scores = rng.normal(size=(64, 3)).astype(np.float32)
    scores[7, 1] = np.nan
    want = oracle.topk(scores, 6, 1, True)
    got = rq_ctx.moe_route(cuda(scores), 6, 1, True).cpu().numpy()
    assert same(got, want)


@pytest.mark.parametrize("first,count", [(0, 16), (4, 8), (12, 4)])
def test_a_ranks_experts_take_their_slots(rq_ctx, oracle, first, count):
    """Routing and planning in one launch, over some of the experts and with the shared one: the bits of the two calls."""
    import torch

    t, experts, top, hidden, ffn, tokens = ol.Q4_K, 16, 5, 512, 256, 4
    gate, up, down, shared = make_bank(oracle, t, experts, hidden, ffn, 61)
    for with_shared in (False, True):
        bank = rq_ctx.moe_prepare(t, gate, up, down, experts, hidden, ffn, expert_first=first, expert_count=count, shared=shared if with_shared else None)
        x, scores = cuda(oracle.normal(61, 8, hidden * tokens, 1.0).reshape(hidden, tokens)), cuda(oracle.normal(61, 9, experts * tokens, 1.0).reshape(experts, tokens))
        routing = rq_ctx.moe_route(scores, top)
        two = rq_ctx.moe_forward(bank, x, routing, top)
        one, weights = rq_ctx.moe_route_forward(bank, scores, x, top)
        assert torch.equal(weights, routing) and torch.equal(one, two)
    rq_ctx.check()


@pytest.mark.parametrize("experts,top", [(8, 8), (16, 10), (16, 11), (32, 13), (32, 14), (32, 32), (64, 18), (64, 19), (128, 29), (128, 30), (143, 31), (143, 32), (144, 32)])
@pytest.mark.parametrize("scoring", [0, 1])
def test_bits_on_both_sides_of_the_rule(rq_ctx, oracle, experts, top, scoring):
    """One warp picks up to 8 + experts / 6; beyond, every thread counts its expert's place."""
    rng = np.random.default_rng(experts + top)
    scores = rng.normal(size=(experts, 3)).astype(np.float32)
    scores[:, 1] = np.float32(rng.integers(-2, 3, size=experts))  # ties
    assert same(rq_ctx.moe_route(cuda(scores), top, scoring, True).cpu().numpy(), oracle.topk(scores, top, scoring, True))
    rq_ctx.check()
