"""An expert bank's down rows side by side in a warp: the bits of the partial sums that more slots than a warp holds take. GPU only (-m gpu)."""
import numpy as np
import pytest

from tests import oracle_lib as ol
from tests.test_gpu_moe import cuda, make_bank

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("t", [ol.Q4_K, ol.Q6_K, ol.Q8_0, ol.Q4_0])
@pytest.mark.parametrize("hidden,ffn,top,tokens", [(256, 256, 1, 1), (512, 256, 8, 3), (256, 512, 2, 5), (768, 512, 8, 2), (256, 768, 3, 1), (256, 768, 4, 3), (512, 1024, 4, 2), (256, 1024, 3, 1),
                                                   (256, 1536, 2, 2), (256, 2048, 2, 1), (256, 1792, 1, 2)])
@pytest.mark.parametrize("with_shared", [False, True])
def test_the_warps_sums_are_the_partial_sums(rq_ctx, oracle, t, hidden, ffn, top, tokens, with_shared):
    import torch

    experts = 10
    gate, up, down, shared = make_bank(oracle, t, experts, hidden, ffn, 51)
    bank = rq_ctx.moe_prepare(t, gate, up, down, experts, hidden, ffn, shared=shared if with_shared else None)
    x = oracle.normal(51, 8, hidden * tokens, 1.0).reshape(hidden, tokens)
    x[:, 0] *= np.where(np.arange(hidden) % 37 == 0, 3000.0, 1.0)  # inputs far apart: h has groups whose largest stay out of the digits
    weights = np.zeros((experts, tokens), np.float32)
    for i in range(tokens):
        at = (3 * i + 2 * np.arange(top)) % experts if top <= 5 else np.arange(i, i + top) % experts
        weights[at, i] = np.linspace(0.1, 1.0, top)
    if tokens > 1:
        weights[:, -1] = 0.0  # a token nobody is routed to
    xd, wd = cuda(x), cuda(weights)
    y = rq_ctx.moe_forward(bank, xd, wd, top)
    # more slots spoken for than a warp holds: from two units a sub-row on the partial sums
    lanes = 1 << (ffn // 256 - 1).bit_length()
    many = rq_ctx.moe_forward(bank, xd, wd, min(15, max(top, 16 // lanes) + 1))
    assert not torch.isnan(y).any() and torch.equal(y, many)
    if tokens > 1 and not with_shared:
        assert (y[:, -1] == 0).all()
    strided = torch.full((tokens, hidden + 5), float("nan"), device="cuda")
    rq_ctx.moe_forward(bank, xd, wd, top, y=strided[:, :hidden].T)
    assert torch.equal(strided[:, :hidden].T, y) and torch.isnan(strided[:, hidden:]).all()
    rq_ctx.check()


def routed(experts, top, tokens):
    """Weights of `top` neighbouring experts a token, the last token's none."""
    weights = np.zeros((experts, tokens), np.float32)
    for i in range(tokens - 1):
        weights[(3 * i + np.arange(top)) % experts, i] = np.linspace(0.1, 1.0, top)
    return weights


# Rows enough for several stages a CTA (296 CTAs, shared by the tokens): a stage is one or two passes of the seven warps, with two a thread takes two rows and the
# second pass is a piece of its own. `first`, `rest`: rows of a pass; of the last stage of most CTAs, once the whole ones are taken off.
@pytest.mark.parametrize("t", [ol.Q4_K, ol.Q6_K, ol.Q8_0, ol.Q4_0])
@pytest.mark.parametrize("hidden,ffn,top,tokens,first,rest", [
    (2048, 512, 8, 16, 7, (1, 2)),     # two rows a thread over Q4_K and Q4_0, the last stage inside its first piece; a row a thread, one row past whole passes, elsewhere
    (2304, 512, 8, 17, 7, (9, 10)),    # the last stage ends in its second piece
    (2048, 768, 2, 17, 14, (8, 9)),    # two rows a thread in every format: 120 or 121 of stages of 28
    (2048, 1024, 4, 32, 7, (3, 4)),
])
def test_many_stages_of_rows_are_the_partial_sums(rq_ctx, oracle, t, hidden, ffn, top, tokens, first, rest):
    import torch

    ctas = 2 * torch.cuda.get_device_properties(0).multi_processor_count // tokens
    lanes = 1 << (ffn // 256 - 1).bit_length()
    assert first == 7 * (16 // (lanes * top)) and hidden // ctas > 4 * first
    assert {hidden // ctas % (2 * first), -(-hidden // ctas) % (2 * first)} == set(rest)
    experts = 10
    gate, up, down, _ = make_bank(oracle, t, experts, hidden, ffn, 52)
    bank = rq_ctx.moe_prepare(t, gate, up, down, experts, hidden, ffn)
    xd, wd = cuda(oracle.normal(52, 8, hidden * tokens, 1.0).reshape(hidden, tokens)), cuda(routed(experts, top, tokens))
    y = rq_ctx.moe_forward(bank, xd, wd, top)
    many = rq_ctx.moe_forward(bank, xd, wd, 16 // lanes + 1)
    assert not torch.isnan(y).any() and torch.equal(y, many) and (y[:, -1] == 0).all()
    strided = torch.full((tokens, hidden + 5), float("nan"), device="cuda")
    rq_ctx.moe_forward(bank, xd, wd, top, y=strided[:, :hidden].T)
    assert torch.equal(strided[:, :hidden].T, y) and torch.isnan(strided[:, hidden:]).all()
    rq_ctx.check()


@pytest.mark.parametrize("t", [ol.Q4_K, ol.Q6_K, ol.Q8_0, ol.Q4_0])
@pytest.mark.parametrize("hidden,tokens", [(256, 9), (256, 12), (2048, 16), (2304, 5)])
def test_slots_of_one_unit(rq_ctx, oracle, t, hidden, tokens):
    """Fifteen of them fit a warp: against partial sums where those are taken for nine slots (8 to 12 rows a CTA), and against the slots one by one everywhere."""
    import torch

    experts, ffn, top = 10, 256, 8
    gate, up, down, _ = make_bank(oracle, t, experts, hidden, ffn, 53)
    bank = rq_ctx.moe_prepare(t, gate, up, down, experts, hidden, ffn)
    weights = routed(experts, top, tokens)
    xd, wd = cuda(oracle.normal(53, 8, hidden * tokens, 1.0).reshape(hidden, tokens)), cuda(weights)
    y = rq_ctx.moe_forward(bank, xd, wd, top)
    ctas = 2 * torch.cuda.get_device_properties(0).multi_processor_count // tokens
    if 8 <= -(-hidden // ctas) <= 12:
        assert torch.equal(y, rq_ctx.moe_forward(bank, xd, wd, top + 1))
    total, size = torch.zeros((hidden, tokens), dtype=torch.float64, device="cuda"), torch.zeros((hidden, tokens), dtype=torch.float64, device="cuda")
    for e in range(experts):
        one = np.zeros_like(weights)
        one[e] = weights[e] != 0
        term = rq_ctx.moe_forward(bank, xd, cuda(one), 1).double() * wd[e].double()
        total += term
        size += term.abs()
    # a chain of `top` multiply-adds, each rounded once: no partial sum is larger than the sum of the terms' sizes
    assert ((y.double() - total).abs() <= top * 2.0**-24 * size * (1 + 2.0**-20)).all()
    rq_ctx.check()
