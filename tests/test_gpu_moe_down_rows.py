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
