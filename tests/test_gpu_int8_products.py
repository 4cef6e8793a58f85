"""Int8 activations over Q8_0 / Q4_0, more than 64 tokens: products of bytes, at the edges of row tiles (256), token tiles (64), units and half
units (256, 128 inputs) and of the ring of scales, in both activation steps. GPU only (-m gpu)."""
import pytest

from tests import oracle_lib as ol

pytestmark = pytest.mark.gpu


def _rounded(x, step):
    """int8 codes times their steps, fp32 arithmetic as the format defines it, in 64 bits (a last group may be short, a group may be zeros)."""
    import torch

    parts = []
    for g in x.split(step, dim=1):
        best = g.gather(1, g.abs().argmax(1, keepdim=True))
        inverse = torch.where(best == 0, 0.0, torch.full_like(best, -127.0) / best)
        d = torch.where(best == 0, 0.0, torch.ones_like(inverse) / inverse)
        parts.append(torch.round(g * inverse).clamp(-128, 127).double() * d.double())
    return torch.cat(parts, 1)


@pytest.mark.parametrize("t", [ol.Q8_0, ol.Q4_0])
@pytest.mark.parametrize("rows,cols,tokens", [(1, 32, 65), (127, 96, 66), (128, 128, 127), (129, 160, 128), (255, 256, 129), (257, 288, 191), (256, 512, 192), (300, 1120, 65), (513, 2304, 257),
                                              (5000, 768, 100), (40, 4352, 130), (19000, 256, 70)])
@pytest.mark.parametrize("step", [32, 256])
def test_sums_lose_no_more_than_their_additions(rq_ctx, t, rows, cols, tokens, step):
    import torch

    gen = torch.Generator(device="cuda").manual_seed(rows + cols + t)
    w32 = 0.02 * torch.randn(rows * cols, generator=gen, device="cuda")
    w32[: min(64, rows * cols)] = 0.3  # a block of one value: the largest code in every place
    w = rq_ctx.weight_from_device(t, rq_ctx.quantize(t, w32), rows, cols)
    dense = rq_ctx.dequant(w).reshape(rows, cols).double()
    x = torch.randn((tokens, cols), generator=gen, device="cuda")
    x[0] = 1.0  # the largest code in every place
    x[-1] = 0.0
    coded = _rounded(x, step)
    y = torch.full((tokens, rows), float("nan"), device="cuda")
    rq_ctx.matmul(w, x, y=y, act_mode=1, step=step)
    # Each group's sum is exact; its two scales' product and the multiply-add round once each, a run of at most eight groups is added up in a chain
    # whose rounding is within 2^-24 of what it has added so far, and totals carry what they round off: (2 + 8 + 2) * 2^-24 of the terms' magnitudes
    # (those of single products bound a group's).
    bound = 12 * 2.0**-24 * (coded.abs() @ dense.abs().T) + 1e-30
    assert not torch.isnan(y).any()
    assert ((y.double() - coded @ dense.T).abs() <= bound).all()
    strided = torch.full((tokens, rows + 3), float("nan"), device="cuda")
    rq_ctx.matmul(w, x, y=strided[:, :rows], act_mode=1, step=step)
    assert torch.equal(strided[:, :rows], y) and torch.isnan(strided[:, rows:]).all()
    rq_ctx.check()
