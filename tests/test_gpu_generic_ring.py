"""The decode-only formats' matvec with a ring of rows in shared memory (one token, four rows a warp and more) against the kernel without one,
which two tokens take: the same additions in the same order, so the same bits. GPU only (-m gpu)."""
import pytest

from tests import oracle_lib as ol

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("t", [ol.Q4_1, ol.Q5_0, ol.Q5_1, ol.Q5_K, ol.IQ4_NL, ol.Q8_1, ol.Q2_K, ol.Q3_K, ol.Q8_K, ol.IQ4_XS])
@pytest.mark.parametrize("rows_past,units", [(0, 4), (-1, 4), (3, 5), (1500, 2), (4 * 148 * 16, 8), (7, 32)])
def test_the_ring_gives_the_same_bits(rq_ctx, t, rows_past, units):
    import numpy as np
    import torch

    # from the first row count that takes the ring: four rows a warp, eight warps a CTA, two CTAs an SM
    rows, cols = torch.cuda.get_device_properties(0).multi_processor_count * 2 * 8 * 4 + rows_past, 256 * units
    blocks = ol.random_blocks(t, 64 * cols // (256 if t in (ol.Q5_K, ol.Q2_K, ol.Q3_K, ol.Q8_K, ol.IQ4_XS) else 32), np.random.default_rng(t + units))
    flat = torch.from_numpy(np.ascontiguousarray(blocks).reshape(64, -1)).cuda()
    pick = torch.from_numpy(np.random.default_rng(rows).integers(0, 64, rows)).cuda()  # rows drawn from 64 different ones
    w = rq_ctx.weight_from_device(t, flat[pick].contiguous(), rows, cols)
    gen = torch.Generator(device="cuda").manual_seed(rows)
    x = torch.randn((1, cols), generator=gen, device="cuda")
    y1 = torch.full((1, rows), float("nan"), device="cuda")
    y2 = torch.full((2, rows), float("nan"), device="cuda")
    rq_ctx.matvec(w, x, y=y1, act_mode=0)
    rq_ctx.matvec(w, x.expand(2, cols).contiguous(), y=y2, act_mode=0)
    assert torch.equal(y1[0].view(torch.int32), y2[0].view(torch.int32))
    assert not torch.isnan(y1).all()
    wide = torch.zeros((1, 2 * cols), device="cuda")  # an input of another stride
    wide[:, ::2] = x
    y3 = torch.full((1, rows), float("nan"), device="cuda")
    rq_ctx.matvec(w, wide[:, ::2], y=y3, act_mode=0)
    assert torch.equal(y3.view(torch.int32), y1.view(torch.int32))
    rq_ctx.check()
