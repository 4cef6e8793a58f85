"""The decode-only formats' matvec with a ring of rows in shared memory (one token) against the kernel without one, which two tokens
take: the same additions in the same order, so the same bits; and against 64 bits. Which calls have a ring: tests/test_ring_rule.py, which
holds the list. GPU only (-m gpu)."""
import pytest

from tests import oracle_lib as ol
from tests.test_ring_rule import RING

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("t,rows,cols", RING)
def test_the_ring_gives_the_same_bits(rq_ctx, oracle, t, rows, cols):
    import numpy as np
    import torch

    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("the list is for 148 SMs")
    blocks = ol.random_blocks(t, 64 * cols // ol.GEOMETRY[t][0], np.random.default_rng(t + cols))
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
    dense = torch.from_numpy(oracle.dequantize(t, blocks).astype(np.float64).reshape(64, cols)).cuda()
    want, size = dense @ x[0].double(), dense.abs() @ x[0].abs().double()
    # codes are exact, a group's sum is a chain of eight fused products in each of two accumulators: a few 2^-24 of the sum of magnitudes
    assert ((y1[0].double() - want[pick]).abs() <= 2.0**-20 * size[pick] + 1e-30).all()
    wide = torch.zeros((1, 2 * cols), device="cuda")  # an input of another stride
    wide[:, ::2] = x
    y3 = torch.full((1, rows), float("nan"), device="cuda")
    rq_ctx.matvec(w, wide[:, ::2], y=y3, act_mode=0)
    assert torch.equal(y3.view(torch.int32), y1.view(torch.int32))
    rq_ctx.check()
