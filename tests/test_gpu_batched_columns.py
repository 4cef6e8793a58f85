"""The batched product at the edges of its token tiles (16, 32, 48, 64 columns of one row half, 64, 96, 128 of two) and of Q4_K's windows of
four superblocks, whole and cut between CTAs. GPU only (-m gpu)."""
import pytest

from tests import oracle_lib as ol

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("t", [ol.Q4_K, ol.Q6_K, ol.Q8_0, ol.Q4_0])
@pytest.mark.parametrize("rows,units,counts", [(300, 1, (12, 16, 17, 65)), (129, 5, (32, 33, 96, 97)), (700, 9, (48, 49, 64, 128, 129)), (5000, 14, (63, 112, 193)), (19072, 3, (20, 90))])
def test_edges_of_the_token_tiles(rq_ctx, t, rows, units, counts):
    import torch

    cols = 256 * units
    gen = torch.Generator(device="cuda").manual_seed(rows + t)
    w = rq_ctx.weight_from_device(t, rq_ctx.quantize(t, 0.02 * torch.randn(rows * cols, generator=gen, device="cuda")), rows, cols)
    dense = rq_ctx.dequant(w).reshape(rows, cols).double()
    for tokens in counts:
        x = torch.randn((tokens, cols), generator=gen, device="cuda")
        # int8 over Q8_0 / Q4_0 has kernels of its own; its codes times its steps are what a call over them as fp32 numbers multiplies
        g = x.reshape(tokens, -1, 32)
        best = g.gather(2, g.abs().argmax(2, keepdim=True))
        inverse = torch.full_like(best, -127.0) / best
        coded = (torch.round(g * inverse).clamp(-128, 127).double() * (torch.ones_like(inverse) / inverse).double()).reshape(x.shape)
        for mode, xd in ((0, x.double()), (1, coded)):
            y = torch.full((tokens, rows), float("nan"), device="cuda")
            rq_ctx.matmul(w, x, y=y, act_mode=mode)
            worst = (y.double() - xd @ dense.T).abs().max().item()
            # as in test_gpu_batched_tiles.py: 3e-6 of an output's usual size (22 mantissa bits an input, sums of 64 products truncated once each)
            assert not torch.isnan(y).any() and worst <= 3e-6 * 5.0 * 0.02 * cols**0.5, (tokens, mode, worst)
    rq_ctx.check()
