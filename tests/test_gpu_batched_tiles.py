"""The batched product where few tiles are left over once every SM has its whole ones: outputs filled with NaN beforehand and every one
of them compared, all formats and both activation modes; and the work area such calls were reserved. GPU only (-m gpu)."""
import pytest

from tests import oracle_lib as ol

pytestmark = pytest.mark.gpu


def _rounded(x, step):
    """int8 codes times their steps, fp32 arithmetic as the format defines it, in 64 bits."""
    import torch

    g = x.reshape(x.shape[0], -1, step)
    best = g.gather(2, g.abs().argmax(2, keepdim=True))
    inverse = torch.full_like(best, -127.0) / best
    return (torch.round(g * inverse).clamp(-128, 127).double() * (torch.ones_like(inverse) / inverse).double()).reshape(x.shape)


@pytest.mark.parametrize("t", [ol.Q4_K, ol.Q6_K, ol.Q8_0, ol.Q4_0])
@pytest.mark.parametrize("tiles,rows,cols,tokens", [(1, 0, 512, 16), (2, -5, 4096, 16), (3, 0, 256, 33), (0, 19200, 2560, 100), (0, 14336, 4096, 700), (0, 8192, 2048, 400)])
def test_every_output_is_written(rq_ctx, t, tiles, rows, cols, tokens):
    import torch

    # `tiles` row tiles more than the GPU has SMs, the last of them `-rows` rows short, or `rows` as given
    rows = 128 * (torch.cuda.get_device_properties(0).multi_processor_count + tiles) + rows if tiles else rows
    gen = torch.Generator(device="cuda").manual_seed(rows + t)
    w = rq_ctx.weight_from_device(t, rq_ctx.quantize(t, 0.02 * torch.randn(rows * cols, generator=gen, device="cuda")), rows, cols)
    x = torch.randn((tokens, cols), generator=gen, device="cuda")
    dense = rq_ctx.dequant(w).reshape(rows, cols)
    for mode in (0, 1):
        y = torch.full((tokens, rows), float("nan"), device="cuda")
        rq_ctx.matmul(w, x, y=y, act_mode=mode)
        torch.cuda.synchronize()
        xd, worst = x.double() if mode == 0 else _rounded(x, 32), 0.0
        for r in range(0, rows, 4096):
            worst = max(worst, (y[:, r : r + 4096].double() - xd @ dense[r : r + 4096].double().T).abs().max().item())
        # 3e-6 of an output's usual size: 22 mantissa bits an input, sums of 64 products truncated once each, fp32 additions after that
        assert not torch.isnan(y).any() and worst <= 3e-6 * 5.0 * 0.02 * cols**0.5
    rq_ctx.check()


@pytest.mark.parametrize("tokens", [48, 49, 56, 64])
def test_a_reserved_context_holds_the_widest_window(tokens):
    """Rows enough for every SM, windows where fp32 calls over the 32-value formats go to two row halves."""
    import recipe_dev_b200 as rq
    import torch

    rows, cols = 14336, 1024
    ctx = rq.Context(0)
    ctx.reserve(rows, cols, tokens)
    x = torch.randn((tokens, cols), device="cuda")
    ws = [ctx.weight_from_device(t, ctx.quantize(t, 0.02 * torch.randn(rows * cols, device="cuda")), rows, cols) for t in (ol.Q4_K, ol.Q6_K, ol.Q8_0, ol.Q4_0)]
    calls = [(w, n, mode, torch.empty((n, rows), device="cuda")) for w in ws for n in {tokens, 48} for mode in (0, 1)]
    torch.cuda.synchronize()
    stream = ctx.sequence_begin()  # a recorded call that would have to allocate is refused
    for w, n, mode, y in calls:
        ctx.matmul(w, x[:n], y=y, act_mode=mode, stream=stream)
    seq = ctx.sequence_end()
    seq.run()
    torch.cuda.synchronize()
    ctx.check()
    for w, n, mode, y in calls:
        assert torch.equal(y, ctx.matmul(w, x[:n], act_mode=mode))
    seq.free()


@pytest.mark.parametrize("t,mode", [(ol.Q4_K, 0), (ol.Q6_K, 1), (ol.Q8_0, 0)])
def test_more_tokens_than_one_grid_layer_takes(rq_ctx, t, mode):
    import torch

    rows, cols, tokens = 9, 256, 8 * 65535 + 100
    gen = torch.Generator(device="cuda").manual_seed(t)
    w = rq_ctx.weight_from_device(t, rq_ctx.quantize(t, 0.02 * torch.randn(rows * cols, generator=gen, device="cuda")), rows, cols)
    x = torch.randn((tokens, cols), generator=gen, device="cuda")
    y = torch.full((tokens, rows), float("nan"), device="cuda")
    rq_ctx.matmul(w, x, y=y, act_mode=mode)
    dense = rq_ctx.dequant(w).reshape(rows, cols).double().T
    worst = 0.0
    for i in range(0, tokens, 1 << 17):
        xd = x[i : i + (1 << 17)]
        worst = max(worst, (y[i : i + (1 << 17)].double() - (xd.double() if mode == 0 else _rounded(xd, 32)) @ dense).abs().max().item())
    assert not torch.isnan(y).any() and worst <= 3e-6 * 5.0 * 0.02 * cols**0.5
    rq_ctx.check()
