"""The batched product over all four stored formats at the edges of its cut: one and two row halves, token tiles that are not full,
rows past a tile, widths that are no whole units, tiles shared by several CTAs, both activation modes. GPU only (-m gpu)."""
import numpy as np
import pytest

from tests import oracle_lib as ol
from tests.test_gpu_parity import rel_err, torch_cuda

pytestmark = pytest.mark.gpu

SHAPES = [  # rows, cols, tokens
    (1, 256, 12), (129, 512, 64), (257, 512, 65), (255, 1024, 96), (300, 768, 97), (520, 2304, 193), (40, 14336, 16), (4000, 256, 13), (9500, 512, 200), (3879, 4352, 63), (2900, 2816, 33), (5000, 1792, 90),
]
RAGGED = [(130, 32, 12), (200, 96, 70), (65, 1120, 31), (300, 2592, 100)]  # 32-value formats only


def _case(oracle, t, rows, cols, tokens):
    per, stride = ol.GEOMETRY[t]
    blocks = oracle.quantize(t, oracle.normal(71, t + rows, rows * cols, 0.02))
    x = oracle.normal(71, 7 + tokens, tokens * cols, 1.0).reshape(tokens, cols)
    pick = np.unique(np.concatenate([np.arange(0, rows, max(1, rows // 24)), [rows - 1, min(rows - 1, 127), min(rows - 1, 128), min(rows - 1, 255), min(rows - 1, 256)]]))
    sub = np.ascontiguousarray(blocks.reshape(rows, cols // per * stride)[pick]).reshape(-1)
    return blocks, x, pick, sub


@pytest.mark.parametrize("t,rows,cols,tokens", [(t, *s) for t in (ol.Q4_K, ol.Q6_K, ol.Q8_0, ol.Q4_0) for s in SHAPES] + [(t, *s) for t in (ol.Q8_0, ol.Q4_0) for s in RAGGED])
def test_batched_product_at_the_edges(rq_ctx, oracle, t, rows, cols, tokens):
    import recipe_dev_b200 as rq

    blocks, x, pick, sub = _case(oracle, t, rows, cols, tokens)
    w = rq_ctx.weight_from_host(t, blocks, rows, cols)
    xd = torch_cuda(x)
    y = rq_ctx.matmul(w, xd).cpu().numpy()
    exact = x.astype(np.float64) @ oracle.dequantize(t, sub).astype(np.float64).reshape(pick.size, cols).T
    # 22 mantissa bits an input, sums of 64 products truncated once each, fp32 additions after that: 3e-6 of the largest output
    # (a handful of outputs may all be small against the sums behind them)
    assert np.max(np.abs(y[:, pick] - exact)) <= 3e-6 * max(np.max(np.abs(exact)), np.sqrt(cols) * 0.02)
    for step in (32, 256):
        y8 = rq_ctx.matmul(w, xd, act_mode=rq.ACT_INT8, step=step).cpu().numpy()
        assert rel_err(y8[:, pick], oracle.matvec(t, sub, pick.size, cols, x, ol.INT8, step)) <= 1e-3
    rq_ctx.check()


def test_channel_major_planes_and_a_requantised_weight(rq_ctx, oracle):
    import torch

    rows, cols, tokens = 140, 512, 70
    blocks, x, _, _ = _case(oracle, ol.Q6_K, rows, cols, tokens)
    w8 = rq_ctx.int8_weight(rq_ctx.weight_from_host(ol.Q6_K, blocks, rows, cols))
    xd = torch_cuda(x)
    want = rq_ctx.matmul(w8, xd, act_mode=1)
    xc, yc = torch_cuda(np.ascontiguousarray(x.T)), torch.zeros((rows, tokens), device="cuda")
    rc = rq_ctx.lib.rq_matmul(rq_ctx.handle, w8.handle, xc.data_ptr(), tokens, 1, tokens, yc.data_ptr(), tokens, 1, 1, 32, torch.cuda.current_stream().cuda_stream)
    assert rc == 0 and torch.equal(yc.T.contiguous(), want)
    rq_ctx.check()


def test_reserved_context_does_not_grow_for_any_format_or_window(rq_ctx, oracle):
    import recipe_dev_b200 as rq
    import torch

    ctx = rq.Context(0)
    ctx.reserve(600, 1024, 200)
    ws = [ctx.weight_from_host(t, oracle.quantize(t, oracle.normal(72, t, 600 * 1024, 0.02)), 600, 1024) for t in (ol.Q4_K, ol.Q6_K, ol.Q8_0, ol.Q4_0)]
    x = torch.randn(200, 1024, device="cuda")
    calls = [(w, n, mode, torch.empty(n, 600, device="cuda")) for w in ws for n in (12, 64, 65, 97, 200) for mode in (0, 1)]
    torch.cuda.synchronize()
    stream = ctx.sequence_begin()  # a recorded call that would have to allocate is refused
    for w, n, mode, y in calls:
        ctx.matmul(w, x[:n], y=y, act_mode=mode, stream=stream)
    seq = ctx.sequence_end()
    seq.run()
    torch.cuda.synchronize()
    ctx.check()
    assert torch.equal(calls[-1][3], ctx.matmul(ws[-1], x, act_mode=1))
    seq.free()
