"""Launches that start before the one ahead of them has ended: a recorded chain in which every call reads what the call before it
wrote, replayed on new inputs, against the same calls with a synchronisation after each, bit for bit. GPU only (-m gpu)."""
import numpy as np
import pytest

from tests import oracle_lib as ol

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("hidden,ffn", [(1024, 2048), (4096, 14336)])
def test_every_call_sees_the_one_before(rq_ctx, oracle, mode, hidden, ffn):
    import recipe_dev_b200 as rq
    import torch

    ctx = rq.Context(0)
    ctx.reserve(ffn, ffn, 16)
    rng = np.random.default_rng(3)
    gen = torch.Generator(device="cuda").manual_seed(1)

    def weight(t, rows, cols):
        w = ctx.weight_from_device(t, ctx.quantize(t, 0.02 * torch.randn(rows * cols, generator=gen, device="cuda")), rows, cols)
        torch.cuda.synchronize()
        return w

    o, gate, up, down = weight(rq.Q4_K, hidden, hidden), weight(rq.Q4_K, ffn, hidden), weight(rq.Q4_K, ffn, hidden), weight(rq.Q6_K, hidden, ffn)
    tail8, tail_k = weight(rq.Q8_0, 512, hidden), weight(rq.Q4_K, 512, hidden)
    other = ctx.weight_from_host(rq.Q5_K, ol.random_blocks(ol.Q5_K, hidden * hidden // 256, rng), hidden, hidden)
    gain = 1.0 + 0.1 * torch.randn(hidden, generator=gen, device="cuda")
    x = torch.empty(hidden, device="cuda")
    b = {n: torch.empty(r, device="cuda") for n, r in (("o", hidden), ("h", hidden), ("n", hidden), ("g", ffn), ("d", hidden), ("e", hidden))}
    many, y8, yk = torch.empty((16, hidden), device="cuda"), torch.empty((16, 512), device="cuda"), torch.empty((16, 512), device="cuda")

    def calls(stream, after):
        for f in (lambda: ctx.matvec(o, x, y=b["o"], act_mode=mode, stream=stream), lambda: ctx.add(x, b["o"], y=b["h"], stream=stream),
                  lambda: ctx.rmsnorm(b["h"], gain, y=b["n"], stream=stream), lambda: ctx.matvec_glu(gate, up, b["n"], y=b["g"], act_mode=mode, stream=stream),
                  lambda: ctx.matvec(down, b["g"], y=b["d"], act_mode=mode, stream=stream), lambda: ctx.matvec(other, b["d"], y=b["e"], stream=stream),
                  lambda: ctx.add(b["e"], b["d"], y=many[0], stream=stream),
                  lambda: ctx.matmul(tail8, many, y=y8, act_mode=mode, stream=stream), lambda: ctx.matmul(tail_k, many, y=yk, act_mode=mode, stream=stream)):
            f()
            after()

    torch.cuda.synchronize()
    stream = ctx.sequence_begin()
    calls(stream, lambda: None)
    seq = ctx.sequence_end()
    planes = list(b.values()) + [many, y8, yk]
    for trial in range(6):
        x.copy_(torch.randn(hidden, generator=gen, device="cuda"))
        rest = torch.randn((16, hidden), generator=gen, device="cuda")
        for p in planes:
            p.fill_(float(trial))
        many.copy_(rest)
        torch.cuda.synchronize()
        seq.run()
        torch.cuda.synchronize()
        got = [p.clone() for p in planes]
        for p in planes:
            p.fill_(-1.0)
        many.copy_(rest)
        torch.cuda.synchronize()
        calls(None, torch.cuda.synchronize)
        for a, want in zip(got, planes):
            assert torch.equal(a, want)
    ctx.check()
    seq.free()


@pytest.mark.parametrize("cols", [768, 4096, 14336])
def test_windows_and_elementwise_steps_see_the_one_before(cols):
    """Four int8 positions whose codes are made from what the launch before wrote, steps in between, a Q4_1 window."""
    import recipe_dev_b200 as rq
    import torch

    ctx = rq.Context(0)
    ctx.reserve(cols, cols, 4)
    gen = torch.Generator(device="cuda").manual_seed(2)
    k8 = ctx.weight_from_device(rq.Q8_0, ctx.quantize(rq.Q8_0, 0.02 * torch.randn(640 * cols, generator=gen, device="cuda")), 640, cols)
    k4 = ctx.weight_from_host(ol.Q4_1, ol.random_blocks(ol.Q4_1, 96 * cols // 32, np.random.default_rng(5)), 96, cols)
    x = torch.empty((4, cols), device="cuda")
    a, c, y8, y1, y4 = torch.empty_like(x), torch.empty_like(x), torch.empty((4, 640), device="cuda"), torch.empty(640, device="cuda"), torch.empty((4, 96), device="cuda")

    def calls(stream, after):
        for f in (lambda: ctx.add(x, x, y=a, stream=stream), lambda: ctx.softcap(a, 30.0, y=c, stream=stream), lambda: ctx.matvec(k8, c, y=y8, act_mode=1, stream=stream),
                  lambda: ctx.add(c, a, y=c, stream=stream), lambda: ctx.matvec(k8, c[0], y=y1, act_mode=1, stream=stream), lambda: ctx.softcap(c, 20.0, y=a, stream=stream),
                  lambda: ctx.matvec(k4, a, y=y4, act_mode=1, stream=stream)):
            f()
            after()

    torch.cuda.synchronize()
    stream = ctx.sequence_begin()
    calls(stream, lambda: None)
    seq = ctx.sequence_end()
    planes = [a, c, y8, y1, y4]
    for trial in range(6):
        x.copy_(20.0 * torch.randn(x.shape, generator=gen, device="cuda"))
        for p in planes:
            p.fill_(float(trial))
        torch.cuda.synchronize()
        seq.run()
        torch.cuda.synchronize()
        got = [p.clone() for p in planes]
        for p in planes:
            p.fill_(-1.0)
        torch.cuda.synchronize()
        calls(None, torch.cuda.synchronize)
        for g, want in zip(got, planes):
            assert torch.equal(g, want)
    ctx.check()
    seq.free()
