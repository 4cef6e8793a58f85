"""A weight made on the GPU and used by the very next launch of the same stream, by the kernels that read weights before they wait. GPU only (-m gpu)."""
import pytest

from tests import oracle_lib as ol

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("target,rows,cols", [(ol.Q4_1, 14400, 4096), (ol.Q4_1, 5000, 1024), (ol.Q8_0, 9000, 2048)])
def test_reencoded_and_multiplied_at_once(rq_ctx, target, rows, cols):
    import torch

    gen = torch.Generator(device="cuda").manual_seed(rows)
    # two sources in turn: memory given back and taken again does not hold the answer already
    sources = [rq_ctx.weight_from_device(ol.Q6_K, rq_ctx.quantize(ol.Q6_K, 0.02 * torch.randn(rows * cols, generator=gen, device="cuda")), rows, cols) for _ in range(2)]
    x = torch.randn((1, cols), generator=gen, device="cuda")
    want = []
    for w in sources:
        settled = rq_ctx.requantize(w, target)
        torch.cuda.synchronize()
        want.append(rq_ctx.matvec(settled, x, act_mode=0).clone())
        torch.cuda.synchronize()
    assert not torch.equal(want[0], want[1])
    for i in range(6):
        fresh = rq_ctx.requantize(sources[i % 2], target)
        got = rq_ctx.matvec(fresh, x, act_mode=0)
        assert torch.equal(got.view(torch.int32), want[i % 2].view(torch.int32))
        torch.cuda.synchronize()
    rq_ctx.check()
