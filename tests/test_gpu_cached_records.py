"""RQ_ACT_INT8_CACHED behind int8 windows over Q8_0 / Q4_0, short ones (matvec kernels) and long ones (the batched kernel): accepted, and
the bits of a call that derives its records itself, from either entry point. GPU only (-m gpu)."""
import pytest

from tests import oracle_lib as ol
from tests.test_gpu_parity import torch_cuda

pytestmark = pytest.mark.gpu


def _call(ctx, entry, w, x, tokens, mode, step):
    import torch

    y = torch.full((tokens, w.rows), float("nan"), device="cuda")
    rc = getattr(ctx.lib, entry)(ctx.handle, w.handle, x.data_ptr(), 1, x.shape[1], tokens, y.data_ptr(), 1, w.rows, mode, step, torch.cuda.current_stream().cuda_stream)
    return rc, y


@pytest.mark.parametrize("t", [ol.Q8_0, ol.Q4_0])
@pytest.mark.parametrize("cols,tokens", [(1024, 8), (1024, 9), (1024, 16), (2560, 100), (14336, 5), (1120, 31), (96, 12), (8224, 7)])
@pytest.mark.parametrize("step", [32, 256])
def test_cached_calls_behind_a_window(rq_ctx, oracle, t, cols, tokens, step):
    import torch

    q, k = (rq_ctx.weight_from_host(t, oracle.quantize(t, oracle.normal(61, r, r * cols, 0.02)), r, cols) for r in (300, 140))
    x = torch_cuda(oracle.normal(62, cols, tokens * cols, 1.0).reshape(tokens, cols))
    want = {e: _call(rq_ctx, e, k, x, tokens, 1, step)[1] for e in ("rq_matvec", "rq_matmul")}
    for first in ("rq_matmul", "rq_matvec"):
        for entry in ("rq_matvec", "rq_matmul", "rq_matvec"):
            rc, _ = _call(rq_ctx, first, q, x, tokens, 1, step)
            assert rc == 0
            for again in (entry, "rq_matmul", entry):  # a cached call leaves the records as they are; it does not read x again
                rc, y = _call(rq_ctx, again, k, torch.zeros_like(x), tokens, 2, step)
                assert rc == 0, rq_ctx.lib.rq_last_error()
                assert torch.equal(y, want[again])
    if cols % 256 == 0:  # the slice sums of the records, which these formats do not read
        six = rq_ctx.weight_from_host(ol.Q6_K, oracle.quantize(ol.Q6_K, oracle.normal(63, t, 70 * cols, 0.02)), 70, cols)
        _, plain = _call(rq_ctx, "rq_matvec", six, x, tokens, 1, step)
        assert _call(rq_ctx, "rq_matmul", q, x, tokens, 1, step)[0] == 0
        rc, y = _call(rq_ctx, "rq_matvec", six, x, tokens, 2, step)
        assert rc == 0 and torch.equal(y, plain)
    assert _call(rq_ctx, "rq_matvec", k, x, tokens - 1, 2, step)[0] == -1  # another token count
    rq_ctx.check()


def test_a_cached_call_allocates_nothing():
    """Records of a matvec call in a work area that has no room for the batched kernel's image: the matvec kernels serve the call."""
    import recipe_dev_b200 as rq
    import torch

    rows, cols, tokens = 20000, 512, 64
    ctx = rq.Context(0)
    w = ctx.weight_from_device(rq.Q8_0, ctx.quantize(rq.Q8_0, 0.02 * torch.randn(rows * cols, device="cuda")), rows, cols)
    x = torch.randn((tokens, cols), device="cuda")
    rc, want = _call(ctx, "rq_matvec", w, x, tokens, 1, 32)
    assert rc == 0
    rc, y = _call(ctx, "rq_matmul", w, x, tokens, 2, 32)
    assert rc == 0 and torch.equal(y, want)
    ctx.check()
