"""Int8 windows of a few positions in the matvec kernel: every position has the bits of its own call, whichever scheme the row length and
the window take (pairs, four tokens a pass with one or two rows a thread, one CTA per SM for long rows). GPU only (-m gpu)."""
import pytest

from tests import oracle_lib as ol
from tests.test_gpu_parity import torch_cuda

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("t", [ol.Q4_K, ol.Q6_K, ol.Q8_0, ol.Q4_0])
@pytest.mark.parametrize("rows,cols", [(1, 256), (700, 768), (4000, 2048), (3001, 2560), (1500, 4096), (37, 8448), (900, 14336), (20, 15360)])
def test_each_position_has_the_bits_of_its_own_call(rq_ctx, oracle, t, rows, cols):
    import torch

    w = rq_ctx.weight_from_host(t, oracle.quantize(t, oracle.normal(95, t, rows * cols, 0.02)), rows, cols)
    x = torch_cuda(oracle.normal(95, cols, 9 * cols, 1.0).reshape(9, cols))
    for step in (32, 256):
        own = torch.stack([rq_ctx.matvec(w, x[i], act_mode=1, step=step) for i in range(9)])
        for tokens in (2, 3, 4, 5, 9):
            assert torch.equal(rq_ctx.matvec(w, x[:tokens], act_mode=1, step=step), own[:tokens])
    rq_ctx.check()


@pytest.mark.parametrize("t", [ol.Q8_0, ol.Q4_0])
@pytest.mark.parametrize("cols", [1024, 2560, 4096, 14336])
def test_long_windows_are_as_close_to_64_bits_as_the_positions_own_calls(rq_ctx, t, cols):
    """The batched kernel adds a row's groups up in another order than the matvec kernel; it may not lose more by it (2 %, the spread of
    the two errors over inputs, is allowed)."""
    import torch

    from tests.test_gpu_batched_tiles import _rounded

    rows = 1024
    gen = torch.Generator(device="cuda").manual_seed(cols + t)
    w = rq_ctx.weight_from_device(t, rq_ctx.quantize(t, 0.02 * torch.randn(rows * cols, generator=gen, device="cuda")), rows, cols)
    dense = rq_ctx.dequant(w).reshape(rows, cols).double()
    for tokens in (16, 64, 128, 300):
        x = torch.randn((tokens, cols), generator=gen, device="cuda") * torch.exp(0.5 * torch.randn((1, cols), generator=gen, device="cuda"))
        want = _rounded(x, 32) @ dense.T
        window, own = ((f(w, x, act_mode=1).double() - want).norm().item() for f in (rq_ctx.matmul, rq_ctx.matvec))
        assert window <= 1.02 * own, (tokens, window / own)
    rq_ctx.check()


@pytest.mark.parametrize("t", [ol.Q8_0, ol.Q4_0])
@pytest.mark.parametrize("tokens", [1, 4, 16, 64, 100])
def test_sums_beyond_the_range_are_infinite(rq_ctx, t, tokens):
    import torch

    rows, cols = 300, 14336
    w = rq_ctx.weight_from_device(t, rq_ctx.quantize(t, 1.0 + torch.rand(rows * cols, device="cuda")), rows, cols)
    x = 1e36 * (1.0 + torch.rand((tokens, cols), device="cuda"))  # all of one sign: some 1e40 whatever the order of the additions
    for call in (rq_ctx.matvec, rq_ctx.matmul):
        assert torch.equal(call(w, x, act_mode=1), torch.full((tokens, rows), float("inf"), device="cuda"))
        assert torch.equal(call(w, -x, act_mode=1), torch.full((tokens, rows), float("-inf"), device="cuda"))
    rq_ctx.check()
