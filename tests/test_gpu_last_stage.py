"""CTAs with no stage, one, and several, a last one that is full or one row: every row is written, once the CTA's last stage ends its warps' work. GPU only (-m gpu)."""
import pytest

from tests import oracle_lib as ol
from tests.test_gpu_parity import rel_err, torch_cuda

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("t", [ol.Q4_K, ol.Q6_K, ol.Q8_0, ol.Q4_0])
@pytest.mark.parametrize("cols,pass_rows", [(1024, 28), (14336, 2)])  # rows side by side in the CTA's seven warps; each row over all of them
@pytest.mark.parametrize("mode", ["float", "int8"])
def test_rows_around_whole_stages(rq_ctx, oracle, t, cols, pass_rows, mode):
    import torch

    import recipe_dev_b200 as rq

    ctas = 2 * torch.cuda.get_device_properties(0).multi_processor_count
    counts = [1, pass_rows, pass_rows + 1, ctas * pass_rows - 1, ctas * pass_rows, ctas * pass_rows + 1, 2 * ctas * pass_rows + 1]
    largest = 4 * ctas * pass_rows + 1 if cols < 4096 else counts[-1]
    act, omode = (rq.ACT_FLOAT, ol.FLOAT_RUN) if mode == "float" else (rq.ACT_INT8, ol.INT8)
    blocks = oracle.quantize(t, oracle.normal(71, t, largest * cols, 0.02))
    row = blocks.size // largest
    x = oracle.normal(71, 99, 2 * cols, 1.0).reshape(2, cols)
    all_rows = torch.empty((2, largest), device="cuda")
    whole = rq_ctx.weight_from_host(t, blocks, largest, cols)
    rq_ctx.matvec(whole, torch_cuda(x), y=all_rows, act_mode=act)
    assert rel_err(all_rows.cpu().numpy(), oracle.matvec(t, blocks, largest, cols, x, omode, 32).reshape(2, largest)) <= 1e-3
    for rows in counts:
        w = rq_ctx.weight_from_host(t, blocks[: rows * row], rows, cols)
        for tokens in (1, 2):
            y = torch.full((tokens, rows + 3), float("nan"), device="cuda")
            rq_ctx.matvec(w, torch_cuda(x[:tokens]), y=y[:, :rows], act_mode=act)
            assert torch.equal(y[:, :rows], all_rows[:tokens, :rows]) and torch.isnan(y[:, rows:]).all(), (rows, tokens)
    # several weights of one call, the shortest of less than a stage
    heights = [counts[2], 1, counts[3]]
    ws = [rq_ctx.weight_from_host(t, blocks[: n * row], n, cols) for n in heights]
    for y, n in zip(rq_ctx.matvec_multi(ws, torch_cuda(x[0]), [torch.empty(n, device="cuda") for n in heights], act_mode=act), heights):
        assert torch.equal(y, all_rows[0, :n])
    rq_ctx.check()
