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
