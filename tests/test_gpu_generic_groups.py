"""The decode-only formats' matvec, a lane per group of 32 values: rows per warp, widths that leave lanes idle or need several chunks of
x, arbitrary block bytes, infinite inputs, strides. GPU only (-m gpu)."""
import numpy as np
import pytest

from tests import oracle_lib as ol
from tests.test_gpu_parity import torch_cuda

pytestmark = pytest.mark.gpu
TYPES = [ol.Q4_1, ol.Q5_0, ol.Q5_1, ol.Q5_K, ol.IQ4_NL, ol.Q8_1, ol.Q2_K, ol.Q3_K, ol.Q8_K, ol.IQ4_XS]


@pytest.mark.parametrize("t", TYPES)
@pytest.mark.parametrize("rows,cols", [(1, 256), (5003, 768), (9600, 256), (33, 8192 + 256), (70, 17 * 1024)])
def test_against_64_bits(rq_ctx, oracle, t, rows, cols):
    values, _ = ol.GEOMETRY[t]
    if values == 32 and cols == 768:
        cols = 736
    blocks = ol.random_blocks(t, rows * cols // values, np.random.default_rng(t + rows))
    w = rq_ctx.weight_from_host(t, blocks, rows, cols)
    x = oracle.normal(91, cols, 2 * cols, 1.0).reshape(2, cols)
    y = rq_ctx.matvec(w, torch_cuda(x)).cpu().numpy()
    dense = oracle.dequantize(t, blocks).astype(np.float64).reshape(rows, cols)
    # codes are exact, a group's sum is a chain of eight fused products in each of two accumulators: a few 2^-24 of the sum of magnitudes
    bound = 2.0**-20 * (np.abs(x.astype(np.float64)) @ np.abs(dense).T) + 1e-30
    assert np.all(np.abs(y - x.astype(np.float64) @ dense.T) <= bound)
    one = rq_ctx.matvec(w, torch_cuda(x[1])).cpu().numpy()
    assert np.array_equal(one, y[1])
    strided = torch_cuda(np.ascontiguousarray(x.T))
    assert np.array_equal(rq_ctx.matvec(w, strided[:, 1]).cpu().numpy(), one)


@pytest.mark.parametrize("t", TYPES)
def test_infinite_inputs_meet_the_weight_itself(rq_ctx, oracle, t):
    values, _ = ol.GEOMETRY[t]
    rows, cols = 40, 512
    blocks = ol.random_blocks(t, rows * cols // values, np.random.default_rng(t))
    w = rq_ctx.weight_from_host(t, blocks, rows, cols)
    dense = oracle.dequantize(t, blocks).reshape(rows, cols)
    x = oracle.normal(92, t, cols, 1.0)
    for at, bad in ((3, np.inf), (300, -np.inf), (17, np.nan)):
        z = x.copy()
        z[at] = bad
        y = rq_ctx.matvec(w, torch_cuda(z)).cpu().numpy()
        with np.errstate(invalid="ignore"):
            want = dense[:, at] * np.float32(bad)
        assert np.array_equal(np.isnan(y), np.isnan(want))
        assert np.array_equal(y[~np.isnan(want)], want[~np.isnan(want)])
