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


def _value_by_value(dense, x):
    """Every weight decoded to fp32 and met with its input by one fused operation: 32 chains over the units of a row, then a tree."""
    units = dense.reshape(dense.shape[0], -1, 32).astype(np.float64)
    acc = np.zeros((dense.shape[0], 32), np.float32)
    for u in range(units.shape[1]):
        acc = (acc.astype(np.float64) + units[:, u] * x[32 * u : 32 * u + 32].astype(np.float64)).astype(np.float32)
    while acc.shape[1] > 1:
        acc = acc[:, : acc.shape[1] // 2] + acc[:, acc.shape[1] // 2 :]
    return acc[:, 0]


@pytest.mark.parametrize("t", TYPES)
@pytest.mark.parametrize("cols", [512, 4096])
def test_as_close_to_64_bits_as_decoding_value_by_value(rq_ctx, oracle, t, cols):
    rows = 600
    blocks = ol.random_blocks(t, rows * cols // ol.GEOMETRY[t][0], np.random.default_rng(t + cols))
    w = rq_ctx.weight_from_host(t, blocks, rows, cols)
    dense = oracle.dequantize(t, blocks).reshape(rows, cols)
    x = oracle.normal(93, t, cols, 1.0)
    exact = dense.astype(np.float64) @ x.astype(np.float64)
    error = np.linalg.norm(rq_ctx.matvec(w, torch_cuda(x)).cpu().numpy() - exact)
    assert error <= np.linalg.norm(_value_by_value(dense, x) - exact)


@pytest.mark.parametrize("t", TYPES)
def test_inputs_whose_products_with_the_codes_leave_the_range(rq_ctx, oracle, t):
    rows, cols = 90, 512
    blocks = ol.random_blocks(t, rows * cols // ol.GEOMETRY[t][0], np.random.default_rng(t + 7))
    w = rq_ctx.weight_from_host(t, blocks, rows, cols)
    dense = oracle.dequantize(t, blocks).reshape(rows, cols).astype(np.float64)
    x = (5e37 * np.clip(oracle.normal(94, t, cols, 1.0), -4, 4)).astype(np.float32)
    y = rq_ctx.matvec(w, torch_cuda(x)).cpu().numpy().astype(np.float64)
    assert np.all(np.abs(y - dense @ x.astype(np.float64)) <= 2.0**-20 * (np.abs(dense) @ np.abs(x.astype(np.float64))))
