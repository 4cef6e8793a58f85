"""fp32 activations in the matvec kernel: inputs as 24-bit integers of their 32-input group, in three digit planes. Accuracy against
64 bits over every format and row layout, inputs at the ends of the range, groups of a few large inputs among small ones, gated pairs
against the two projections. GPU only (-m gpu)."""
import numpy as np
import pytest

from tests import oracle_lib as ol
from tests.test_gpu_parity import torch_cuda

pytestmark = pytest.mark.gpu
TYPES = [ol.Q4_K, ol.Q6_K, ol.Q8_0, ol.Q4_0]


def _setup(rq_ctx, oracle, t, rows, cols):
    blocks = oracle.quantize(t, oracle.normal(81, t + cols, rows * cols, 0.02))
    return rq_ctx.weight_from_host(t, blocks, rows, cols), oracle.dequantize(t, blocks).astype(np.float64).reshape(rows, cols)


@pytest.mark.parametrize("t", TYPES)
@pytest.mark.parametrize("cols", [256, 768, 2048, 2560, 4096, 14336, 16384])  # one warp a row, padded groups, 5, 7 and 8 warps a row, partial sums
@pytest.mark.parametrize("spread", [0.0, 1.0, 6.0])
def test_accuracy_against_64_bits(rq_ctx, oracle, t, cols, spread):
    rows = 65
    w, exact = _setup(rq_ctx, oracle, t, rows, cols)
    x = (oracle.normal(82, cols, cols, 1.0) * np.exp(spread * oracle.normal(82, cols + 1, cols, 1.0))).astype(np.float32)
    y = rq_ctx.matvec(w, torch_cuda(x)).cpu().numpy()
    # an input's rounding is at most 2^-24 of its group's largest magnitude; a row's sum of 32 such errors a group, weighted, stays
    # below 2^-23 of sum |w| * (that magnitude); fp32 additions of the groups are covered by the factor of two
    top = np.repeat(np.abs(x).reshape(-1, 32).max(1), 32).astype(np.float64)
    bound = 2.0**-22 * (np.abs(exact) @ top)
    assert np.all(np.abs(y - exact @ x.astype(np.float64)) <= bound)
    if spread <= 1.0:
        assert np.linalg.norm(y - exact @ x.astype(np.float64)) <= 4e-7 * np.linalg.norm(exact @ x.astype(np.float64))
    # a window of positions gives each the bits of its own call
    xs = np.stack([x, x[::-1], 2 * x, x, np.roll(x, 7)]).astype(np.float32)
    ys = rq_ctx.matvec(w, torch_cuda(xs)).cpu().numpy()
    for i in range(5):
        assert np.array_equal(ys[i], rq_ctx.matvec(w, torch_cuda(xs[i])).cpu().numpy())
    rq_ctx.check()


@pytest.mark.parametrize("t", TYPES)
def test_inputs_at_the_ends_of_the_range(rq_ctx, oracle, t):
    rows, cols = 33, 1024
    w, exact = _setup(rq_ctx, oracle, t, rows, cols)
    base = oracle.normal(83, t, cols, 1.0)
    for scale in (1e-30, 1e-34, 1e30):
        x = (base.astype(np.float64) * scale).astype(np.float32)
        y, want = rq_ctx.matvec(w, torch_cuda(x)).cpu().numpy().astype(np.float64), exact @ x.astype(np.float64)
        # a step below 2^-126 is subnormal: off by up to 2^-150, and an input, 2^23 steps at most, by 2^-127
        assert np.all(np.abs(y - want) <= 1e-6 * np.max(np.abs(want)) + 2.0**-126 * np.sum(np.abs(exact), axis=1))
    assert np.array_equal(rq_ctx.matvec(w, torch_cuda(np.zeros(cols, np.float32))).cpu().numpy(), np.zeros(rows, np.float32))
    for bad in (np.nan, np.inf, -np.inf):
        x = base.copy()
        x[100] = bad
        y = rq_ctx.matvec(w, torch_cuda(x)).cpu().numpy()
        assert not np.any(np.isfinite(y))
    strided = torch_cuda(np.ascontiguousarray(np.stack([base, base]).T))  # every second float: the scalar loads
    assert np.array_equal(rq_ctx.matvec(w, strided[:, 0]).cpu().numpy(), rq_ctx.matvec(w, torch_cuda(base)).cpu().numpy())
    rq_ctx.check()


@pytest.mark.parametrize("t", TYPES)
@pytest.mark.parametrize("rows,cols", [(1, 256), (50, 768), (333, 2048), (1000, 4096), (40, 14336)])
@pytest.mark.parametrize("mode,step", [(0, 32), (1, 32), (1, 256)])
def test_gated_pairs_equal_the_two_projections(rq_ctx, oracle, t, rows, cols, mode, step):
    import torch

    g, _ = _setup(rq_ctx, oracle, t, rows, cols)
    u = rq_ctx.weight_from_host(t, oracle.quantize(t, oracle.normal(84, t, rows * cols, 0.02)), rows, cols)
    x = torch_cuda(oracle.normal(84, 5, 5 * cols, 1.0).reshape(5, cols))
    for tokens in (1, 5):
        xt = x[:tokens]
        y = rq_ctx.matvec_glu(g, u, xt, act_mode=mode, step=step).cpu().numpy()
        gd, ud = (rq_ctx.matvec(w, xt, act_mode=mode, step=step).cpu().numpy() for w in (g, u))
        want = oracle.glu(gd.reshape(-1), ud.reshape(-1)).reshape(tokens, rows)
        # the same sums in the same order wherever the rows have a lane layout; elsewhere to fp32 rounding of the sums
        assert np.max(np.abs(y - want)) <= 2e-6 * np.max(np.abs(want))
        first = rq_ctx.matvec_glu(g, u, x[0], act_mode=mode, step=step)
        assert torch.equal(first, torch.from_numpy(y[0]).cuda())
    if mode == 1:  # the fused launch leaves the records a cached call may use
        y1 = rq_ctx.matvec_glu(g, u, x[0], act_mode=1, step=step)
        cached, plain = torch.empty(rows, device="cuda"), rq_ctx.matvec(g, x[0], act_mode=1, step=step)
        rq_ctx.matvec_glu(g, u, x[0], y=y1, act_mode=1, step=step)
        s = torch.cuda.current_stream().cuda_stream
        assert rq_ctx.lib.rq_matvec(rq_ctx.handle, g.handle, x.data_ptr(), 1, cols, 1, cached.data_ptr(), 1, rows, 2, step, s) == 0
        assert torch.equal(cached, plain)
    rq_ctx.check()


def _with_zero_columns(oracle, t, rows, cols, at, seed):
    """Weights of 0 .. 0.06 (a Q4_K sub-block of them has no minimum) whose columns `at` are exact zeros, as blocks and in 64 bits."""
    dense = np.abs(oracle.normal(85, seed, rows * cols, 0.02)).reshape(rows, cols)
    dense[:, at] = 0.0
    blocks = oracle.quantize(t, np.ascontiguousarray(dense, np.float32).reshape(-1))
    if t == ol.Q4_K:  # no minimums, and codes of zero in those columns
        view = blocks.reshape(rows, cols // 256, 144)
        view[:, :, 2:4] = 0
        for c in at:
            view[:, c // 256, 16 + 32 * (c % 256 // 64) + c % 32] &= 0x0F if c % 64 >= 32 else 0xF0
    exact = oracle.dequantize(t, blocks).astype(np.float64).reshape(rows, cols)
    assert not exact[:, at].any()
    return blocks, exact


def _outlier_columns(cols, kind):
    # one input of a group in every other group; two of a group; three
    return np.concatenate([np.arange(5 + 7 * i, cols, 64) for i in range(kind)])


@pytest.mark.parametrize("t", TYPES)
@pytest.mark.parametrize("cols", [768, 2560, 4096, 14336, 16384])
@pytest.mark.parametrize("kind,size", [(1, 300.0), (1, 1e3), (1, 1e6), (1, 1e20), (2, 1e3), (2, 1e6), (3, 1e6)])
def test_large_inputs_over_zero_weights_take_nothing_from_the_others(rq_ctx, oracle, t, cols, kind, size):
    import torch

    rows, at = 33, _outlier_columns(cols, kind)
    blocks, exact = _with_zero_columns(oracle, t, rows, cols, at, t + cols)
    w = rq_ctx.weight_from_host(t, blocks, rows, cols)
    x = oracle.normal(86, cols, cols, 1.0)
    small = x.copy()
    small[at] = 0.0
    x[at] = np.where(np.arange(at.size) % 3 == 0, -size, size) * np.linspace(1.0, 0.7, at.size)
    y = rq_ctx.matvec(w, torch_cuda(x)).cpu().numpy()
    # the bound of the sum without them: 2^-22 of sum |w| times the group's largest other input (see the first test)
    top = np.repeat(np.abs(small).reshape(-1, 32).max(1), 32).astype(np.float64)
    assert np.all(np.abs(y - exact @ small.astype(np.float64)) <= 2.0**-22 * (np.abs(exact) @ top))
    assert np.linalg.norm(y - exact @ small.astype(np.float64)) <= 4e-7 * np.linalg.norm(exact @ small.astype(np.float64))
    xs = torch_cuda(np.stack([x, small, x[::-1].copy()]).astype(np.float32))
    ys = rq_ctx.matvec(w, xs)
    for i in range(3):
        assert torch.equal(ys[i], rq_ctx.matvec(w, xs[i]))
    strided = torch_cuda(np.ascontiguousarray(np.stack([x, x]).T))
    assert np.array_equal(rq_ctx.matvec(w, strided[:, 0]).cpu().numpy(), y)
    rq_ctx.check()


@pytest.mark.parametrize("t", TYPES)
@pytest.mark.parametrize("cols", [512, 4096])
def test_wide_groups_and_small_inputs_keep_their_bits(rq_ctx, oracle, t, cols):
    rows = 65
    w, exact = _setup(rq_ctx, oracle, t, rows, cols)
    base = oracle.normal(87, cols, cols, 1.0)
    wide = (base * np.exp(8.0 * oracle.normal(87, cols + 1, cols, 1.0))).astype(np.float32)  # twelve powers of two either way
    sparse = np.where(oracle.normal(87, cols + 2, cols, 1.0) > 1.5, base, 0.0).astype(np.float32)
    for x in (wide, sparse, (base * 1e-33).astype(np.float32), (base * 1e-36).astype(np.float32), (base * np.float32(1e-28)).astype(np.float32)):
        want = exact @ x.astype(np.float64)
        error = np.linalg.norm(rq_ctx.matvec(w, torch_cuda(x)).cpu().numpy() - want)
        # outputs of some 2^-126 and less have steps of 2^-149
        assert error <= 4e-7 * np.linalg.norm(want) + 2.0**-149 * np.sqrt(rows)


@pytest.mark.parametrize("t", [ol.Q4_K, ol.Q6_K, ol.Q8_0])
@pytest.mark.parametrize("hidden,ffn,tokens", [(1024, 512, 1), (2560, 256, 3), (2048, 768, 17)])
def test_gated_pairs_and_expert_banks_with_large_inputs(rq_ctx, oracle, t, hidden, ffn, tokens):
    import torch

    experts, at = 4, _outlier_columns(hidden, 1)
    tables = [_with_zero_columns(oracle, t, experts * ffn, hidden, at, 3 * t + i) for i in (0, 1)]
    down = oracle.quantize(t, oracle.normal(88, t, experts * hidden * ffn, 0.02))
    wide_down = oracle.dequantize(t, down).astype(np.float64).reshape(experts, hidden, ffn)
    bank = rq_ctx.moe_prepare(t, tables[0][0], tables[1][0], down, experts, hidden, ffn)
    x = oracle.normal(89, tokens, tokens * hidden, 1.0).reshape(tokens, hidden)
    small = x.astype(np.float64)
    small[:, at] = 0.0
    x[:, at] = 1e6
    routing = np.zeros((experts, tokens), np.float32)
    routing[1], routing[3] = 0.75, 0.25
    y = rq_ctx.moe_forward(bank, torch_cuda(x).T, torch_cuda(routing), 2).cpu().numpy().T
    want = np.zeros((tokens, hidden))
    for e in (1, 3):
        g, u = (small @ tab[1].reshape(experts, ffn, hidden)[e].T for tab in tables)
        want += routing[e, 0] * (g / (1.0 + np.exp(-g)) * u @ wide_down[e].T)
    assert np.linalg.norm(y - want) <= 2e-6 * np.linalg.norm(want)
    gate, up = (rq_ctx.weight_from_host(t, tab[0], experts * ffn, hidden) for tab in tables)
    xd = torch_cuda(x)
    both = rq_ctx.matvec_glu(gate, up, xd).cpu().numpy()
    g, u = (small @ tab[1].T for tab in tables)
    want = g / (1.0 + np.exp(-g)) * u
    assert np.linalg.norm(both - want) <= 2e-6 * np.linalg.norm(want)
    rq_ctx.check()


@pytest.mark.parametrize("t", TYPES)
@pytest.mark.parametrize("cols", [2560, 4096, 14336])
@pytest.mark.parametrize("zeros", [0.5, 0.8])
def test_large_inputs_among_small_ones_and_zeros(rq_ctx, oracle, t, cols, zeros):
    """Zeros take no part in what the inputs of a group are on average."""
    rows, at = 33, _outlier_columns(cols, 1)
    blocks, exact = _with_zero_columns(oracle, t, rows, cols, at, t + cols + 1)
    w = rq_ctx.weight_from_host(t, blocks, rows, cols)
    rng = np.random.default_rng(cols)
    small = np.where(rng.random(cols) < zeros, 0.0, oracle.normal(90, cols, cols, 1.0)).astype(np.float32)
    small[at] = 0.0
    x = small.copy()
    x[at] = 1e6
    for z in (x, small):
        y = rq_ctx.matvec(w, torch_cuda(z)).cpu().numpy()
        assert np.linalg.norm(y - exact @ small.astype(np.float64)) <= 4e-7 * np.linalg.norm(exact @ small.astype(np.float64))
    rq_ctx.check()
