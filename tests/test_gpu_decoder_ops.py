"""Operators of the decoder graph, each alone, against float64 statements (gigusun_oracle.py): odd and unequal
sizes, both activation types, every kernel behind an operator, keys at every kind of edge."""
from __future__ import annotations

import numpy as np
import pytest

import gigusun_oracle as oracle
from gpu_util import stream

pytestmark = pytest.mark.gpu


def cuda(values, dtype=None):
    import torch

    tensor = torch.from_numpy(np.ascontiguousarray(values))
    return tensor.to("cuda", dtype or tensor.dtype)


def activation(values, float32):
    """Device tensor in the activation type, and the float64 values it holds."""
    import torch

    tensor = cuda(np.asarray(values, np.float32), torch.float32 if float32 else torch.bfloat16)
    return tensor, tensor.double().cpu().numpy()


def empty(shape, float32):
    import torch

    return torch.full(shape, float("nan"), dtype=torch.float32 if float32 else torch.bfloat16, device="cuda")


def assert_near(actual, expected, float32, factor=1.0):
    actual = actual.double().cpu().numpy() if hasattr(actual, "cpu") else actual
    bound = (2e-5 if float32 else 1.2e-2) * factor
    scale = np.sqrt(np.mean(expected * expected)) + 1e-30
    worst = np.max(np.abs(actual - expected) / (np.abs(expected) + scale))
    assert np.isfinite(actual).all() and worst < bound, (worst, bound)


TYPES = pytest.mark.parametrize("float32", [0, 1], ids=["bf16", "f32"])


@TYPES
@pytest.mark.parametrize("width", [8, 60, 77, 1536, 8200, 16392])
def test_row_norms(ops, float32, width):
    rng = np.random.default_rng(width)
    rows, eps = 5, 1e-3
    x = rng.normal(0, 0.05, (rows, width)).astype(np.float32)      # small enough that epsilon matters
    gain = rng.uniform(0.5, 1.5, width).astype(np.float32)
    out = empty((rows, width), float32)
    dx, dg = cuda(x), cuda(gain)
    ops.call("rms_norm_residual", dx.data_ptr(), dg.data_ptr(), rows, width, eps, float32, out.data_ptr(), stream())
    assert_near(out, oracle.rms(x.astype(np.float64), eps) * gain, float32)
    coefficients = np.array([0.7, -0.4, 0.3, 0.2], np.float32)
    z, zv = activation(rng.normal(0, 0.8, (rows, width)), float32)
    dc = cuda(coefficients)
    ops.call("poly_norm", z.data_ptr(), dc.data_ptr(), rows, width, eps, float32, out.data_ptr(), stream())
    assert_near(out, oracle.poly_norm(zv, coefficients.astype(np.float64), eps), float32)
    ops.call("poly_norm", z.data_ptr(), dc.data_ptr(), rows, width, eps, float32, z.data_ptr(), stream())
    assert bool((z == out).all())                                  # in place


@pytest.mark.parametrize("width", [48, 51, 9000])
def test_embedding_adds_the_position_before_its_norm(ops, width):
    import torch

    rng = np.random.default_rng(width)
    table, tv = activation(rng.normal(0, 1, (30, width)), 0)
    places, pv = activation(rng.normal(0, 1, (40, width)), 0)
    gain = rng.uniform(0.5, 1.5, width).astype(np.float32)
    tokens = np.array([3, 29, 0, 3], np.int32)
    out, dt, dg = empty((4, width), 1), cuda(tokens), cuda(gain)
    ops.call("embed_positions", dt.data_ptr(), table.data_ptr(), places.data_ptr(), dg.data_ptr(), 4, width, 30, 36, 1e-6,
             out.data_ptr(), stream())
    expected = oracle.embed(tokens, tv, pv, gain.astype(np.float64) - 1.0, 1e-6, first=36)
    assert_near(out, expected, 1)
    bad = cuda(np.array([1, 30, 2, 2], np.int32))                  # an id outside the vocabulary
    ops.call("embed_positions", bad.data_ptr(), table.data_ptr(), places.data_ptr(), dg.data_ptr(), 4, width, 30, 0, 1e-6,
             out.data_ptr(), stream())
    assert ops.status("check_async_errors", stream()) == 2
    assert not out[1].any() and bool(torch.isfinite(out).all())


def test_distance_table(ops):
    r1, r2 = np.array([0.3, 1.7], np.float32), np.array([0.05, 2.5], np.float32)
    d1, d2, table = cuda(r1), cuda(r2), empty((2, 700), 1)
    ops.call("distance_bias_table", d1.data_ptr(), d2.data_ptr(), 2, 700, table.data_ptr(), stream())
    expected = r1[:, None].astype(np.float64) * np.log1p(r2[:, None].astype(np.float64) * np.arange(700))
    assert_near(table, expected, 1)


@pytest.mark.parametrize("rows", [1, 3, 8, 11, 17, 64, 100, 129, 600])
@pytest.mark.parametrize("inner, outer", [(16, 24), (72, 300), (200, 37), (192, 1032), (128, 8)])
def test_f32_results(ops, rows, inner, outer):
    """F32 multiply-adds, and BF16 operands whose F32 accumulator is stored or added without rounding."""
    rng = np.random.default_rng(rows * 1000 + outer)
    x, xv = activation(rng.normal(0, 1, (rows, inner)), 0)
    w, wv = activation(rng.normal(0, 1, (outer, inner)), 0)
    base = rng.normal(0, 1, (rows, outer)).astype(np.float32)
    exact = cuda(rng.normal(0, 1, (rows, inner)).astype(np.float32))
    work = empty((1 << 22,), 1)
    for accumulate in (0, 1):
        out = cuda(base)
        ops.call("f32_linear", exact.data_ptr(), w.data_ptr(), rows, inner, outer, accumulate, out.data_ptr(), stream())
        assert_near(out, exact.double().cpu().numpy() @ wv.T + accumulate * base, 1)
        for workspace in (None, work.data_ptr()):
            out = cuda(base)
            ops.call("bf16_linear_f32_result", x.data_ptr(), w.data_ptr(), rows, inner, outer, accumulate, workspace,
                     work.numel() * 4, out.data_ptr(), stream())
            ops.call("check_async_errors", stream())
            assert_near(out, xv @ wv.T + accumulate * base, 1)


@pytest.mark.parametrize("rows", [2, 31, 33, 48, 90, 97, 128, 161])
@pytest.mark.parametrize("inner, outer", [(8, 5), (100, 129), (130, 127), (264, 128), (520, 260), (1111, 40), (2056, 150)])
def test_f32_products(ops, rows, inner, outer):
    """Every height of the F32 tile and every split of the inner size, whole and ragged: the chains have at most
    16 (ceil(inner / 256) + 4) additions, each rounded to 2^-24 of sums below the sum of the magnitudes."""
    rng = np.random.default_rng(rows * 1000 + inner)
    w, wv = activation(rng.normal(0, 1, (outer, inner)), 0)
    x, base = (rng.normal(0, 1, shape).astype(np.float32) for shape in ((rows, inner), (rows, outer)))
    exact = cuda(x)
    out = cuda(base)
    ops.call("f32_linear", exact.data_ptr(), w.data_ptr(), rows, inner, outer, 1, out.data_ptr(), stream())
    error = np.abs(out.double().cpu().numpy() - (x.astype(np.float64) @ wv.T + base))
    chain = 16 * (-(-inner // 256) + 4)
    assert np.all(error <= chain * 2.0 ** -24 * (np.abs(x).astype(np.float64) @ np.abs(wv).T + np.abs(base)))


@pytest.mark.parametrize("rows, inner, outer", [(1, 1001, 40), (1, 16400, 9), (2, 8, 5), (3, 1111, 70), (12, 2056, 150), (13, 2056, 150),
                                                (16, 100, 129), (16, 520, 260), (17, 520, 260), (13, 8192, 6400), (12, 8192, 6400)])
def test_few_f32_rows(ops, rows, inner, outer):
    """Both sides of the line between a warp per output and the tiles, whole and ragged, and weights on either side of L2.
    A lane of the former adds 8 ceil(inner / 256) products (single ones: ceil(inner / 32)), five lanes' sums and the base."""
    rng = np.random.default_rng(rows * 1000 + inner)
    w, wv = activation(rng.normal(0, 1, (outer, inner)), 0)
    x, base = (rng.normal(0, 1, shape).astype(np.float32) for shape in ((rows, inner), (rows, outer)))
    exact, out = cuda(x), cuda(base)
    ops.call("f32_linear", exact.data_ptr(), w.data_ptr(), rows, inner, outer, 1, out.data_ptr(), stream())
    error = np.abs(out.double().cpu().numpy() - (x.astype(np.float64) @ wv.T + base))
    chain = 16 * (-(-inner // 256) + 4)  # of the tiles; the lanes' is shorter
    assert np.all(error <= chain * 2.0 ** -24 * (np.abs(x).astype(np.float64) @ np.abs(wv).T + np.abs(base)))


@pytest.mark.parametrize("rows, inner, outer", [(17, 64, 127), (32, 64, 1), (33, 72, 129), (96, 200, 128), (97, 1080, 260), (128, 2048, 40),
                                                (129, 136, 1000), (3, 2056, 6150), (16, 4104, 2049), (2, 264, 4096), (2, 2056, 4099)])
def test_f32_products_on_the_tensor_cores(ops, rows, inner, outer):
    """Every row tile, K blocks and weight tiles with remainders, one CTA and clusters that divide K, and two rows.  A block
    of 64 products is cut at 2^-23 of a sum of at most its magnitudes four times with the largest plane (8 units of 2^-24; the smaller
    planes' eight cuts are 2^-8 of these), the blocks' and the CTAs' sums are rounded: 16 + inner / 512 + 8 units allow for that
    with clusters of eight, and for 8 units beyond.  (A product more than 2^-11 below the largest is cut as well, at 2^-25 of
    it: 32 units if all but one were, a tenth of a unit here.)  Then values that are not finite: the same infinities and NaNs as
    multiply-adds give."""
    import torch

    rng = np.random.default_rng(rows * 1000 + inner)
    w, wv = activation(rng.normal(0, 1, (outer, inner)), 0)
    x, base = (rng.normal(0, 1, shape).astype(np.float32) for shape in ((rows, inner), (rows, outer)))
    x *= np.exp(rng.normal(0, 2, x.shape)).astype(np.float32)
    exact, out = cuda(x), cuda(base)
    ops.call("f32_linear", exact.data_ptr(), w.data_ptr(), rows, inner, outer, 1, out.data_ptr(), stream())
    error = np.abs(out.double().cpu().numpy() - (x.astype(np.float64) @ wv.T + base))
    bound = (16 + inner / 64 / 8 + 8) * 2.0 ** -24 if rows > 2 else 16 * (-(-inner // 256) + 4) * 2.0 ** -24
    assert np.all(error <= bound * (np.abs(x).astype(np.float64) @ np.abs(wv).T + np.abs(base)))

    odd = torch.zeros(rows, inner, device="cuda")
    odd[0, 1], odd[0, 5] = float("inf"), 2.0
    odd[1, inner - 1], odd[1, 2] = float("nan"), 1.0
    if rows > 2:
        odd[2, 3], odd[2, inner - 2] = float("-inf"), float("inf")
        odd[rows - 1, 7] = 1.5  # meets the infinite weight with planes that are zero
    w[:, 1], w[:, 3], w[:, inner - 2] = 1.0, -2.0, -0.5
    w[outer // 2, 7] = float("inf")
    out = empty((rows, outer), 1)
    ops.call("f32_linear", odd.data_ptr(), w.data_ptr(), rows, inner, outer, 0, out.data_ptr(), stream())
    ops.call("check_async_errors", stream())
    expected = torch.zeros(rows, outer, dtype=torch.float64, device="cuda")
    for k in (1, 2, 3, 5, 7, inner - 2, inner - 1):  # (0 times an infinity is a NaN here too)
        expected += odd[:, k:k + 1].double() * w[:, k].double()
    assert torch.equal(out.isnan(), expected.isnan())
    assert torch.equal(out.isinf(), expected.isinf())
    finite = expected.isfinite()
    assert torch.equal(out[out.isinf()].sign().double(), expected[out.isinf()].sign())
    assert torch.allclose(out[finite].double(), expected[finite], rtol=2e-7, atol=0.0)


@pytest.mark.parametrize("spread", [0.0, 2.0])
@pytest.mark.parametrize("rows, inner", [(128, 256), (90, 2056), (40, 8448)])
def test_f32_products_of_one_sign(ops, rows, inner, spread):
    """The tensor cores' cuts do not cancel here: a block's four cuts with the largest plane take up to 2^-23 of its sum each, half
    of that on average, so results are too small by at most 4 units of 2^-24 on average, and too large by no more than the
    roundings' own mean (a tenth of a unit)."""
    rng = np.random.default_rng(inner + int(spread))
    w, wv = activation(np.abs(rng.normal(0, 1, (384, inner))), 0)
    x = np.abs(rng.normal(0, 1, (rows, inner)) * np.exp(rng.normal(0, 1, (rows, inner)) * spread)).astype(np.float32)
    exact, out = cuda(x), empty((rows, 384), 1)
    ops.call("f32_linear", exact.data_ptr(), w.data_ptr(), rows, inner, 384, 0, out.data_ptr(), stream())
    expected = x.astype(np.float64) @ wv.T
    mean = np.mean((out.double().cpu().numpy() - expected) / expected)
    assert -4 * 2.0 ** -24 <= mean <= 0.1 * 2.0 ** -24


@pytest.mark.parametrize("exponent", [-100, -110, -118, -126, -132, -140, -149])
def test_f32_products_of_the_smallest_values(ops, exponent):
    """What lies below 2^-133 of a value is lost, and nothing else: 2^-133 of a weight beside the bound of other values and half
    of the smallest F32 number per addition."""
    rng = np.random.default_rng(-exponent)
    rows, inner, outer = 40, 264, 130
    w, wv = activation(rng.normal(0, 1, (outer, inner)) * np.exp2(rng.integers(0, 30, (outer, 1))), 0)
    x = (rng.normal(0, 1, (rows, inner)) * 2.0 ** exponent).astype(np.float32)
    exact, out = cuda(x), empty((rows, outer), 1)
    ops.call("f32_linear", exact.data_ptr(), w.data_ptr(), rows, inner, outer, 0, out.data_ptr(), stream())
    xv = x.astype(np.float64)
    error = np.abs(out.double().cpu().numpy() - xv @ wv.T)
    bound = (24 + inner / 512) * 2.0 ** -24 * (np.abs(xv) @ np.abs(wv).T) + 2.0 ** -133 * np.abs(wv).sum(1) + inner * 2.0 ** -150
    assert np.all(error <= bound)


def projected(pkg, ops, x, w, float32, **more):
    """x . W^T through the kernels of the F32 profile (1: F32 rows, 2: BF16 rows)."""
    import ctypes

    out = empty((x.shape[0], w.shape[-2]), 1)
    args = pkg.Projection(input=x.data_ptr(), weight=w.data_ptr(), output=out.data_ptr(), rows=x.shape[0], in_features=w.shape[-1],
                          out_features=w.shape[-2], alpha=1.0, float32=float32, f32_result=1, row_fanout=1, **more)
    ops.call("projection", ctypes.addressof(args), stream())
    return out


@pytest.mark.parametrize("float32", [1, 2], ids=["f32", "bf16"])
@pytest.mark.parametrize("rows, inner, outer", [(17, 64, 127), (96, 200, 129), (97, 1080, 260), (128, 2048, 40), (40, 4104, 2049)])
def test_products_of_rows_and_weights_that_are_not_finite(pkg, ops, float32, rows, inner, outer):
    """Infinities and NaNs come out as multiply-adds give them, whole rows of them, NaNs whose payload lies in their lower half,
    columns with infinite weights (some meet infinite values) and with a NaN; everything else is as if they were not there."""
    import torch

    rng = np.random.default_rng(rows + inner)
    x, w = cuda(rng.normal(0, 1, (rows, inner)).astype(np.float32)), cuda(rng.normal(0, 1, (outer, inner)).astype(np.float32)).bfloat16()
    inf, nan = float("inf"), float("nan")
    x[0], x[1, inner // 2], x[2, 5], x[3, inner - 1] = nan, nan, inf, -inf
    x[4, 9], x[4, inner - 4] = inf, -inf
    x[5], x[6, ::2], x[7, 8] = inf, -inf, 3e38
    w[1, 5], w[outer // 2, 8], w[outer - 1, inner - 1], w[3, 6], w[7, 5] = inf, inf, -inf, nan, 0.0
    x[8, 6], x[8, 8] = 0.0, 1.5
    w[4] = 2.0 ** -20 * w[4]
    w[4, 5:9] = 2.0 ** -100
    if float32 == 1:
        x.view(torch.int32)[9, 3], x.view(torch.int32)[10, inner - 2] = 0x7f800001, -0x007ffffe   # NaNs with one bit below
    else:
        x = x.bfloat16()
    out = projected(pkg, ops, x, w, float32)
    ops.call("check_async_errors", stream())
    expected = torch.zeros(rows, outer, dtype=torch.float64, device="cuda")
    for begin in range(0, inner, 64):  # (products before sums: infinities that meet zeros)
        expected += (x[:, None, begin:begin + 64].double() * w[None, :, begin:begin + 64].double()).sum(2)
    assert torch.equal(out.isnan(), expected.isnan())
    bound = expected.abs() > 3e38  # (finite in 64 bits, not in 32)
    assert torch.equal(out.isinf() | bound, expected.isinf() | bound)
    assert torch.equal(out[expected.isinf()].sign().double(), expected[expected.isinf()].sign())
    finite = expected.isfinite() & ~bound
    magnitudes = torch.nan_to_num(x.double().abs(), 0.0, 0.0) @ torch.nan_to_num(w.double().abs(), 0.0, 0.0).T
    assert bool(((out.double() - expected).abs() <= (24 + inner / 512) * 2.0 ** -24 * magnitudes)[finite].all())
    if float32 == 1:  # added to an old result: once, whichever way a result took
        old = torch.randn(rows, outer, device="cuda")
        added = old.clone()
        ops.call("f32_linear", x.data_ptr(), w.data_ptr(), rows, inner, outer, 1, added.data_ptr(), stream())
        assert torch.equal(added.isnan(), out.isnan()) and torch.equal(added.isinf(), out.isinf())
        sums = old + out
        assert torch.equal(added[sums.isfinite()], sums[sums.isfinite()])


def test_rows_that_fill_up_a_tile_cost_no_more_than_rows(pkg, ops):
    """An expert's tile holds a live row and what lay in the workspace: its values change nothing, and NaNs and infinities no
    more than the time of another pass over the weights and a slower unpacking (every result made again: 34 times as long)."""
    import torch

    experts, inner, outer = 8, 2048, 2816
    w = torch.randn(experts, outer, inner, device="cuda").bfloat16()
    group, count = torch.arange(experts, device="cuda", dtype=torch.int32), torch.tensor([experts], device="cuda", dtype=torch.int32)
    live = torch.randn(experts, inner, device="cuda")
    seen = []
    for fill in (0.5, float("nan"), float("inf")):
        x = torch.full((experts, 128, inner), fill, device="cuda")
        x[:, 0] = live
        call = lambda: projected(pkg, ops, x.view(-1, inner), w, 1, groups=experts, tile_group=group.data_ptr(),
                                 tile_count=count.data_ptr(), tile_rows=128)
        out = call().view(experts, 128, outer)[:, 0].clone()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            call()
        times = []
        for _ in range(8):
            begin, end = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            begin.record()
            graph.replay()
            end.record()
            torch.cuda.synchronize()
            times.append(begin.elapsed_time(end))
        seen.append((out, min(times)))
    assert all(torch.equal(out, seen[0][0]) and time < 6 * seen[0][1] for out, time in seen), [time for _, time in seen]


@pytest.mark.parametrize("rows, fanout, inner, outer", [(2, 2, 264, 4099), (4, 2, 72, 6146), (8, 4, 2048, 2056), (12, 3, 1024, 4096)])
def test_a_few_rows_that_share_inputs(pkg, ops, rows, fanout, inner, outer):
    """row_fanout without groups, at sizes at which other rows go to other kernels: row r is input row r / row_fanout, of which there
    are no more than that.  Chains of inner / 32 products, a sum over 32 lanes."""
    import ctypes

    rng = np.random.default_rng(rows + inner)
    (x, xv), (w, wv) = activation(rng.normal(0, 1, (rows // fanout, inner)), 1), activation(rng.normal(0, 1, (outer, inner)), 0)
    out = empty((rows, outer), 1)
    args = pkg.Projection(input=x.data_ptr(), weight=w.data_ptr(), output=out.data_ptr(), rows=rows, in_features=inner,
                          out_features=outer, alpha=1.0, float32=1, f32_result=1, row_fanout=fanout)
    ops.call("projection", ctypes.addressof(args), stream())
    bound = (inner / 32 + 8) * 2.0 ** -24 * (np.abs(xv) @ np.abs(wv).T)
    assert np.all(np.abs(out.double().cpu().numpy() - (xv @ wv.T).repeat(fanout, 0).reshape(rows, outer)) <= bound.repeat(fanout, 0))


@pytest.mark.parametrize("float32", [1, 2], ids=["f32", "bf16"])
@pytest.mark.parametrize("rows, inner, outer", [(2, 8, 4096), (2, 264, 4099), (3, 2056, 4096), (3, 256, 4097), (4, 520, 6144), (4, 72, 6146)])
def test_a_few_wide_rows(pkg, ops, float32, rows, inner, outer):
    """Three columns a warp, with remainders of columns and of the inner size, bias, alpha and soft cap.  A chain of products has
    ceil(inner / 256) * 8 terms, the lanes' sum five and the epilogue three: so many units of 2^-24 of the magnitudes, and the
    soft cap's own 4 of its bound."""
    import ctypes
    import torch

    rng = np.random.default_rng(rows + inner + outer)
    (x, xv), (w, wv) = activation(rng.normal(0, 1, (rows, inner)), float32 == 1), activation(rng.normal(0, 1, (outer, inner)), 0)
    bias = rng.normal(0, 1, outer).astype(np.float32)
    db, out = cuda(bias), empty((rows, outer), 1)
    for softcap in (0.0, 50.0):
        args = pkg.Projection(input=x.data_ptr(), weight=w.data_ptr(), output=out.data_ptr(), bias=db.data_ptr(), rows=rows,
                              in_features=inner, out_features=outer, alpha=0.5, softcap=softcap, float32=float32, f32_result=1,
                              row_fanout=1)
        ops.call("projection", ctypes.addressof(args), stream())
        expected = 0.5 * (xv @ wv.T) + bias
        bound = (8 * -(-inner // 256) + 8) * 2.0 ** -24 * (0.5 * (np.abs(xv) @ np.abs(wv).T) + np.abs(bias))
        if softcap:
            expected, bound = softcap * np.tanh(expected / softcap), bound + 4 * 2.0 ** -23 * softcap
        assert np.all(np.abs(out.double().cpu().numpy() - expected) <= bound)


def test_few_f32_rows_cost_less_than_a_tile(ops):
    """Two rows are a stream of the weights, 32 a tile (7.4 us against 15.7 at this size, on the GPU alone: a call through ctypes
    can take as long as the two rows)."""
    import torch

    w = torch.randn(8448, 2048, device="cuda").bfloat16()

    def microseconds(rows):
        x, out = torch.randn(rows, 2048, device="cuda"), torch.empty(rows, 8448, device="cuda")
        graph, times = torch.cuda.CUDAGraph(), []
        with torch.cuda.graph(graph):
            for _ in range(10):
                ops.call("f32_linear", x.data_ptr(), w.data_ptr(), rows, 2048, 8448, 0, out.data_ptr(), stream())
        for _ in range(12):
            begin, end = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            begin.record()
            graph.replay()
            end.record()
            torch.cuda.synchronize()
            times.append(begin.elapsed_time(end))
        return min(times)

    assert microseconds(2) < 0.5 * microseconds(32)


# ---------------------------------------------------------------- attention
def window_case(pkg, ops, *, rows, position, heads, kv_heads, dim, vdim, window, keep_first, kernel, float32=0, softcap=15.0,
                sink=1, gated=True, biased=True, seed=0, edit=None):
    """Runs one call; returns (output, expected [rows, heads, vdim]).  `edit(q, k, v)` may plant values."""
    rng = np.random.default_rng(seed)
    total, capacity = position + rows, position + rows + 5
    q = rng.normal(0, 1, (rows, heads, dim))
    k = rng.normal(0, 1, (capacity, kv_heads, dim))
    v = rng.normal(0, 1, (capacity, kv_heads, vdim))
    if edit is not None:
        edit(q, k, v)
    k[total:], v[total:] = 1e4, 1e4                                 # what lies behind the last key is never read
    (dq, q), (dk, k), (dv, v) = (activation(x, float32) for x in (q, k, v))
    gate, gv = activation(rng.normal(0, 1, (rows, heads + 3)), float32)
    r1, r2 = rng.uniform(0.1, 0.8, heads), rng.uniform(0.05, 1.0, heads)
    bias = (r1[:, None] * np.log1p(r2[:, None] * np.arange(total))).astype(np.float32)
    db, out = cuda(bias), empty((rows, heads, vdim), float32)
    scale = dim ** -0.5
    import ctypes

    args = pkg.WindowAttention(query=dq.data_ptr(), key_cache=dk.data_ptr(), value_cache=dv.data_ptr(),
                               gate=gate.data_ptr() if gated else None, gate_stride=heads + 3,
                               distance_bias=db.data_ptr() if biased else None, bias_stride=total, output=out.data_ptr(),
                               rows=rows, position=position, capacity=capacity, heads=heads, kv_heads=kv_heads, dim=dim,
                               value_dim=vdim, window=window, keep_first=keep_first, scale=scale, softcap=softcap, sink=sink,
                               float32=float32, kernel=kernel)
    ops.call("window_attention", ctypes.addressof(args), stream())
    ops.call("check_async_errors", stream())
    expected = np.zeros((rows, heads, vdim))
    for r in range(rows):
        i = position + r
        seen = oracle.visible_keys(i, window if window else i + 1, keep_first)
        for h in range(heads):
            s = (k[seen, h // (heads // kv_heads)] @ q[r, h]) * scale
            if softcap:
                s = softcap * np.tanh(s / softcap)
            if biased:
                s = s - r1[h] * np.log1p(r2[h] * (i - seen))
            p = oracle.softmax_with_sink(s) if sink else np.exp(s - s.max()) / np.exp(s - s.max()).sum()
            expected[r, h] = p @ v[seen, h // (heads // kv_heads)]
        if gated:
            expected[r] *= oracle.sigmoid(gv[r, :heads])[:, None]
    return out, expected


ROW, TILE, TENSOR = 1, 2, 3


@TYPES
@pytest.mark.parametrize("kernel", [ROW, TILE], ids=["row", "tile"])
@pytest.mark.parametrize("heads, kv_heads, dim, vdim", [(6, 2, 40, 24), (3, 1, 17, 5), (4, 4, 200, 136), (2, 1, 96, 256),
                                                         (8, 2, 64, 72)])
def test_attention_sizes(pkg, ops, float32, kernel, heads, kv_heads, dim, vdim):
    for rows, position in ((1, 0), (1, 61), (7, 30), (45, 3)):
        out, expected = window_case(pkg, ops, rows=rows, position=position, heads=heads, kv_heads=kv_heads, dim=dim, vdim=vdim,
                                    window=21, keep_first=3, kernel=kernel, float32=float32, seed=rows)
        assert_near(out, expected, float32)


@pytest.mark.parametrize("dim, vdim", [(64, 64), (96, 96), (128, 72), (72, 128), (128, 128)])
@pytest.mark.parametrize("rows, position, window, keep_first", [
    (1, 0, 7, 0), (130, 0, 64, 4), (200, 0, 0, 0), (150, 300, 96, 6), (64, 500, 65, 70), (300, 1, 128, 1), (129, 63, 1, 0),
    (257, 700, 200, 129)])
def test_attention_tensor_cores(pkg, ops, dim, vdim, rows, position, window, keep_first):
    out, expected = window_case(pkg, ops, rows=rows, position=position, heads=4, kv_heads=2, dim=dim, vdim=vdim, window=window,
                                keep_first=keep_first, kernel=TENSOR)
    assert_near(out, expected, 0, factor=2.0)                       # the probabilities are BF16 operands as well


@pytest.mark.parametrize("kernel", [ROW, TILE, TENSOR])
@pytest.mark.parametrize("softcap, sink, gated, biased", [(0.0, 1, True, True), (90.0, 1, True, True), (1.5, 1, True, True), (3.0, 0, True, True), (15.0, 1, False, True),
                                                           (15.0, 1, True, False), (0.0, 0, False, False)])
def test_attention_options(pkg, ops, kernel, softcap, sink, gated, biased):
    out, expected = window_case(pkg, ops, rows=70, position=90, heads=4, kv_heads=1, dim=64, vdim=80, window=33, keep_first=2,
                                kernel=kernel, softcap=softcap, sink=sink, gated=gated, biased=biased)
    assert_near(out, expected, 0)


@pytest.mark.parametrize("kernel", [ROW, TILE, TENSOR])
@pytest.mark.parametrize("key_at", ["oldest in the window", "just outside", "last kept", "first after the kept", "own", "next"])
def test_one_key_stands_out(pkg, ops, kernel, key_at):
    """One key that every query scores far above the rest, at the edges of what a query sees: its value dominates
    exactly where it is visible."""
    rows, position, window, keep = 140, 200, 50, 5
    target = {"oldest in the window": position + 60 - window + 1, "just outside": position + 60 - window,
              "last kept": keep - 1, "first after the kept": keep, "own": position + 60, "next": position + 61}[key_at]

    def plant(q, k, v):
        q[..., 0], k[..., 0] = 4.0, 0.0
        k[target, :, 0], v[target] = 20.0, 9.0

    out, expected = window_case(pkg, ops, rows=rows, position=position, heads=4, kv_heads=2, dim=64, vdim=64, window=window,
                                keep_first=keep, kernel=kernel, gated=False, softcap=30.0, edit=plant)
    visible = np.array([target <= i and (i - target < window or target < keep) for i in range(position, position + rows)])
    assert_near(out, expected, 0)
    mean = out.float().cpu().numpy().mean(axis=(1, 2))
    assert (mean[visible] > 3.0).all() and (np.abs(mean[~visible]) < 1.0).all()
    # the query at index 60 is the one whose edge the key lies on
    assert visible[60] == (key_at in ("oldest in the window", "last kept", "own"))


@pytest.mark.parametrize("kernel", [ROW, TILE, TENSOR])
def test_the_sink_alone(pkg, ops, kernel):
    """Scores far below zero leave almost everything to the sink."""
    def plant(q, k, v):
        q[..., 0], k[..., 0], v[:] = 10.0, -20.0, 5.0

    out, expected = window_case(pkg, ops, rows=66, position=10, heads=2, kv_heads=1, dim=64, vdim=64, window=16, keep_first=1,
                                kernel=kernel, gated=False, softcap=12.0, edit=plant)
    assert np.abs(out.float().cpu().numpy()).max() < 1e-2 and np.abs(expected).max() < 1e-2


def test_attention_refusals(pkg, ops):
    with pytest.raises(pkg.OpsError) as error:
        window_case(pkg, ops, rows=40, position=0, heads=2, kv_heads=1, dim=40, vdim=64, window=8, keep_first=0, kernel=TENSOR)
    assert error.value.code == 5
    for size in ("dim", "vdim"):                                     # wide heads run in the row kernel only
        with pytest.raises(pkg.OpsError) as error:
            window_case(pkg, ops, **(dict(rows=2, position=0, heads=2, kv_heads=1, dim=16, vdim=16, window=8, keep_first=0,
                                          kernel=TILE) | {size: 300}))
        assert error.value.code == 5
    for bad in (dict(heads=3, kv_heads=2), dict(dim=1032), dict(softcap=-1.0)):
        case = dict(rows=2, position=0, heads=2, kv_heads=1, dim=16, vdim=16, window=8, keep_first=0, kernel=0) | bad
        with pytest.raises(pkg.OpsError) as error:
            window_case(pkg, ops, **case)
        assert error.value.code == 2


@TYPES
@pytest.mark.parametrize("dim, vdim", [(40, 24), (17, 33), (128, 200)])
def test_head_norms_and_cache_rows(pkg, ops, float32, dim, vdim):
    import ctypes

    rng = np.random.default_rng(dim)
    rows, position, capacity, heads, kv_heads, eps = 5, 7, 14, 6, 2, 1e-2
    key_column = heads * dim + 3
    value_column = key_column + kv_heads * dim + 1
    stride = value_column + kv_heads * vdim + 9
    x, xv = activation(rng.normal(0, 0.3, (rows, stride)), float32)
    gq, gk = (rng.uniform(0.5, 1.5, dim).astype(np.float32) for _ in range(2))
    dq, dk = cuda(gq), cuda(gk)
    query, keys, values = (empty(s, float32) for s in ((rows, heads, dim), (capacity, kv_heads, dim), (capacity, kv_heads, vdim)))
    args = pkg.HeadNorm(projection=x.data_ptr(), stride=stride, key_column=key_column, value_column=value_column,
                        query_gain=dq.data_ptr(), key_gain=dk.data_ptr(), query=query.data_ptr(), key_cache=keys.data_ptr(),
                        value_cache=values.data_ptr(), rows=rows, position=position, capacity=capacity, heads=heads,
                        kv_heads=kv_heads, dim=dim, value_dim=vdim, epsilon=eps, float32=float32)
    ops.call("head_norm_append", ctypes.addressof(args), stream())
    assert_near(query, oracle.rms(xv[:, :heads * dim].reshape(rows, heads, dim), eps) * gq, float32)
    assert_near(keys[position:position + rows],
                oracle.rms(xv[:, key_column:key_column + kv_heads * dim].reshape(rows, kv_heads, dim), eps) * gk, float32)
    assert bool((values[position:position + rows].reshape(rows, -1) ==
                 x[:, value_column:value_column + kv_heads * vdim]).all())
    assert bool(keys[:position].isnan().all()) and bool(values[position + rows:].isnan().all())   # neighbours untouched
    args.position = capacity - rows + 1
    assert ops.status("head_norm_append", ctypes.addressof(args), stream()) == 2


# ---------------------------------------------------------------- recurrences
class Recurrence:
    """One recurrent mixer with random inputs; run() pushes the next rows through it."""

    def __init__(self, pkg, ops, *, delta, rows, heads, kv_heads, dim, vdim, float32, taps=4, rank=5, tau=9.0, seed=0,
                 projection_scale=1.0):
        self.pkg, self.ops = pkg, ops
        rng = np.random.default_rng(seed)
        up = lambda n: (n + 7) // 8 * 8
        self.delta, self.heads, self.kv_heads, self.dim, self.vdim, self.float32 = delta, heads, kv_heads, dim, vdim, float32
        qk = (kv_heads if delta else heads) * dim
        self.key_column = up(qk)
        self.value_column = self.key_column + up(qk)
        self.gate_column = self.value_column + up(heads * vdim)
        self.beta_column = self.gate_column + up(heads * vdim)
        self.decay_column = self.beta_column + up(heads if delta else rank)
        self.stride = self.decay_column + (up(heads) if delta else 0)
        self.taps, self.rank, self.tau, self.eps = taps, rank, tau, 1e-5
        self.projection, self.values = activation(rng.normal(0, projection_scale, (rows, self.stride)), float32)
        f32 = lambda *shape, low=-1.0, high=1.0: rng.uniform(low, high, shape).astype(np.float32)
        self.conv, self.rate, self.shift = f32(self.gate_column, taps), -np.exp(f32(heads, low=-3.0)), f32(heads)
        self.weight, self.bias, self.norm = f32(rank, heads * dim), f32(heads * dim, high=4.0), f32(vdim, low=0.5, high=1.5)
        self.device = [cuda(x) for x in (self.conv, self.rate, self.shift, self.weight, self.bias, self.norm)]
        self.state = empty((heads, dim, vdim), 1)
        self.history = empty((max(1, taps - 1), self.gate_column), float32)
        self.at = 0

    def run(self, rows):
        import ctypes

        conv, rate, shift, weight, bias, norm = self.device
        size = self.ops.lib.evo_b200_recurrent_workspace_bytes(int(self.delta), rows, self.heads, self.kv_heads, self.dim,
                                                               self.vdim, self.float32)
        work, out = empty((size // 4 + 1,), 1), empty((rows, self.heads * self.vdim), self.float32)
        part = self.projection[self.at:self.at + rows].contiguous()
        args = self.pkg.Recurrent(
            delta=int(self.delta), projection=part.data_ptr(), stride=self.stride, key_column=self.key_column,
            value_column=self.value_column, gate_column=self.gate_column, beta_column=self.beta_column,
            decay_column=self.decay_column, rows=rows, heads=self.heads, kv_heads=self.kv_heads, dim=self.dim,
            value_dim=self.vdim, conv=conv.data_ptr(), conv_taps=self.taps, conv_history=self.history.data_ptr(),
            decay_rate=rate.data_ptr(), decay_shift=shift.data_ptr(), decay_weight=weight.data_ptr(),
            decay_bias=bias.data_ptr(), decay_rank=self.rank, tau=self.tau, output_norm=norm.data_ptr(), epsilon=self.eps,
            state=self.state.data_ptr(), fresh=int(self.at == 0), workspace=work.data_ptr(), output=out.data_ptr(),
            float32=self.float32)
        self.ops.call("recurrent_mixer", ctypes.addressof(args), stream())
        self.ops.call("check_async_errors", stream())
        self.at += rows
        return out

    def restart(self):
        self.at = 0

    def expected(self, rows):
        x, H, G, dim, vdim = self.values[:rows], self.heads, self.kv_heads, self.dim, self.vdim
        cut = lambda column, n, shape: x[:, column:column + n].reshape(rows, *shape)
        gate = cut(self.gate_column, H * vdim, (H, vdim))
        if self.delta:
            mixed = oracle.silu(oracle.causal_convolution(x[:, :self.gate_column], self.conv.astype(np.float64)))
            q = oracle.unit_vectors(mixed[:, :G * dim].reshape(rows, G, dim)) * dim ** -0.5
            k = oracle.unit_vectors(mixed[:, self.key_column:self.key_column + G * dim].reshape(rows, G, dim))
            v = mixed[:, self.value_column:self.value_column + H * vdim].reshape(rows, H, vdim)
            beta = oracle.sigmoid(cut(self.beta_column, H, (H,)))
            g = np.exp(self.rate.astype(np.float64) * oracle.softplus(cut(self.decay_column, H, (H,)) + self.shift))
            o, state = oracle.gated_delta_rule(q, k, v, beta, g)
        else:
            q = cut(0, H * dim, (H, dim)) * dim ** -0.5
            k, v = cut(self.key_column, H * dim, (H, dim)), cut(self.value_column, H * vdim, (H, vdim))
            z = cut(self.beta_column, self.rank, (self.rank,)) @ self.weight.astype(np.float64) + self.bias
            alpha = np.exp(-oracle.softplus(-z) / self.tau).reshape(rows, H, dim)
            o, state = oracle.gated_linear_attention(q, k, v, alpha)
        return (oracle.rms(o, self.eps) * self.norm * oracle.silu(gate)).reshape(rows, -1), state


RECURRENT_SIZES = [(4, 2, 28, 20), (3, 3, 5, 33), (6, 1, 64, 40), (2, 2, 96, 17), (4, 1, 128, 64), (2, 1, 200, 24)]


@TYPES
@pytest.mark.parametrize("delta", [False, True], ids=["linear", "delta"])
@pytest.mark.parametrize("heads, kv_heads, dim, vdim", RECURRENT_SIZES)
def test_recurrences(pkg, ops, float32, delta, heads, kv_heads, dim, vdim):
    rows = 150
    case = Recurrence(pkg, ops, delta=delta, rows=rows, heads=heads, kv_heads=kv_heads if delta else heads, dim=dim, vdim=vdim,
                      float32=float32, taps=1 + dim % 5)
    expected, state = case.expected(rows)
    assert_near(case.run(rows), expected, float32, factor=4.0)
    assert_near(case.state, state, float32 or not delta)            # (BF16 rounds the convolved values, not the state)


@pytest.mark.parametrize("delta", [False, True], ids=["linear", "delta"])
@pytest.mark.parametrize("taps", [1, 2, 6])
@pytest.mark.parametrize("portions", [[2] * 30, [1] * 60, [16, 1, 17, 2, 24], [3, 57], [60], [5, 4, 1, 1, 1, 48]])
def test_recurrences_in_portions(pkg, ops, delta, taps, portions):
    """The state and the convolution's history carry over any cut; a restart forgets both."""
    case = Recurrence(pkg, ops, delta=delta, rows=60, heads=4, kv_heads=2 if delta else 4, dim=36, vdim=40, float32=1, taps=taps,
                      seed=3)
    expected, state = case.expected(60)
    for _ in range(2):
        parts = [case.run(n).cpu().numpy() for n in portions]
        assert_near(np.concatenate(parts).astype(np.float64), expected, 1, factor=4.0)
        assert_near(case.state, state, 1)
        case.restart()


@pytest.mark.parametrize("delta", [False, True], ids=["linear", "delta"])
def test_a_lost_state_would_show(pkg, ops, delta):
    """Slow decays: what the first tokens wrote still dominates far away."""
    case = Recurrence(pkg, ops, delta=delta, rows=300, heads=2, kv_heads=2, dim=32, vdim=16, float32=1, seed=5, tau=4000.0,
                      projection_scale=0.3)
    case.rate[:] = -1e-4
    case.device[1].copy_(cuda(case.rate))
    expected, _ = case.expected(300)
    out = np.concatenate([case.run(n).cpu().numpy() for n in (100, 1, 150, 49)]).astype(np.float64)
    assert_near(out, expected, 1, factor=6.0)
    case.restart()
    case.run(100)
    case.at = 0                                                     # forget the state: a fresh start at row 100
    case.projection = case.projection[100:].contiguous()
    forgotten = case.run(200).double().cpu().numpy()
    assert np.abs(forgotten[-50:] - expected[-50:]).max() > 1e-2


def test_extreme_gates_stay_finite(pkg, ops):
    for delta in (False, True):
        case = Recurrence(pkg, ops, delta=delta, rows=40, heads=2, kv_heads=2, dim=24, vdim=16, float32=1, projection_scale=60.0,
                          tau=0.5)
        expected, _ = case.expected(40)
        out = case.run(40).double().cpu().numpy()
        assert np.isfinite(out).all() and np.isfinite(expected).all()
        assert_near(out, expected, 1, factor=50.0)


@TYPES
@pytest.mark.parametrize("delta, heads, kv_heads, dim, vdim, taps, rank", [
    (True, 4, 1, 40, 64, 4, 5), (True, 4, 1, 40, 66, 1, 5), (True, 4, 1, 40, 66, 6, 5), (True, 16, 2, 64, 256, 2, 5),
    (True, 5, 1, 24, 512, 4, 5), (True, 3, 1, 256, 100, 6, 5), (False, 2, 2, 40, 256, 4, 3), (False, 2, 2, 40, 257, 4, 16),
    (False, 3, 3, 128, 512, 4, 17), (False, 4, 4, 256, 8, 4, 24), (False, 2, 2, 20, 264, 4, 9)])
def test_single_steps_of_wide_groups(pkg, ops, float32, delta, heads, kv_heads, dim, vdim, taps, rank):
    """32 and 33 columns a CTA and many blocks of them, taps that are held and that are not, decays of whole and partial batches
    of ranks: six tokens, one after another, carry the state and the history.  (BF16 rounds the six tokens' values, each by 2^-9 of
    itself; with terms that cancel a cell of the state can be half as large as they are: 2 6 2^-9.)"""
    case = Recurrence(pkg, ops, delta=delta, rows=6, heads=heads, kv_heads=kv_heads, dim=dim, vdim=vdim, float32=float32, taps=taps,
                      rank=rank, seed=dim + vdim + taps)
    expected, state = case.expected(6)
    assert_near(np.concatenate([case.run(1).float().cpu().numpy() for _ in range(6)]).astype(np.float64), expected, float32, factor=4.0)
    assert_near(case.state, state, float32 or not delta, factor=2.0)


@TYPES
def test_steps_with_keys_and_queries_of_infinite_length(pkg, ops, float32):
    """Squares that overflow give zero vectors: nothing is read from the state or written to it, and nothing is NaN.  A product
    of the vectors that is summed before they are scaled is infinite here."""
    case = Recurrence(pkg, ops, delta=True, rows=3, heads=4, kv_heads=2, dim=40, vdim=24, float32=float32, seed=11)
    case.conv[:] = np.abs(case.conv) + 0.1
    case.device[0].copy_(cuda(case.conv))
    case.projection[:, :case.value_column] = case.projection[:, :case.value_column].abs() * 1e20 + 1e20
    for _ in range(3):
        assert bool((case.run(1) == 0).all()) and bool((case.state == 0).all())


CAPTURED_FIRST = """
import sys
sys.path.insert(0, sys.argv[1])
import conftest, torch
ops = conftest.load_package().ops()
x, w, out = torch.randn(40, 64, device="cuda"), torch.randn(96, 64, device="cuda").bfloat16(), torch.zeros(40, 96, device="cuda")
torch.cuda.synchronize()
graph, side = torch.cuda.CUDAGraph(), torch.cuda.Stream()
with torch.cuda.graph(graph, stream=side):
    ops.call("f32_linear", x.data_ptr(), w.data_ptr(), 40, 64, 96, 0, out.data_ptr(), side.cuda_stream)
graph.replay()
torch.cuda.synchronize()
exact = x.double() @ w.double().T
assert float((out - exact).abs().max()) <= 32 * 2.0 ** -24 * float((x.double().abs() @ w.double().abs().T).max())
"""


def test_first_product_of_a_process_can_be_captured():
    """The per-device error word is made by the first kernel that needs it, also while the caller captures that launch."""
    import subprocess
    import sys
    from pathlib import Path

    run = subprocess.run([sys.executable, "-c", CAPTURED_FIRST, str(Path(__file__).parent)], capture_output=True, text=True, timeout=300)
    assert run.returncode == 0, run.stderr[-2000:]
