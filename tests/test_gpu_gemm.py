"""GPU parity of the tcgen05 / CUDA-core projections through the C ABI.

Small shapes are checked against the CPU oracle; shapes too large for it are
checked against an F32 matmul of the same BF16 operands (tolerance 0.02 abs +
0.02 rel, the gate upstream applies to its cuBLASLt linear,
tests/test_cuda_ops.cu:252-369)."""
from __future__ import annotations

import ctypes

import numpy as np
import pytest
import torch

from gpu_util import assert_close_bits, dev, dev_bits, empty_bits, host_bits, p, rand_bf16, stream
from oracle_lib import bf16_to_f32, f32_to_bf16, ptr

pytestmark = pytest.mark.gpu


def _linear(ops, x, w, bias, residual, bias_mode, path):
    rows, inner = x.shape
    columns = w.shape[0]
    out = empty_bits(rows, columns)
    ops.call("bf16_linear", p(x), p(w), p(bias), p(residual), rows, inner, columns, bias_mode,
             path, p(out), stream())
    ops.call("check_async_errors", stream())
    return out


@pytest.mark.parametrize("path", [0, 1])
@pytest.mark.parametrize("rows,inner,columns", [(128, 256, 256), (200, 1920, 640), (16, 4096, 512),
                                               (1, 256, 128), (333, 320, 1000)])
def test_bf16_linear_against_oracle(ops, oracle, rows, inner, columns, path):
    rng = np.random.default_rng(rows + inner + columns)
    x, w = rand_bf16(rng, rows, inner), rand_bf16(rng, columns, inner, scale=0.05)
    bias, residual = rand_bf16(rng, columns), rand_bf16(rng, rows, columns)
    dx, dw, db, dr = dev_bits(x), dev_bits(w), dev_bits(bias), dev_bits(residual)
    for bias_mode, use_residual in [(0, False), (1, False), (2, True), (1, True)]:
        out = _linear(ops, dx, dw, db if bias_mode else None, dr if use_residual else None,
                      bias_mode, path)
        expected = np.empty((rows, columns), np.uint16)
        oracle.linear_bf16(ptr(x), ptr(w), ptr(bias) if bias_mode else None,
                           ptr(residual) if use_residual else None, rows, inner, columns,
                           bias_mode, ptr(expected))
        assert_close_bits(host_bits(out), expected, atol=0.02, rtol=0.02, min_cosine=0.9999)


def test_bf16_linear_tiny_fixture_shapes_use_cuda_core_path(ops, oracle):
    """Width 8 / inner 12 (the 50-layer test fixture) cannot be described to TMA."""
    rng = np.random.default_rng(1)
    for rows, inner, columns in [(4, 8, 24), (9, 12, 8), (1, 8, 512)]:
        x, w = rand_bf16(rng, rows, inner), rand_bf16(rng, columns, inner)
        out = _linear(ops, dev_bits(x), dev_bits(w), None, None, 0, 0)
        expected = np.empty((rows, columns), np.uint16)
        oracle.linear_bf16(ptr(x), ptr(w), None, None, rows, inner, columns, 0, ptr(expected))
        assert_close_bits(host_bits(out), expected, atol=0.02, rtol=0.02)


@pytest.mark.parametrize("rows,inner,columns", [(1024, 4096, 4096), (8192, 4096, 512), (2048, 11264, 4096),
                                               (1000, 1920, 5760)])
def test_bf16_linear_large_against_f32_matmul(ops, rows, inner, columns):
    torch.manual_seed(rows)
    x = torch.randn(rows, inner, device="cuda").bfloat16()
    w = (torch.randn(columns, inner, device="cuda") * 0.02).bfloat16()
    out = torch.empty(rows, columns, device="cuda", dtype=torch.bfloat16)
    ops.call("bf16_linear", p(x), p(w), None, None, rows, inner, columns, 0, 0, p(out), stream())
    ops.call("check_async_errors", stream())
    reference = x.float() @ w.float().T
    error = (out.float() - reference).abs()
    bound = 0.02 + 0.02 * reference.abs()
    assert bool((error <= bound).all()), float((error - bound).max())
    cosine = torch.nn.functional.cosine_similarity(out.float().flatten(), reference.flatten(), dim=0)
    assert float(cosine) > 0.99995


def test_pair_kernel_epilogues_at_ragged_sizes(ops):
    """600 rows (two full pair tiles and a ragged third) x 6400 / 12800 columns run on CTA pairs.
    Gated: the fused up-projection equals two linears and the gate bit for bit (same accumulators,
    same rounding points).  Bias + residual: against an F32 matmul with the BF16 rounding chain."""
    torch.manual_seed(600)
    rows, inner, hidden = 600, 512, 6400
    x = torch.randn(rows, inner, device="cuda").bfloat16()
    w1 = (torch.randn(hidden, inner, device="cuda") * 0.08).bfloat16()
    w2 = (torch.randn(hidden, inner, device="cuda") * 0.08).bfloat16()
    packed = torch.empty(2 * hidden, inner, device="cuda", dtype=torch.bfloat16)
    ops.call("interleave_gate_weights", p(w1), p(w2), hidden, inner, p(packed), stream())
    fused = torch.empty(rows, hidden, device="cuda", dtype=torch.bfloat16)
    ops.call("bf16_gated_up_projection", p(x), p(packed), rows, inner, hidden, 0, p(fused), stream())
    first, second = (torch.empty(rows, hidden, device="cuda", dtype=torch.bfloat16) for _ in range(2))
    ops.call("bf16_linear", p(x), p(w1), None, None, rows, inner, hidden, 0, 0, p(first), stream())
    ops.call("bf16_linear", p(x), p(w2), None, None, rows, inner, hidden, 0, 0, p(second), stream())
    unfused = torch.empty_like(fused)
    ops.call("bf16_gated_elementwise", p(first), p(second), rows * hidden, 0, p(unfused), stream())
    ops.call("check_async_errors", stream())
    assert torch.equal(fused.view(torch.int16), unfused.view(torch.int16))
    bias = torch.randn(hidden, device="cuda").bfloat16()
    residual = torch.randn(rows, hidden, device="cuda").bfloat16()
    out = torch.empty(rows, hidden, device="cuda", dtype=torch.bfloat16)
    ops.call("bf16_linear", p(x), p(w1), p(bias), p(residual), rows, inner, hidden, 1, 0, p(out), stream())
    ops.call("check_async_errors", stream())
    reference = ((x.float() @ w1.float().T + bias.float()).bfloat16().float() + residual.float())
    error = (out.float() - reference).abs()
    assert bool((error <= 0.03 + 0.02 * reference.abs()).all()), float(error.max())


@pytest.mark.parametrize("rows,inner,columns", [(520, 72, 4000), (520, 1920, 4225), (769, 520, 3073), (2999, 264, 2050), (1500, 128, 1920),
                                               (600, 2080, 4096), (2999, 2080, 1920)])
def test_pair_tiles_of_192_columns(ops, rows, inner, columns):
    """Sizes whose narrow tiles take no more waves than the wide ones, with remainders in every direction: BF16 results with
    bias and residual, F32 results stored and added, E4M3 operands.  The products are exact, sums of `inner` of them rounded
    to F32 (at most inner + 4 times 2^-24 of the magnitudes' sum), and once or twice to BF16 (2^-8 of the result, or of 4)."""
    torch.manual_seed(rows + inner)
    x = torch.randn(rows, inner, device="cuda").bfloat16()
    w = (torch.randn(columns, inner, device="cuda") * 0.05).bfloat16()
    bias, residual = torch.randn(columns, device="cuda").bfloat16(), torch.randn(rows, columns, device="cuda").bfloat16()
    exact, spread = x.double() @ w.double().T, (inner + 4) * 2.0 ** -24 * (x.double().abs() @ w.double().abs().T)
    out = _linear(ops, x, w, bias, residual, 1, 0).view(torch.bfloat16)
    first = exact + bias.double()
    error = (out.double() - (first + residual.double())).abs()
    assert bool((error <= spread + 2.0 ** -8 * (first.abs() + (first + residual.double()).abs() + 0.01)).all())
    base = torch.randn(rows, columns, device="cuda")
    for accumulate in (0, 1):
        sums = base.clone()
        ops.call("bf16_linear_f32_result", p(x), p(w), rows, inner, columns, accumulate, None, 0, p(sums), stream())
        ops.call("check_async_errors", stream())
        assert bool(((sums.double() - exact - accumulate * base.double()).abs() <= spread + 2.0 ** -23 * (exact.abs() + base.double().abs())).all())
    if inner % 16 == 0:
        codes = (torch.randn(columns, inner, device="cuda") * 0.5).to(torch.float8_e4m3fn)
        scratch, out = torch.empty(rows * inner, dtype=torch.uint8, device="cuda"), empty_bits(rows, columns)
        ops.call("e4m3_tensorcore_linear", p(x), p(codes), rows, inner, columns, 4.0, 0.25, p(scratch), p(out), stream())
        ops.call("check_async_errors", stream())
        rounded = (x.float() * 4.0).clamp(-448, 448).to(torch.float8_e4m3fn).double()
        exact = rounded @ codes.double().T * 0.25
        spread = (inner + 4) * 2.0 ** -24 * 0.25 * (rounded.abs() @ codes.double().abs().T)
        assert bool(((out.view(torch.bfloat16).double() - exact).abs() <= spread + 2.0 ** -8 * exact.abs()).all())


def test_gated_up_projection_matches_two_linears_and_gate(ops, oracle):
    rng = np.random.default_rng(11)
    rows, inner, hidden = 150, 256, 384
    x = rand_bf16(rng, rows, inner)
    w1, w2 = rand_bf16(rng, hidden, inner, scale=0.08), rand_bf16(rng, hidden, inner, scale=0.08)
    dx, dw1, dw2 = dev_bits(x), dev_bits(w1), dev_bits(w2)
    packed = empty_bits(2 * hidden, inner)
    ops.call("interleave_gate_weights", p(dw1), p(dw2), hidden, inner, p(packed), stream())
    for activation in (0, 1):
        out = empty_bits(rows, hidden)
        ops.call("bf16_gated_up_projection", p(dx), p(packed), rows, inner, hidden, activation,
                 p(out), stream())
        ops.call("check_async_errors", stream())
        first = _linear(ops, dx, dw1, None, None, 0, 0)
        second = _linear(ops, dx, dw2, None, None, 0, 0)
        unfused = empty_bits(rows, hidden)
        ops.call("bf16_gated_elementwise", p(first), p(second), rows * hidden, activation, p(unfused),
                 stream())
        # same accumulators, same rounding points: identical bits
        mismatch = np.flatnonzero(host_bits(out).ravel() != host_bits(unfused).ravel())
        assert mismatch.size == 0, (activation, mismatch[:8], mismatch.size)
        if activation == 0:
            expected = np.empty((rows, hidden), np.uint16)
            first_bits, second_bits = host_bits(first), host_bits(second)
            oracle.gate(ptr(first_bits), ptr(second_bits), rows * hidden, 0, ptr(expected))
            assert np.array_equal(host_bits(out), expected)


@pytest.mark.parametrize("rows,inner,columns", [(64, 256, 384), (100, 1920, 5760), (16, 4096, 12288)])
def test_e4m3_tensorcore_linear_against_exact_products(ops, oracle, rows, inner, columns):
    rng = np.random.default_rng(columns)
    x = rand_bf16(rng, rows, inner)
    w_f = (rng.standard_normal((columns, inner)) * 0.02).astype(np.float32)
    w_scale = np.float32(448.0 / np.abs(w_f).max())
    w_codes = np.empty((columns, inner), np.uint8)
    oracle.quantize_f32(ptr(w_f), w_f.size, float(w_scale), ptr(w_codes))
    in_scale = np.float32(448.0 / np.abs(bf16_to_f32(x)).max())
    out_scale = float(np.float32(1.0 / in_scale) * np.float32(1.0 / w_scale))
    scratch = torch.empty(rows * inner, dtype=torch.uint8, device="cuda")
    out = empty_bits(rows, columns)
    ops.call("e4m3_tensorcore_linear", p(dev_bits(x)), p(dev(w_codes)), rows, inner, columns,
             float(in_scale), out_scale, p(scratch), p(out), stream())
    ops.call("check_async_errors", stream())
    if rows * inner * columns <= 1.2e9:
        expected = np.empty((rows, columns), np.uint16)
        oracle.e4m3_exact_linear(ptr(x), ptr(w_codes), rows, inner, columns, float(in_scale),
                                 out_scale, ptr(expected))
        # exact E4M3 products, F32 accumulation: only summation-order rounding
        assert_close_bits(host_bits(out), expected, atol=2e-3, rtol=1e-2, min_cosine=0.99999)
    # and the emulation profile stays within the tolerance gate of the tensor-core one
    emulated = empty_bits(rows, columns)
    ops.call("software_e4m3_h100_linear", p(dev_bits(x)), p(dev(w_codes)), rows, inner, columns,
             float(in_scale), out_scale, p(scratch), p(emulated), stream())
    assert_close_bits(host_bits(out), host_bits(emulated), atol=0.02, rtol=0.02, min_cosine=0.9999)


@pytest.mark.parametrize("rows,inner,columns", [(16, 4096, 4096), (32, 4096, 12288), (24, 11264, 4096),
                                               (31, 4096, 512), (9, 2048, 1024), (64, 4096, 4096),
                                               (100, 1920, 5760), (128, 4096, 22528), (128, 11264, 4096),
                                               (48, 4096, 512), (33, 4096, 200)])
def test_split_k_projection_against_f32_matmul(ops, rows, inner, columns):
    """9..128 rows with a workspace: the weights are the 128-row tensor-core operand and the tokens
    the narrow one, K is split over several CTAs per 128 weight rows, F32 partials are added in
    split order; bias, residual and their rounding points as in the one-pass kernel."""
    torch.manual_seed(rows + columns)
    x = torch.randn(rows, inner, device="cuda").bfloat16()
    w = (torch.randn(columns, inner, device="cuda") * 0.02).bfloat16()
    bias = (torch.randn(columns, device="cuda") * 0.5).bfloat16()
    residual = torch.randn(rows, columns, device="cuda").bfloat16()
    workspace = torch.empty(8 * rows * columns, device="cuda")
    out = torch.empty(rows, columns, device="cuda", dtype=torch.bfloat16)
    plain = torch.empty_like(out)
    for bias_mode in (1, 2):
        ops.call("bf16_linear_split_k", p(x), p(w), p(bias), p(residual), rows, inner, columns, bias_mode, 0,
                 p(workspace), workspace.numel() * 4, p(out), stream())
        ops.call("bf16_linear", p(x), p(w), p(bias), p(residual), rows, inner, columns, bias_mode, 0, p(plain),
                 stream())
        ops.call("check_async_errors", stream())
        reference = x.float() @ w.float().T + bias.float() + residual.float()
        error = (out.float() - reference).abs()
        assert bool((error <= 0.03 + 0.02 * reference.abs()).all()), float(error.max())
        # the one-pass kernel rounds the same sums: at most a BF16 ulp apart where F32 sums differ
        assert float((out.float() - plain.float()).abs().max()) <= 0.07
        assert float((out != plain).float().mean()) < 0.05
    # a workspace too small for any split falls back to the one-pass kernel: identical bits
    ops.call("bf16_linear_split_k", p(x), p(w), p(bias), p(residual), rows, inner, columns, 2, 0, p(workspace), 64,
             p(out), stream())
    assert torch.equal(out, plain)


def test_split_k_gated_up_projection(ops):
    torch.manual_seed(5)
    for rows, inner, hidden in ((28, 4096, 2048), (100, 4096, 11264)):
        _check_split_k_gated(ops, rows, inner, hidden)


def _check_split_k_gated(ops, rows, inner, hidden):
    x = torch.randn(rows, inner, device="cuda").bfloat16()
    w1 = (torch.randn(hidden, inner, device="cuda") * 0.02).bfloat16()
    w2 = (torch.randn(hidden, inner, device="cuda") * 0.02).bfloat16()
    packed = torch.empty(2 * hidden, inner, device="cuda", dtype=torch.bfloat16)
    ops.call("interleave_gate_weights", p(w1), p(w2), hidden, inner, p(packed), stream())
    workspace = torch.empty(8 * rows * 2 * hidden, device="cuda")
    for activation in (0, 1):
        split = torch.empty(rows, hidden, device="cuda", dtype=torch.bfloat16)
        fused = torch.empty_like(split)
        ops.call("bf16_linear_split_k", p(x), p(packed), None, None, rows, inner, 2 * hidden, 0, activation + 1,
                 p(workspace), workspace.numel() * 4, p(split), stream())
        ops.call("bf16_gated_up_projection", p(x), p(packed), rows, inner, hidden, activation, p(fused), stream())
        ops.call("check_async_errors", stream())
        first = (x.float() @ w1.float().T).bfloat16().float()
        if activation == 1:
            first = torch.nn.functional.gelu(first).bfloat16().float()
        reference = first * (x.float() @ w2.float().T).bfloat16().float()
        # a BF16 ulp of the product where a factor rounded the other way (values reach ~10 at 1.1 M outputs)
        assert bool(((split.float() - reference).abs() <= 0.05 + 0.02 * reference.abs()).all())
        assert bool(((split.float() - fused.float()).abs() <= 0.05 + 0.02 * fused.float().abs()).all())
        assert float((split != fused).float().mean()) < 0.05


@pytest.mark.parametrize("columns", [1, 37, 256, 1184, 5000])
@pytest.mark.parametrize("inner", [64, 264, 1920, 2056, 4104, 6152, 8192, 8448, 11264, 14336, 16384, 16392])
def test_one_row_streams(ops, inner, columns):
    """One row at the edges of its kernels: fewer columns than CTAs, pieces of 8 (16) values that leave lanes or whole
    warps without work, every number of pieces per thread of the F32 weight stream (1, 2, 3, 4, 5, 6 and 8), and an inner
    size beyond its registers.  A result passes through as many roundings as the kernel that takes the size chains."""
    lanes = 8 * (-(-inner // 256)) + 5 + 2                     # a warp per output: a lane's products, the lanes, the base
    stream_chain = 8 + 7 + 5 + 3 + 2                           # a piece's products, the pieces, lanes, warps, the base
    f32_chain = stream_chain if 1024 <= inner <= 16384 else lanes
    bf16_chain = 8 * (-(-inner // 2048)) + 5 + 8 + 2           # a CTA per four outputs: a thread's products, lanes, warps
    e4m3_chain = 16 * (-(-inner // 4096)) + 5 + 8 + 2
    generator = torch.Generator("cuda").manual_seed(inner + columns)
    x, w = (torch.randn(n, inner, device="cuda", generator=generator) for n in (1, columns))
    xb, wb = x.bfloat16(), w.bfloat16()
    base = torch.randn(1, columns, device="cuda", generator=generator)

    def check(out, left, right, add, chain):
        left, right = left.double(), right.double()
        bound = chain * 2.0 ** -24 * (left.abs() @ right.abs().T + add.double().abs())
        assert bool(((out.double() - (left @ right.T + add)).abs() <= bound).all())

    out = base.clone()
    ops.call("f32_linear", p(x), p(wb), 1, inner, columns, 1, p(out), stream())
    check(out, x, wb, base, f32_chain)
    work = torch.empty(1 << 20, device="cuda")
    ops.call("bf16_linear_f32_result", p(xb), p(wb), 1, inner, columns, 0, p(work), work.numel() * 4, p(out), stream())
    check(out, xb, wb, torch.zeros_like(base), bf16_chain)
    bits = torch.empty(1, columns, dtype=torch.bfloat16, device="cuda")
    if inner % 16 == 0:
        codes, weights = (t.to(torch.float8_e4m3fn) for t in (x, w))
        ops.call("e4m3_codes_linear", p(codes.view(torch.uint8)), None, p(weights.view(torch.uint8)), None, None, 1, inner,
                 columns, 1.0, 0, 0, p(bits), stream())
        expected = codes.double() @ weights.double().T
        bound = 2.0 ** -8 * expected.abs() + e4m3_chain * 2.0 ** -24 * (codes.double().abs() @ weights.double().abs().T)
        assert bool(((bits.double() - expected).abs() <= bound).all())
    if columns % 128 == 0:
        pair = torch.randn(2 * columns, inner, device="cuda", generator=generator).bfloat16()
        ops.call("bf16_gated_up_projection", p(xb), p(pair), 1, inner, columns, 0, p(bits), stream())
        first, second = (xb.double() @ pair.view(-1, 2, 128, inner)[:, i].reshape(columns, inner).double().T for i in (0, 1))
        # both factors and the product are rounded to BF16 (2^-8 each), behind F32 sums with the bound above
        slack = bf16_chain * 2.0 ** -24 * inner
        bound = 3.1 * 2.0 ** -8 * (first * second).abs() + slack * (first.abs() + second.abs())
        assert bool(((bits.double() - first * second).abs() <= bound).all())
    ops.call("check_async_errors", stream())


@pytest.mark.parametrize("columns", [8192, 8201])
@pytest.mark.parametrize("inner", [528, 4224, 12288, 14336, 16400, 24576, 24592])
def test_one_row_e4m3_streams(ops, inner, columns):
    """Every number of pieces per thread of the E4M3 weight stream (1 to 6) and an inner size beyond it."""
    generator = torch.Generator("cuda").manual_seed(inner + columns)
    x, w = (torch.randn(n, inner, device="cuda", generator=generator).to(torch.float8_e4m3fn) for n in (1, columns))
    out = torch.empty(1, columns, dtype=torch.bfloat16, device="cuda")
    ops.call("e4m3_codes_linear", p(x.view(torch.uint8)), None, p(w.view(torch.uint8)), None, None, 1, inner, columns, 1.0, 0,
             0, p(out), stream())
    ops.call("check_async_errors", stream())
    xd, wd = x.double(), w.double()
    expected = xd @ wd.T
    # a piece's products, the pieces, lanes and warps; beyond the stream a thread's products, lanes and warps
    chain = 16 + 5 + 5 + 3 if inner <= 24576 else 16 * (-(-inner // 4096)) + 5 + 8
    bound = 2.0 ** -8 * expected.abs() + chain * 2.0 ** -24 * (xd.abs() @ wd.abs().T)
    assert bool(((out.double() - expected).abs() <= bound).all())


@pytest.mark.parametrize("columns", [5, 300, 1184])
@pytest.mark.parametrize("inner", [264, 1032, 2056, 4104, 6152, 8200, 11264, 14336, 16384, 16392])
def test_grouped_row_streams(pkg, ops, inner, columns):
    """Rows with a weight each: every number of pieces per thread of the BF16 weight stream (1, 2, 3, 4, 5, 6 and 8), and
    sizes on either side of it."""
    generator = torch.Generator("cuda").manual_seed(inner + columns)
    x = torch.randn(2, inner, device="cuda", generator=generator).bfloat16()
    w = torch.randn(3, columns, inner, device="cuda", generator=generator).bfloat16()
    group = torch.tensor([2, 0, 1, 2], dtype=torch.int32, device="cuda")
    out = torch.empty(4, columns, device="cuda")
    arguments = pkg.Projection(input=p(x), weight=p(w), output=p(out), rows=4, in_features=inner, out_features=columns, alpha=1.0,
                               f32_result=1, row_group=p(group), row_fanout=2, groups=3)
    ops.call("projection", ctypes.addressof(arguments), stream())
    ops.call("check_async_errors", stream())
    chain = 8 + 7 + 5 + 3 + 1 if 1024 <= inner <= 16384 else 8 * (-(-inner // 2048)) + 5 + 8 + 1
    for r in range(4):
        xd, wd = x[r // 2].double(), w[group[r]].double()
        assert bool(((out[r].double() - wd @ xd).abs() <= chain * 2.0 ** -24 * (wd.abs() @ xd.abs())).all())
