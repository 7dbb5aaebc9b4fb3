"""The bit-exact E4M3 projection at the edges of its kernels: one and two rows with two and four lanes per column,
row tiles of 16, 32 and 64 with remainders, one group of 32 products and several, operands that are zero, subnormal,
of extreme exponents, or cancel.  Every result equals the scalar restatement of the accumulation bit for bit."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from gpu_util import dev, dev_bits, empty_bits, host_bits, p, stream
from oracle_lib import f32_to_bf16, ptr

pytestmark = pytest.mark.gpu


def _codes(rng, kind, shape):
    codes = rng.integers(0, 256, shape).astype(np.uint8)
    if kind == "sparse":  # whole groups without a product
        codes[rng.random(shape) < 0.95] = 0
    elif kind == "subnormal":
        codes &= 0x87
    elif kind == "extreme":  # the smallest next to the largest
        codes = np.where(rng.random(shape) < 0.5, rng.choice([0x01, 0x81], shape), rng.choice([0x7e, 0xfe], shape))
    elif kind == "cancel":  # one magnitude, either sign
        codes = np.where(rng.random(shape) < 0.5, 0x3f, 0xbf)
    codes = codes.astype(np.uint8)
    codes[(codes & 0x7f) == 0x7f] ^= 1  # no NaN
    return np.ascontiguousarray(codes)


@pytest.mark.parametrize("kind", ["any", "sparse", "subnormal", "extreme", "cancel"])
@pytest.mark.parametrize("rows,inner,columns", [(1, 32, 33), (1, 544, 70), (2, 96, 31), (1, 64, 18944), (2, 32, 18950),
                                               (3, 32, 5), (16, 160, 65), (17, 96, 64), (33, 64, 129), (65, 32, 9409),
                                               (128, 64, 9472), (125, 64, 9473), (509, 32, 2433)])
def test_emulated_projection_at_kernel_edges(ops, oracle, rows, inner, columns, kind):
    rng = np.random.default_rng(rows * 31 + inner + columns)
    x, w = _codes(rng, kind, (rows, inner)), _codes(rng, kind, (columns, inner))
    values = torch.from_numpy(x).view(torch.float8_e4m3fn).float().numpy()
    scratch = torch.empty(x.size, dtype=torch.uint8, device="cuda")
    out = empty_bits(rows, columns)
    # every E4M3 value is exact in BF16, and quantising it with scale 1 gives its code again
    ops.call("software_e4m3_h100_linear", p(dev_bits(f32_to_bf16(values))), p(dev(w)), rows, inner, columns, 1.0,
             0.0625, p(scratch), p(out), stream())
    expected = np.empty((rows, columns), np.uint16)
    oracle.qgmma_codes(ptr(x), ptr(w), rows, inner, columns, 0.0625, ptr(expected))
    assert np.array_equal(host_bits(out), expected)


@pytest.mark.parametrize("rows,inner,columns", [(2, 288, 65), (8, 32, 15), (9, 160, 17), (16, 96, 4736), (64, 96, 18944),
                                               (256, 64, 4737), (449, 32, 2433)])
def test_emulated_projection_with_every_weight_code(ops, oracle, rows, inner, columns):
    """Weights of all codes, in tiles of 8, 16 and 64 rows (the last on tcgen05: 64 x 18944 and 256 x 4737) with remainders and groups
    that do not fill a stage.  The code of a NaN counts as 480 (the oracle has none): it meets one value of 0.5 in its group."""
    rng = np.random.default_rng(rows + inner + columns)
    x = _codes(rng, "any", (rows, inner))
    w = rng.permutation(np.resize(np.arange(256, dtype=np.uint8), columns * inner)).reshape(columns, inner)
    w[(w & 0x7f) == 0x7f] ^= 1
    x[rows // 2], x[rows // 2, inner - 7] = 0, 0x30
    w = np.ascontiguousarray(w)
    values = torch.from_numpy(x).view(torch.float8_e4m3fn).float().numpy()
    scratch = torch.empty(x.size, dtype=torch.uint8, device="cuda")
    expected = np.empty((rows, columns), np.uint16)
    oracle.qgmma_codes(ptr(x), ptr(w), rows, inner, columns, 0.0625, ptr(expected))
    for code in (None, 0x7f, 0xff):
        if code is not None:
            w[columns - 1, inner - 7] = code
            expected[rows // 2, columns - 1] = f32_to_bf16(np.float32([15.0 if code == 0x7f else -15.0]))[0]
        out = empty_bits(rows, columns)
        ops.call("software_e4m3_h100_linear", p(dev_bits(f32_to_bf16(values))), p(dev(w)), rows, inner, columns, 1.0,
                 0.0625, p(scratch), p(out), stream())
        got = host_bits(out)
        if code is not None:  # (the other rows meet 480 as well)
            got = got[rows // 2], expected[rows // 2]
            assert np.array_equal(*got)
        else:
            assert np.array_equal(got, expected)


@pytest.mark.parametrize("kind", ["any", "sparse", "subnormal", "extreme", "cancel", "gaps"])
@pytest.mark.parametrize("inner", [32, 64, 128, 160, 288, 1056])
@pytest.mark.parametrize("rows,columns", [(129, 6001), (321, 7701)])
def test_emulated_products_in_tensor_memory(ops, oracle, rows, columns, inner, kind):
    """Tiles of 64 rows x 128 columns with remainders, on an SM each and in more than one wave of two an SM, so that tensor memory
    changes hands while others compute; group counts that fill the rings of unpacked groups several times over, odd ones and one
    and two.  The rows and the weights repeat every 43 and every 203, which no tile does."""
    rng = np.random.default_rng(rows + inner)
    x, w = (_codes(rng, "any" if kind == "gaps" else kind, (lines, inner)) for lines in (43, 203))
    if kind == "gaps":  # groups without a product between large and small ones
        scale = rng.integers(0, 3, (1, inner // 32)).repeat(32, 1)
        x = np.ascontiguousarray(np.where(scale == 0, 0, np.where(scale == 1, x & 0x87, x)).astype(np.uint8))
    expected = np.empty((43, 203), np.uint16)
    oracle.qgmma_codes(ptr(x), ptr(w), 43, inner, 203, 0.0625, ptr(expected))
    x, w = x[np.arange(rows) % 43], w[np.arange(columns) % 203]
    values = torch.from_numpy(x).view(torch.float8_e4m3fn).float().numpy()
    scratch, out = torch.empty(x.size, dtype=torch.uint8, device="cuda"), empty_bits(rows, columns)
    ops.call("software_e4m3_h100_linear", p(dev_bits(f32_to_bf16(values))), p(dev(w)), rows, inner, columns, 1.0, 0.0625, p(scratch),
             p(out), stream())
    ops.call("check_async_errors", stream())
    assert np.array_equal(host_bits(out), expected[np.arange(rows) % 43][:, np.arange(columns) % 203])


@pytest.mark.parametrize("kind", ["any", "sparse", "subnormal", "extreme", "cancel"])
@pytest.mark.parametrize("inner,columns", [(32, 1), (64, 33), (96, 14209), (128, 31), (160, 65), (480, 40), (512, 64), (544, 14208),
                                           (576, 14240), (1056, 129), (2080, 14209), (24576, 5)])
def test_one_emulated_row(ops, oracle, inner, columns, kind):
    """Four and two lanes per column on either side of their limit; group counts around batches of four and the 16 groups that
    are read ahead; and a weight of code 0x7f (480) against one value of 0.5."""
    rng = np.random.default_rng(inner + columns)
    x, w = _codes(rng, kind, (1, inner)), _codes(rng, kind, (columns, inner))
    scratch = torch.empty(x.size, dtype=torch.uint8, device="cuda")

    def product():
        out = empty_bits(1, columns)
        values = torch.from_numpy(x).view(torch.float8_e4m3fn).float().numpy()
        ops.call("software_e4m3_h100_linear", p(dev_bits(f32_to_bf16(values))), p(dev(w)), 1, inner, columns, 1.0, 0.0625, p(scratch),
                 p(out), stream())
        return host_bits(out)

    expected = np.empty((1, columns), np.uint16)
    oracle.qgmma_codes(ptr(x), ptr(w), 1, inner, columns, 0.0625, ptr(expected))
    assert np.array_equal(product(), expected)
    x[0], x[0, inner // 2] = 0, 0x30
    w[columns - 1, inner // 2] = 0xff
    assert product()[0, columns - 1] == f32_to_bf16(np.float32([-15.0]))[0]
