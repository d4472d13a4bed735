"""The integer conversions between FP64 and FP32 at the ends of the mixed-precision forms, on a
1 x 1 bond whose environments are 1, so that y is x through FP64 -> FP32 -> operand format -> FP32
-> FP64 and a product with 1.  Rounding is to nearest even into FP32, then into the operand format
(BF16: to nearest even; TF32: to nearest, ties away from zero, the conversion instruction's rule).
Normal values, rounding carries and ties, both zeros, infinities and NaN come out exactly; below
FP32's normal range the operand formats may lose the value, so there the error is bounded by 2^-126
alone.  3xTF32 adds TF32 of the rest, 2^-24 of the value off in each of the two GEMMs, whose FP32
sums of three products add at most 2^-23 each: below 2^-20 in all."""

import numpy as np
import pytest

import finitemptools_gb300 as fm
from finitemptools_gb300 import DeviceTensor as DT

pytestmark = pytest.mark.gpu


def _values():
    rng = np.random.default_rng(0)
    v = [0.0, 1.0, 1.0 / 3.0, np.nextafter(2.0, 0.0), np.nextafter(1.0, 2.0),
         2.0 - 2.0 ** -24, 2.0 - 2.0 ** -25,                       # carry into the exponent, below it
         1.0 + 2.0 ** -24, 1.0 + 3 * 2.0 ** -24, 1.0 + 2.0 ** -24 + 2.0 ** -52,   # FP32 ties
         1.0 + 2.0 ** -8, 1.0 + 3 * 2.0 ** -8, 1.0 + 2.0 ** -11, 1.0 + 3 * 2.0 ** -11,
         2.0 ** -126, 2.0 ** -126 * (2 - 2.0 ** -23), 2.0 ** 127, 2.0 ** 100 / 3]
    v += list(rng.standard_normal(12) * 2.0 ** rng.integers(-120, 120, 12))
    return v + [-a for a in v]


def _tf32(f):
    """FP32 -> TF32, to nearest, ties away from zero"""
    b = np.float32(f).view(np.uint32)
    return np.uint32((int(b) + 0x1000) & 0xFFFFE000).view(np.float32)


def _bf16(f):
    b = int(np.float32(f).view(np.uint32))
    return np.uint32(((b + 0x7FFF + ((b >> 16) & 1)) & 0xFFFF0000) & 0xFFFFFFFF).view(np.float32)


def _expected(v, precision):
    f = np.float32(v)
    if precision == "bf16":
        return float(_bf16(f))
    return float(_tf32(f))


def _through(values, precision):
    one = DT.from_numpy(np.ones((1, 1, 1)))
    op = fm.HeffOp("c", one, one, precision=precision, dtype=np.float64)
    return [float(op(DT.from_numpy(np.array([[v]]))).numpy()[0, 0]) for v in values]


@pytest.mark.parametrize("precision", ["bf16", "tf32", "tf32x3"])
def test_normal_values(precision):
    values = _values()
    for v, y in zip(values, _through(values, precision)):
        if precision == "tf32x3":
            assert abs(y - v) <= 2.0 ** -20 * abs(v) + 2.0 ** -126, v
        else:
            assert y == _expected(v, precision), v


@pytest.mark.parametrize("precision", ["bf16", "tf32"])
def test_special_values(precision):
    inf = np.inf
    big = [inf, 2.0 ** 128, 1e300, 2.0 ** 128 - 2.0 ** 103]   # FP32's overflow threshold
    for s in (1.0, -1.0):
        assert _through([s * b for b in big], precision) == [s * inf] * len(big)
    assert np.isnan(_through([np.nan], precision)[0])
    tiny = [2.0 ** -127, 2.0 ** -149, 3 * 2.0 ** -150, 2.0 ** -150, 1e-300, 5e-324]
    for v, y in zip(tiny, _through(tiny, precision)):
        assert abs(y - v) <= 2.0 ** -126


@pytest.mark.parametrize("precision", ["bf16", "tf32", "tf32x3"])
def test_many_lanes(precision):
    """the same values side by side in one tensor: a rare value next to ordinary ones"""
    D = 40
    rng = np.random.default_rng(1)
    x = rng.standard_normal((D, D)) * 2.0 ** rng.integers(-60, 60, (D, D))
    x[3, 5], x[17, 31], x[39, 0] = 2.0 ** -140, -(2.0 ** -130), 0.0
    one = DT.from_numpy(np.eye(D)[:, None, :])
    op = fm.HeffOp("c", one, one, precision=precision, dtype=np.float64)
    y = op(DT.from_numpy(x)).numpy()
    u = {"bf16": 2.0 ** -8, "tf32": 2.0 ** -10, "tf32x3": 2.0 ** -20}[precision]
    assert (np.abs(y - x) <= u * np.abs(x) + 2.0 ** -126).all()
