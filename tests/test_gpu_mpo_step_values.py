"""Values that the FP64 MPO step copies instead of multiplying (an output's first term with coefficient
+-1): infinities, NaN, denormals and both zeros keep what a multiply-add with +0 makes of them, alone
and with further terms after the copy.  A 1 x 1 bond with environments 1 makes the operator the 4 x 4
matrix M of one site: y_q = sum over M[q, s] != 0 of M[q, s] x_s in the order of s, exactly, and +0
for a zero of either sign (every chain of multiply-adds starts from +0)."""

from fractions import Fraction

import numpy as np
import pytest

import finitemptools_gb300 as fm
from finitemptools_gb300 import DeviceTensor as DT

pytestmark = pytest.mark.gpu

INF, NAN, TINY = np.inf, np.nan, 5e-324
M1 = np.diag([1.0, -1.0, 1.0, -1.0])
M2 = np.array([[1.0, 2.0, 0.0, 0.0], [-1.0, 0.0, 0.5, 0.0], [0.0, -1.0, 0.0, 1.0],
               [2.0, 1.0, 0.0, 0.0]])


def fma(a, b, c):
    if np.isfinite(a * b) or not np.isfinite([a, b, c]).all():
        return a * b + c                       # the coefficients are powers of two: exact products
    exact = Fraction(a) * Fraction(b) + Fraction(c)
    try:
        return float(exact)
    except OverflowError:
        return INF if exact > 0 else -INF


@pytest.mark.parametrize("M", [M1, M2])
@pytest.mark.parametrize("x", [
    [INF, -INF, NAN, 1.0], [-0.0, 0.0, -0.0, -0.0], [TINY, -TINY, 2.0 ** -1050, -1e-310],
    [1e308, -1e308, 3.0, INF], [0.0, -0.0, 0.0, 0.0], [1.5, -2.25, 4.0, -0.125],
    [INF, 1.0, 2.0, 3.0], [1.0, NAN, 2.0, -INF],
])
def test_copied_terms(M, x):
    one = DT.from_numpy(np.ones((1, 1, 1)))
    op = fm.HeffOp("ac", one, one, W1=M[None, :, None, :], dtype=np.float64)
    y = op(DT.from_numpy(np.array(x).reshape(1, 4, 1))).numpy().ravel()
    with np.errstate(all="ignore"):
        for q in range(4):
            ref = 0.0
            for s in np.nonzero(M[q])[0]:
                ref = fma(M[q, s], x[s], ref)
            if np.isnan(ref):
                assert np.isnan(y[q])
            else:
                assert y[q] == ref and (ref != 0.0 or not np.signbit(y[q])), (q, y[q], ref)
