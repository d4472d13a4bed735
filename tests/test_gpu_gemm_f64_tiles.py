"""Edges of the small-problem FP64 GEMM (one warp per 8 x 4 tile, slabs of 32 along K, K split
over the grid): tile and slab remainders, every transposition, alpha / beta, real and complex.

Tolerance: k multiply-adds (four per complex one) and the alpha / beta update, each rounded to
2^-53, on both sides: (2 k + 4) 2^-52 times the sum of the terms' magnitudes."""

import numpy as np
import pytest

import finitemptools_gb300 as fm
from finitemptools_gb300 import DeviceTensor as DT
from finitemptools_gb300.auxiliary import gemm

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("ta,tb,m,n,k,alpha,beta", [
    ("N", "N", 1, 1, 1, 1.0, 0.0),
    ("N", "T", 8, 4, 32, 1.0, 0.0),
    ("T", "N", 9, 5, 33, -2.0, 0.0),
    ("C", "C", 17, 3, 31, 1.0, 1.0),
    ("R", "N", 7, 130, 129, 0.5, 0.0),
    ("N", "R", 130, 7, 127, 1.0, -0.25),
    ("T", "T", 24, 20, 161, 1.0, 0.0),
    ("N", "N", 40, 36, 700, 1.5, 2.0),         # K split
    ("C", "N", 33, 30, 1000, 1.0, 0.0),        # K split
    ("N", "T", 320, 256, 64, 1.0, 0.0),
])
def test_gemm_f64_tile_edges(cplx, ta, tb, m, n, k, alpha, beta):
    h = fm.default_handle()
    rng = np.random.default_rng(m + 100 * n + k)

    def mat(r, c):
        a = rng.standard_normal((r, c))
        return a + 1j * rng.standard_normal((r, c)) if cplx else a

    if cplx and alpha != 1.0:
        alpha, beta = alpha * (1 - 0.5j), beta * (1 + 2j)
    A = mat(m, k) if ta in "NR" else mat(k, m)
    B = mat(k, n) if tb in "NR" else mat(n, k)
    C0 = mat(m, n)
    op = {"N": lambda x: x, "T": lambda x: x.T, "C": lambda x: x.conj().T, "R": np.conj}
    a, b = op[ta](A), op[tb](B)
    C = DT.from_numpy(C0, h)
    gemm(DT.from_numpy(A, h), DT.from_numpy(B, h), (m, n), m, n, k, ta, tb, alpha=alpha,
         beta=beta, C=C, lda=A.shape[0], ldb=B.shape[0])
    ref = alpha * (a @ b) + beta * C0
    size = abs(alpha) * (np.abs(a) @ np.abs(b)) + abs(beta) * np.abs(C0)
    kk = k * (4 if cplx else 1)
    assert (np.abs(C.numpy() - ref) <= (2 * kk + 4) * 2.0 ** -52 * size).all()
