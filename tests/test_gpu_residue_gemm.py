"""Edges of the FP64-accurate residue GEMM (csrc/ozaki.cu): tile remainders, the 1024-long
exactness chunks of K, the switch from 15 to 16 moduli, K ranges beyond one launch, results
below the normal range and every alpha / beta path.

Tolerance.  An operand entry is rounded to t >= 53 bits below a power of two that is less
than twice its row (column) maximum: |da| <= 2^-53 max_a.  The products are exact and the
result is rounded once, so |dC| <= K 2^-53 (2 max_a max_b) + 2^-53 |C|; the float64
reference is off by at most K 2^-53 |A| |B| itself.
"""

import numpy as np
import pytest

import finitemptools_gb300 as fm
from finitemptools_gb300 import DeviceTensor as DT
from finitemptools_gb300.auxiliary import gemm

pytestmark = pytest.mark.gpu

TC_GEMM = 0      # FMPT_K_TC_GEMM


def op(A, t):
    return {"N": A, "T": A.T, "C": A.conj().T, "R": A.conj()}[t]


@pytest.mark.parametrize("cplx,ta,tb,m,n,k,alpha,beta,scale", [
    (False, "N", "N", 256, 256, 1024, 1.0, 0.0, 0),
    (False, "N", "T", 257, 255, 1025, 1.0, 0.0, 0),
    (False, "T", "N", 511, 130, 1783, 1.0, 0.0, 0),
    (False, "T", "T", 513, 100, 1700, -0.5, 0.0, 0),
    (False, "N", "N", 300, 301, 2048, 1.0, 2.0, 0),
    (False, "T", "N", 33, 1030, 2049, 1.5, -1.0, 0),
    (False, "N", "N", 257, 130, 131100, 1.0, 0.0, 0),
    (False, "N", "T", 256, 256, 1024, 1.0, 0.0, -520),
    (True, "N", "N", 250, 129, 513, 1.0, 0.0, 0),
    (True, "C", "N", 129, 257, 900, 0.5, 0.0, 0),
    (True, "R", "T", 200, 300, 1024, 0.5 - 2.0j, 1.0 + 0.5j, 0),
    (True, "T", "C", 200, 150, 70001, 1.0, 1.0, 0),
])
def test_residue_gemm_edges(cplx, ta, tb, m, n, k, alpha, beta, scale):
    h = fm.default_handle()
    rng = np.random.default_rng(m * n + k)

    def mat(r, c):
        a = rng.standard_normal((r, c)) * 2.0 ** scale
        return a + 1j * rng.standard_normal((r, c)) * 2.0 ** scale if cplx else a

    A = mat(m, k) if ta in "NR" else mat(k, m)
    B = mat(k, n) if tb in "NR" else mat(n, k)
    C0 = mat(m, n) if beta else np.zeros((m, n))
    a, b = op(A, ta), op(B, tb)
    # a power-of-two scale is taken out of the reference's products and put back at the end,
    # so that its own terms do not underflow
    ref = alpha * ((a * 2.0 ** -scale) @ (b * 2.0 ** -scale)) * 2.0 ** scale * 2.0 ** scale
    ref = ref + beta * C0
    h.set_f64_engine("tensor_cores")
    h.profile(True)
    h.profile_read(TC_GEMM)
    try:
        C = DT.from_numpy(C0, h, np.complex128 if cplx else np.float64)
        gemm(DT.from_numpy(A, h), DT.from_numpy(B, h), (m, n), m, n, k, ta, tb, alpha=alpha,
             beta=beta, C=C, lda=A.shape[0], ldb=B.shape[0])
        launches, _ = h.profile_read(TC_GEMM)
    finally:
        h.profile(False)
        h.set_f64_engine("cuda_cores")
    assert launches >= 1
    kk = k * (2 if cplx else 1)
    mx = 2.0 * np.abs(a).max(axis=1)[:, None] * np.abs(b).max(axis=0)[None, :]
    tol = 2.0 ** -53 * (abs(alpha) * kk * (mx + np.abs(a) @ np.abs(b)) +
                        4 * (np.abs(ref) + abs(beta) * np.abs(C0))) + 2.0 ** -1074
    assert (np.abs(C.numpy() - ref) <= tol).all()
