"""Mixed-precision Lanczos steps, whose vectors are written to the operator's operand planes as they
are scaled (bond dimension a multiple of eight) or converted by the operator (others).  Against a
Lanczos recurrence on the host that applies the same operator from outside: both round the same
vectors, up to FP64 rounding, so a lowest Ritz value of four steps differs by no more than the
form's own error (3.5e-3 BF16, 4e-4 TF32, 2e-6 3xTF32, of the largest coefficient), while a plane
that holds another vector than V_j changes it by order one."""

import numpy as np
import pytest

import finitemptools_gb300 as fm
from finitemptools_gb300 import DeviceTensor as DT
from finitemptools_gb300.utilities import heisenberg_xxz_mpo

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,tol", [("tf32x3", 2e-6), ("tf32", 4e-4), ("bf16", 3.5e-3)])
@pytest.mark.parametrize("dl,dr,sites", [(8, 8, 2), (16, 24, 2), (17, 24, 2), (24, 10, 1),
                                         (15, 16, 1), (264, 40, 2)])
def test_lanczos_from_planes(dl, dr, sites, precision, tol):
    rng = np.random.default_rng(dl + dr)
    W = heisenberg_xxz_mpo(1.0, 0.7, 0.3)[1].dense()

    def herm(D):
        e = rng.standard_normal((D, W.shape[0], D))
        return DT.from_numpy((e + e.transpose(2, 1, 0)) / np.sqrt(D))

    x = rng.standard_normal((dl, 2, 2, dr) if sites == 2 else (dl, 2, dr))
    dx = DT.from_numpy(x)
    op = fm.HeffOp("ac2" if sites == 2 else "ac", herm(dl), herm(dr), W1=W,
                   W2=W if sites == 2 else None, precision=precision, dtype=dx.dtype)
    k = 4
    E, _, _, n = op.lanczos(dx, k, 1e-12)
    assert n == k
    v, vp, b = x / np.linalg.norm(x), 0.0, 0.0
    T = np.zeros((k, k))
    for j in range(k):
        y = op(DT.from_numpy(v)).numpy()
        T[j, j] = np.vdot(v, y)
        y = y - T[j, j] * v - b * vp
        b = np.linalg.norm(y)
        if j + 1 < k:
            T[j, j + 1] = T[j + 1, j] = b
        vp, v = v, y / b
    assert abs(E - np.linalg.eigvalsh(T)[0]) <= tol * np.abs(T).max()
