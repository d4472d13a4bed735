"""Row maxima formed by the MPO step of the FP64-accurate tensor-core H_eff*x (they set the scale
of each row of its second GEMM): both forms of the step's launch (below and above 16 blocks per
SM), one and two sites, complex, nine physical values (more than a thread's four), odd sizes, rows
scaled by 10^+-8 and a zero row, and operators that take turns on one handle.  A row's error
follows the row's own scale: entries carry at least 53 bits below their row's maximum, so a sum
of K <= 2100 random products is off by about 2^-53 sqrt(K) / sqrt(K) of the row's norm in either
GEMM; the bound is 1e-13."""

import numpy as np
import pytest

import finitemptools_gb300 as fm
import oracle as O
from finitemptools_gb300 import DeviceTensor as DT

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dl,dr,d,w,sites,cplx", [
    (64, 96, 2, 5, 2, False), (129, 75, 2, 5, 2, False), (96, 64, 3, 4, 2, False),
    (200, 130, 2, 3, 1, True), (100, 66, 2, 3, 2, True), (560, 600, 2, 3, 2, False),
])
def test_row_maxima(dl, dr, d, w, sites, cplx):
    rng = np.random.default_rng(dl + 7 * dr + w)

    def r(*s):
        a = rng.standard_normal(s)
        return a + 1j * rng.standard_normal(s) if cplx else a

    W = r(w, d, w, d) * (rng.random((w, d, w, d)) < 0.25)
    W[0, :, 0, :] = np.eye(d)
    scale = 10.0 ** rng.integers(-8, 9, dl)
    scale[dl // 2] = 0.0
    R = r(dr, w, dr)
    ops, xs, refs = [], [], []
    for k in range(2):                     # two operators on one handle
        L = r(dl, w, dl) * scale[:, None, None]
        x = r(dl, d, d, dr) if sites == 2 else r(dl, d, dr)
        dt = DT.from_numpy(x)
        ops.append(fm.HeffOp("ac2" if sites == 2 else "ac", DT.from_numpy(L), DT.from_numpy(R),
                             W1=W, W2=W if sites == 2 else None, precision="fp64_tc",
                             dtype=dt.dtype))
        xs.append(dt)
        refs.append(O.ac2_prime(x, W, W, L, R) if sites == 2 else O.ac_prime(x, W, L, R))
    first = [op(x).numpy() for op, x in zip(ops, xs)]
    for k in (1, 0, 0):                    # the maxima start from zero each time
        assert np.array_equal(ops[k](xs[k]).numpy(), first[k])
    for y, ref in zip(first, refs):
        err = np.linalg.norm((y - ref).reshape(dl, -1), axis=1)
        assert np.all(err <= 1e-13 * np.linalg.norm(ref.reshape(dl, -1), axis=1))
