"""The MPO step of the FP64 H_eff*x at the edges of its launch rule: one thread per output
below eight blocks per SM (n1 * n2 < 155648 on 152 SMs), all outputs in one thread above, and
the small (32 outputs, 96 terms) and large coefficient tables.  Against the oracle, at the
1e-12 relative bar of the FP64 path."""

import numpy as np
import pytest

import oracle as O
import finitemptools_gb300 as fm
from finitemptools_gb300 import DeviceTensor as DT

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("dl,dr,w,dense", [
    (1, 3, 3, False), (129, 1, 5, False), (7, 11, 4, True),
    (394, 395, 2, False), (395, 395, 2, False), (395, 396, 3, True),
])
def test_mpo_step_launch_rule(dl, dr, w, dense, cplx):
    rng = np.random.default_rng(dl * dr + w)

    def r(*s):
        a = rng.standard_normal(s)
        return a + 1j * rng.standard_normal(s) if cplx else a

    W = r(w, 2, w, 2)
    if not dense:        # identities on the first and last channel, one column between
        mask = np.zeros((w, 1, w, 1))
        mask[0, :, :, :] = mask[:, :, w - 1, :] = 1.0
        W = W * mask
    x, L, R = r(dl, 2, 2, dr), r(dl, w, dl), r(dr, w, dr)
    y = fm.ac2_prime(DT.from_numpy(x), W, W, DT.from_numpy(L), DT.from_numpy(R)).numpy()
    ref = O.ac2_prime(x, W, W, L, R)
    assert np.linalg.norm(y - ref) <= 1e-12 * np.linalg.norm(ref)
