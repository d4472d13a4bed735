"""Small tensor-core GEMMs (one CTA per 128 x 64 / 128 / 256 tile and K piece, pieces added over
a cluster) against FP64, at tile edges and at K lengths with 1 to 4 pieces; bounds of the
mixed-precision forms: 2e-6 (or 1e-8 per unit of K) for 3xTF32, 3e-3 for TF32, 2e-2 for BF16
(relative Frobenius norm), the complex forms with K doubled."""

import numpy as np
import pytest

import finitemptools_gb300 as fm
from finitemptools_gb300 import DeviceTensor as DT
from finitemptools_gb300.utilities import heisenberg_xxz_mpo

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["tf32x3", "tf32", "bf16"])
@pytest.mark.parametrize("dl,dr,cplx", [
    (33, 40, False), (64, 31, True), (65, 129, False), (128, 64, False), (129, 127, True),
    (257, 255, False), (300, 385, False),
])
def test_small_tc_gemm_edges(prec, dl, dr, cplx):
    rng = np.random.default_rng(dl + dr)

    def r(*s):
        a = rng.standard_normal(s)
        return DT.from_numpy(a + 1j * rng.standard_normal(s) if cplx else a)

    W = heisenberg_xxz_mpo(1.0, 0.8, 0.1)[1].dense()
    x, L, R = r(dl, 2, 2, dr), r(dl, 5, dl), r(dr, 5, dr)
    y = fm.ac2_prime(x, W, W, L, R, precision=prec).numpy()
    ref = fm.ac2_prime(x, W, W, L, R).numpy()
    K = 5 * max(dl, dr) * (2 if cplx else 1)
    bound = {"tf32x3": max(2e-6, 1e-8 * K), "tf32": 3e-3, "bf16": 2e-2}[prec]
    assert np.linalg.norm(y - ref) < bound * np.linalg.norm(ref)
