"""The Krylov exponential at the edges of its orthogonalisation step's launch shapes: one block
(up to 4 chunks of 32 elements of a component), 1, 2, 4 or 8 chunks per block up to 128
blocks, and looping warps beyond 1024 chunks.  Against a Taylor series of the oracle's
one-site operator in double precision, with |t H| below 1 and 30 Krylov vectors, where both
are exact to rounding: 1e-12 relative, about 40 operator applications of rounding 1e-15 on
either side and 30 vectors orthogonal to 1e-15."""

import numpy as np
import pytest

import oracle as O
import finitemptools_gb300 as fm
from finitemptools_gb300 import DeviceTensor as DT
from finitemptools_gb300.utilities import tfi_mpo

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dl,dr,cplx", [
    (1, 2, True), (2, 4, True), (8, 4, True), (8, 4, False), (9, 4, True), (16, 16, True),
    (32, 65, True), (65, 64, False), (64, 64, True), (91, 94, True), (130, 130, False),
    # one cluster of 4 (5 chunks), 8 (10, 16) and 16 blocks (18, 64), the first beyond it (66)
    (9, 8, False), (8, 10, True), (8, 16, True), (12, 12, True), (32, 16, True), (32, 32, False),
    (33, 16, True),
])
def test_exponential_launch_shapes(dl, dr, cplx):
    rng = np.random.default_rng(dl * dr + cplx)
    W = tfi_mpo([0.7])[1].dense()

    def herm(D):
        h = rng.standard_normal((D, 3, D))
        if cplx:
            h = h + 1j * rng.standard_normal((D, 3, D))
        return (h + h.conj().transpose(2, 1, 0)) / (4 * np.sqrt(D))

    L, R = herm(dl), herm(dr)
    x = rng.standard_normal((dl, 2, dr))
    if cplx:
        x = x + 1j * rng.standard_normal(x.shape)
    t = -0.05j if cplx else -0.05
    op = fm.HeffOp("ac", DT.from_numpy(L), DT.from_numpy(R), W1=W,
                   dtype=np.complex128 if cplx else np.float64)
    y = op.exponentiate(t, DT.from_numpy(x), 1e-12, 30).numpy()
    ref, term = x, x
    for k in range(1, 30):
        term = (t / k) * O.ac_prime(term, W, L, R)
        ref = ref + term
    assert np.linalg.norm(y - ref) <= 1e-12 * np.linalg.norm(ref)
