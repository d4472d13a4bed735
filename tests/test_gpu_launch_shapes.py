"""Exponentials whose launches differ in their cluster sizes (orthogonalisation clusters of 1, 4, 8 and
16 blocks or a cooperative grid, tensor-core GEMMs with 1 to 4 K pieces per cluster) take turns on
one handle.  Each result is, bit for bit, that of the same operator alone on a handle of its own and
that of the orthogonalisation's separate launches."""

import numpy as np
import pytest

import finitemptools_gb300 as fm
from finitemptools_gb300 import DeviceTensor as DT
from finitemptools_gb300.utilities import tfi_mpo

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,cplx,dims", [
    ("fp64", True, [(4, 4), (8, 10), (16, 16), (2, 8), (20, 22), (64, 48), (8, 16)]),
    ("tf32x3", True, [(4, 8), (16, 16), (40, 24), (12, 12), (96, 100)]),
    ("tf32x3", False, [(16, 16), (256, 128), (100, 200), (64, 300)]),
])
def test_shapes_take_turns(precision, cplx, dims):
    W = tfi_mpo([0.7])[1].dense()
    t = -0.05j if cplx else -0.05

    def job(dl, dr, h):
        rng = np.random.default_rng(31 * dl + dr)

        def r(*s):
            a = rng.standard_normal(s)
            return a + 1j * rng.standard_normal(s) if cplx else a

        L, R = ((e + e.transpose(2, 1, 0).conj()) / (4 * D)
                for D, e in ((D, r(D, W.shape[0], D)) for D in (dl, dr)))
        x = r(dl, 2, dr)
        dx = DT.from_numpy(x / np.linalg.norm(x), h)
        op = fm.HeffOp("ac", DT.from_numpy(L, h), DT.from_numpy(R, h), W1=W, precision=precision,
                       dtype=dx.dtype)
        return lambda: op.exponentiate(t, dx, 1e-8, 8).numpy()

    alone = []
    for d in dims:
        h = fm.Handle()
        alone.append(job(*d, h)())
    h = fm.Handle()
    jobs = [job(*d, h) for d in dims]
    for fused in (True, False, True):
        h.set_fused_krylov(fused)
        for run, ref in zip(jobs, alone):
            assert np.array_equal(run(), ref)
