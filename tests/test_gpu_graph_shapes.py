"""Exponentials whose launches differ in their cluster sizes take turns on one handle:
orthogonalisation clusters of 1, 4, 8 and 16 blocks and tensor-core GEMMs with 1 to 4 K pieces per
cluster.  Whatever ran before, and with graphs allowed or not, every result is the first one, bit
for bit (the same launches).  An executable graph that is updated from one operator to the next
keeps the old cluster sizes, without an error."""

import numpy as np
import pytest

import finitemptools_gb300 as fm
from finitemptools_gb300 import DeviceTensor as DT
from finitemptools_gb300.utilities import tfi_mpo

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,cplx,dims", [
    ("fp64", True, [(4, 4), (8, 10), (16, 16), (2, 8), (20, 22), (8, 16)]),
    ("tf32x3", True, [(4, 8), (16, 16), (40, 24), (12, 12), (96, 100)]),
    ("tf32x3", False, [(16, 16), (256, 128), (100, 200), (64, 300)]),
])
def test_graphs_of_many_shapes(precision, cplx, dims):
    rng = np.random.default_rng(7)
    W = tfi_mpo([0.7])[1].dense()
    h = fm.default_handle()

    def herm(D):
        e = rng.standard_normal((D, W.shape[0], D))
        e = e + 1j * rng.standard_normal(e.shape) if cplx else e
        return (e + e.transpose(2, 1, 0).conj()) / (4 * D)

    jobs = []
    for dl, dr in dims:
        x = rng.standard_normal((dl, 2, dr))
        x = x + 1j * rng.standard_normal(x.shape) if cplx else x
        dx = DT.from_numpy(x / np.linalg.norm(x))
        jobs.append((fm.HeffOp("ac", DT.from_numpy(herm(dl)), DT.from_numpy(herm(dr)), W1=W,
                               precision=precision, dtype=dx.dtype), dx))
    t = -0.05j if cplx else -0.05

    def run():
        return [op.exponentiate(t, x, 1e-8, 8).numpy() for op, x in jobs]

    h.set_graphs(False)
    try:
        ref = run()
    finally:
        h.set_graphs(True)
    for _ in range(3):
        for y, r in zip(run(), ref):
            assert np.array_equal(y, r)
