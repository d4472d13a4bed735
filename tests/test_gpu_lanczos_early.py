"""Lanczos solves that end before their last allowed step.  The step after the one that ends the
solve has been queued by then: it must not change the result, and where the operator is large its
GEMMs must do no work.

An operator L x with three distinct eigenvalues 1, 2, 4 exhausts the Krylov space in three steps.
Its betas are of order 1 until then and of the size of the operator's rounding u |H| = 4 u after
(u = 2^-53, 3xTF32 2^-22, TF32 2^-12, BF16 2^-9); the bounds leave a factor of about six for the
recurrence."""

import numpy as np
import pytest

import finitemptools_gb300 as fm
from finitemptools_gb300 import DeviceTensor as DT
from finitemptools_gb300.u1 import U1Space
from oracle import u1 as OU

pytestmark = pytest.mark.gpu

TC_GEMM, F64_GEMM, GROUPED = 0, 1, 4      # FMPT_K_*


@pytest.mark.parametrize("precision,tol", [("fp64", 1e-10), ("fp64_tc", 1e-10), ("tf32x3", 1e-5),
                                           ("tf32", 0.01), ("bf16", 0.05)])
@pytest.mark.parametrize("D", [15, 64, 330, 1300])
@pytest.mark.parametrize("reorth", [False, True])
def test_three_steps(D, precision, tol, reorth):
    rng = np.random.default_rng(D)
    lam = np.repeat([1.0, 2.0, 4.0], (D + 2) // 3)[:D]
    L = DT.from_numpy(np.diag(lam)[:, None, :])
    R = DT.from_numpy(np.eye(D)[:, None, :])
    op = fm.HeffOp("c", L, R, precision=precision, dtype=np.float64)
    x = DT.from_numpy(rng.standard_normal((D, D)))
    E, v, info, k = op.lanczos(x, 20, tol, reorth=reorth)
    assert (k, info) == (3, 0)
    v = v.numpy()
    assert abs(E - 1.0) <= tol
    assert abs(np.linalg.norm(v) - 1.0) <= tol
    assert np.linalg.norm(lam[:, None] * v - v) <= 4 * tol
    # the same solve with no step left to queue
    E3, v3, _, k3 = op.lanczos(x, 3, tol, reorth=reorth)
    assert k3 == 3 and E3 == E and np.array_equal(v3.numpy(), v)


def _gemm_ms(h, kernel, run):
    h.profile(True)
    try:
        h.profile_read(kernel)
        run()
        return h.profile_read(kernel)
    finally:
        h.profile(False)


@pytest.mark.parametrize("precision,D,kernel", [("fp64", 800, F64_GEMM), ("fp64_tc", 1200, TC_GEMM),
                                                ("tf32x3", 3000, TC_GEMM),
                                                ("bf16", 4000, TC_GEMM)])
def test_queued_step_does_no_gemm(precision, D, kernel):
    one = DT.from_numpy(np.eye(D)[:, None, :])
    op = fm.HeffOp("c", one, one, precision=precision, dtype=np.float64)
    x = DT.from_numpy(np.random.default_rng(0).standard_normal((D, D)))
    tol = 0.05
    for kmax in (1, 20):
        assert op.lanczos(x, kmax, tol)[3] == 1
    n1, t1 = _gemm_ms(op.h, kernel, lambda: op.lanczos(x, 1, tol))
    n20, t20 = _gemm_ms(op.h, kernel, lambda: op.lanczos(x, 20, tol))
    assert n1 > 0 and n20 > 0
    assert t20 < 1.5 * t1                     # two applications would take twice as long


def test_queued_block_sparse_step_does_nothing():
    dims = (200, 500, 450, 150)
    Vl = OU.Leg(list(enumerate(dims)))
    Vr = OU.Leg([(q + 1, d) for q, d in enumerate(dims)])
    W = np.eye(2)[None, :, None, :]
    L, R = DT.from_numpy(np.eye(Vl.dim)[:, None, :]), DT.from_numpy(np.eye(Vr.dim)[:, None, :])
    op = fm.U1HeffOp(L, R, W, W, U1Space(Vl.items()), U1Space(Vr.items()), (0, 1), (0, 1),
                     [0], [0], [0])
    x = DT.from_numpy(np.random.default_rng(0).standard_normal(op.n))
    op.h.set_graphs(False)
    try:
        for kmax in (1, 20):
            assert op.lanczos(x, kmax, 1e-8)[3] == 1
        n1, t1 = _gemm_ms(op.h, GROUPED, lambda: op.lanczos(x, 1, 1e-8))
        n20, t20 = _gemm_ms(op.h, GROUPED, lambda: op.lanczos(x, 20, 1e-8))
    finally:
        op.h.set_graphs(True)
    assert n1 > 0 and t20 < 1.5 * t1
