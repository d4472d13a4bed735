"""The digit-product FP64 GEMM (csrc/ozaki_digits.cu), which FP64_TC operators run inside the Lanczos
solve: real and complex, odd dimensions, every way its plan cuts a tile into pieces (1, 3 or 5 level
sets, 1 to 4 K ranges), K below and beyond an exactness chunk (1792 for the longest level), one and
two sites and bond matrices.  Against the same solve in FP64.

Entries carry 54 bits below their row's maximum, so an application is off by 2^-54 sqrt(K) of its
norm per term of random sign, below 1e-14 for these K; four steps with betas of order |H| / 2
multiply that by less than 100.  The vectors' signs are the solver's."""

import numpy as np
import pytest

import finitemptools_gb300 as fm
from finitemptools_gb300 import DeviceTensor as DT
from finitemptools_gb300._native import FMPTError
from finitemptools_gb300.utilities import heisenberg_xxz_mpo, tfi_mpo

pytestmark = pytest.mark.gpu

TC_GEMM = 0      # FMPT_K_TC_GEMM


def _env(rng, D, w, cplx):
    e = rng.standard_normal((D, w, D))
    if cplx:
        e = e + 1j * rng.standard_normal(e.shape)
    return (e + e.transpose(2, 1, 0).conj()) / np.sqrt(D)


@pytest.mark.parametrize("kind,dl,dr,model,cplx", [
    ("ac2", 129, 75, "xxz", False), ("ac2", 256, 256, "xxz", False), ("ac2", 301, 411, "xxz", False),
    ("ac2", 100, 140, "tfi", True), ("ac2", 333, 150, "xxz", True), ("ac", 1200, 1201, "tfi", False),
    ("ac", 640, 601, "xxz", True), ("c", 512, 700, "tfi", False), ("c", 2100, 300, None, False),
    ("c", 1300, 2049, None, False), ("c", 255, 257, "xxz", True),
])
def test_solve_matches_fp64(kind, dl, dr, model, cplx):
    rng = np.random.default_rng(dl + 3 * dr)
    dt = np.complex128 if cplx else np.float64
    W = {"xxz": heisenberg_xxz_mpo(1.0, 0.7, 0.3), "tfi": tfi_mpo([0.7])}[model][1].dense() \
        if model else np.ones((1, 1, 1, 1))
    L = DT.from_numpy(_env(rng, dl, W.shape[0], cplx), dtype=dt)
    R = DT.from_numpy(_env(rng, dr, W.shape[0], cplx), dtype=dt)
    x = rng.standard_normal((dl,) + (2,) * {"ac2": 2, "ac": 1, "c": 0}[kind] + (dr,))
    if cplx:
        x = x + 1j * rng.standard_normal(x.shape)
    x = DT.from_numpy(x, dtype=dt)
    args = {"ac2": {"W1": W, "W2": W}, "ac": {"W1": W}, "c": {}}[kind]
    out = {}
    for precision in ("fp64", "fp64_tc"):
        op = fm.HeffOp(kind, L, R, precision=precision, dtype=dt, **args)
        h = op.h
        h.profile(True)
        h.profile_read(TC_GEMM)
        try:
            E, v, _, k = op.lanczos(x, 4, 1e-10)
            launches = h.profile_read(TC_GEMM)[0]
        finally:
            h.profile(False)
        assert k == 4 and (launches >= 4) == (precision == "fp64_tc")
        out[precision] = E, v.numpy()
        assert np.array_equal(op.lanczos(x, 4, 1e-10)[1].numpy(), out[precision][1])
    (E0, v0), (E1, v1) = out["fp64"], out["fp64_tc"]
    assert abs(E1 - E0) <= 1e-12 * max(1.0, abs(E0))
    # (random channels make the XXZ operator unsymmetric, and the vector is then not of norm 1)
    sign = np.sign(np.vdot(v0, v1).real)
    assert np.linalg.norm(v1 - sign * v0) <= 1e-11 * np.linalg.norm(v0)


def test_infinite_entry():
    """rows that hold Inf come out as NaN, which the solve reports"""
    D = 400
    e = _env(np.random.default_rng(0), D, 1, False)
    e[7, 0, 9] = np.inf
    L, R = DT.from_numpy(e), DT.from_numpy(np.eye(D)[:, None, :])
    op = fm.HeffOp("c", L, R, precision="fp64_tc", dtype=np.float64)
    with pytest.raises(FMPTError) as err:
        op.lanczos(DT.from_numpy(np.ones((D, D))), 3, 1e-10)
    assert err.value.status == -6
