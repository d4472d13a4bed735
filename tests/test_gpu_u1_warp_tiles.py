"""The 8x4 warp tiles of the grouped block-sparse kernel, which small programs run by default:
blocks of 1 to 33 rows and columns (edges of tiles and of the 16-deep slabs), more segments per
block than a warp holds at a time (32), several launches of one program, and environment
updates in both directions.  Every output is the same chain of FMAs over segments and k as with
the block tiles, so the results are equal bit for bit; against the oracle the bound is the
block-sparse path's 1e-12 (the sums have at most about 3000 terms: expected 1e-14)."""

import numpy as np
import pytest

import finitemptools_gb300 as fm
import oracle as O
from finitemptools_gb300 import DeviceTensor as DT
from finitemptools_gb300.u1 import U1Space
from oracle import u1 as OU

pytestmark = pytest.mark.gpu
QP = (0, 1)


def _diagonal_mpo(rng, wl, wr):
    """Charge-conserving MPO site tensor whose channels all have charge 0."""
    W = np.zeros((wl, 2, wr, 2))
    for s in range(2):
        W[:, s, :, s] = rng.standard_normal((wl, wr))
    return W


@pytest.mark.parametrize("dims,wl,wm,wr", [((1, 1), 1, 1, 1), ((3, 7, 4), 2, 3, 5),
                                           ((1, 9, 17, 8, 5), 36, 2, 40),
                                           ((16, 33, 2, 15), 33, 1, 32)])
def test_warp_tiles(dims, wl, wm, wr):
    rng = np.random.default_rng(sum(dims) + wr)
    Vl = OU.Leg(list(enumerate(dims)))
    Vr = OU.Leg([(q + 1, d) for q, d in enumerate(reversed(dims))])
    W1, W2 = _diagonal_mpo(rng, wl, wm), _diagonal_mpo(rng, wm, wr)
    qs = [0] * wl, [0] * wm, [0] * wr
    Lm = rng.standard_normal((Vl.dim, wl, Vl.dim)) * OU.allowed_env(Vl, qs[0])
    Rm = rng.standard_normal((Vr.dim, wr, Vr.dim)) * OU.allowed_env(Vr, qs[2])
    ql, qr = Vl.basis_charges(), Vr.basis_charges()
    charge = ql[:, None, None] + np.arange(2)[None, :, None] + np.arange(2)[None, None, :]
    X = rng.standard_normal((Vl.dim, 2, 2, Vr.dim)) * (charge[..., None] == qr)
    # one-site tensors from the left leg and into the right one, for the environments
    one = ql[:, None, None] + np.arange(2)[None, :, None]
    A = rng.standard_normal((Vl.dim, 2, Vr.dim)) * (one == qr)
    dL, dR = DT.from_numpy(Lm), DT.from_numpy(Rm)
    dA = DT.from_numpy(A)
    sl, sr = U1Space(Vl.items()), U1Space(Vr.items())
    x = DT.from_numpy(OU.pack2(X, Vl, Vr, list(QP), list(QP)))
    We = _diagonal_mpo(rng, wl, wr)
    h, out = dL.h, {}
    try:
        for mode in (0, 1):
            h.set_tuning(mode)
            op = fm.U1HeffOp(dL, dR, W1, W2, sl, sr, QP, QP, *qs)
            assert op.flops() < 2e7 and op.tile() == (32 if mode else 8)
            ys = [op(x).numpy() for _ in range(3)]
            assert all(np.array_equal(ys[0], y) for y in ys)
            out[mode] = [ys[0],
                         fm.u1_updateleft(dL, dA, We, dA, sl, sr, QP, qs[0], qs[2]).numpy(),
                         fm.u1_updateright(dR, dA, We, dA, sl, sr, QP, qs[0], qs[2]).numpy()]
    finally:
        h.set_tuning(0)
    for a, b in zip(out[0], out[1]):
        assert np.array_equal(a, b)
    ref = OU.pack2(O.ac2_prime(X, W1, W2, Lm, Rm), Vl, Vr, list(QP), list(QP))
    assert np.linalg.norm(out[0][0] - ref) <= 1e-12 * np.linalg.norm(ref)
