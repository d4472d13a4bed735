"""fmpt_lanczos_ground returns host scalars and therefore synchronises: when it returns, its stream
is idle and the vector can be read on any other stream, here a second handle's.  Dense operators in
every precision that solves differently, block-sparse ones with and without the graph, a solve
that converges after one step (an identity operator), and one that fails (an infinite environment)."""

import numpy as np
import pytest

import finitemptools_gb300 as fm
from finitemptools_gb300 import DeviceTensor as DT
from finitemptools_gb300._native import FMPTError, lib
from finitemptools_gb300.u1 import U1Space
from oracle import u1 as OU

pytestmark = pytest.mark.gpu
QP = (0, 1)


def idle(h):
    torch = pytest.importorskip("torch")
    return torch.cuda.ExternalStream(lib().fmpt_get_stream(h.ptr)).query()


def elsewhere(x):
    """x read on the stream of a handle of its own"""
    other = fm.Handle()
    try:
        y = DT(x.shape, x.dtype, other)
        other.check(lib().fmpt_memcpy_d2d(other.ptr, y.ptr, x.ptr, x.nbytes))
        out = y.numpy()
        del y
        return out
    finally:
        other.close()


def check(op, x, kmax):
    _, v, _, k = op.lanczos(x, kmax, 1e-10)
    assert idle(op.h)
    assert np.array_equal(elsewhere(v), v.numpy())
    return k, v.numpy()


@pytest.mark.parametrize("precision", ["fp64", "fp64_tc", "tf32x3", "bf16"])
@pytest.mark.parametrize("D,kmax", [(24, 12), (512, 3), (1200, 20)])
def test_dense(precision, D, kmax):
    rng = np.random.default_rng(D)

    def env():
        e = rng.standard_normal((D, 1, D))
        return DT.from_numpy((e + e.transpose(2, 1, 0)) / np.sqrt(D))

    op = fm.HeffOp("c", env(), env(), precision=precision, dtype=np.float64)
    k, v = check(op, DT.from_numpy(rng.standard_normal((D, D))), kmax)
    assert k == kmax and np.isfinite(v).all() and v.any()


@pytest.mark.parametrize("precision", ["fp64", "fp64_tc"])
def test_converged_start(precision):
    D = 1024
    one = DT.from_numpy(np.eye(D)[:, None, :])
    op = fm.HeffOp("c", one, one, precision=precision, dtype=np.float64)
    x = np.random.default_rng(1).standard_normal((D, D))
    k, v = check(op, DT.from_numpy(x), 20)
    assert k == 1 and np.allclose(v, x / np.linalg.norm(x), rtol=0, atol=1e-15)


@pytest.mark.parametrize("graphs", [False, True])
def test_block_sparse(graphs):
    rng = np.random.default_rng(3)
    dims = (60, 170, 110, 40)
    Vl = OU.Leg(list(enumerate(dims)))
    Vr = OU.Leg([(q + 1, d) for q, d in enumerate(reversed(dims))])
    W = np.zeros((3, 2, 3, 2))
    for s in range(2):
        W[:, s, :, s] = rng.standard_normal((3, 3))
    q = [0] * 3
    L = rng.standard_normal((Vl.dim, 3, Vl.dim)) * OU.allowed_env(Vl, q)
    R = rng.standard_normal((Vr.dim, 3, Vr.dim)) * OU.allowed_env(Vr, q)
    dl, dr = DT.from_numpy(L), DT.from_numpy(R)
    op = fm.U1HeffOp(dl, dr, W, W, U1Space(Vl.items()), U1Space(Vr.items()), QP, QP, q, q, q)
    x = DT.from_numpy(rng.standard_normal(op.n))
    op.h.set_graphs(graphs)
    try:
        k, _ = check(op, x, 12)
    finally:
        op.h.set_graphs(True)
    assert k == 12


def test_failed_solve():
    D = 700
    e = np.eye(D)[:, None, :]
    bad = e.copy()
    bad[3, 0, 3] = np.inf
    op = fm.HeffOp("c", DT.from_numpy(bad), DT.from_numpy(e), dtype=np.float64)
    with pytest.raises(FMPTError):
        op.lanczos(DT.from_numpy(np.ones((D, D))), 5, 1e-10)
    assert idle(op.h)
