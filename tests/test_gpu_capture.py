"""Applications recorded into a caller's stream capture, on operators that were used before with the
other FP64 engine: a Lanczos solve (digit products) before a captured application (residue
products), or a handle whose engine is switched in between.  Workspaces cannot grow inside the
capture, so such an application runs on what is there, on the CUDA cores if need be; it is not
refused.  Against a direct application: either engine is within 1e-14 of the exact product (K <=
1500 terms rounded at 2^-53, random signs), the bound is 1e-13."""

import numpy as np
import pytest

import finitemptools_gb300 as fm
from finitemptools_gb300 import DeviceTensor as DT
from finitemptools_gb300.utilities import heisenberg_xxz_mpo

pytestmark = pytest.mark.gpu


def _operator(dl, dr, sites, precision):
    rng = np.random.default_rng(dl + dr)
    W = heisenberg_xxz_mpo(1.0, 0.7, 0.3)[1].dense()

    def env(D):
        e = rng.standard_normal((D, W.shape[0], D))
        return DT.from_numpy((e + e.transpose(2, 1, 0)) / np.sqrt(D))

    x = DT.from_numpy(rng.standard_normal((dl,) + (2,) * sites + (dr,)))
    op = fm.HeffOp("ac2" if sites == 2 else "ac", env(dl), env(dr), W1=W,
                   W2=W if sites == 2 else None, precision=precision, dtype=np.float64)
    return op, x


def _captured(op, x):
    """two replays of one recorded application, the second on another vector"""
    torch = pytest.importorskip("torch")
    h = op.h
    buf, y = x.copy(), DT(x.shape, np.float64, h)
    stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    h.synchronize()
    h.set_stream(stream.cuda_stream)
    try:
        with torch.cuda.graph(graph, stream=stream, capture_error_mode="thread_local"):
            op(buf, out=y)
        graph.replay()
        torch.cuda.synchronize()
        first = y.numpy()
        two = DT.from_numpy(2.0 * x.numpy(), h)
        h.check(fm._native.lib().fmpt_memcpy_d2d(h.ptr, buf.ptr, two.ptr, x.nbytes))
        h.synchronize()
        graph.replay()
        torch.cuda.synchronize()
        return first, y.numpy()
    finally:
        torch.cuda.synchronize()
        h.set_stream(None)
        del graph


def _check(op, x):
    first, second = _captured(op, x)
    ref = op(x).numpy()
    assert np.linalg.norm(first - ref) <= 1e-13 * np.linalg.norm(ref)
    assert np.array_equal(second, 2.0 * first)            # a power of two: the same roundings


@pytest.mark.parametrize("dl,dr,sites", [(64, 64, 2), (96, 96, 2), (256, 256, 2), (300, 140, 2),
                                         (200, 333, 1), (97, 290, 1)])
def test_after_a_solve(dl, dr, sites):
    op, x = _operator(dl, dr, sites, "fp64_tc")
    op.lanczos(x, 2, 1e-10)
    _check(op, x)


@pytest.mark.parametrize("dl,dr,sites", [(96, 96, 2), (256, 200, 2), (97, 290, 1)])
def test_after_an_engine_switch(dl, dr, sites):
    op, x = _operator(dl, dr, sites, "fp64")
    op(x)
    op.h.set_f64_engine("tensor_cores")
    try:
        _check(op, x)
    finally:
        op.h.set_f64_engine("cuda_cores")


@pytest.mark.parametrize("dl,dr,sites", [(256, 200, 2), (330, 401, 1)])
def test_residue_application(dl, dr, sites):
    """an operator that was applied before is recorded on the residue engine; direct applications
    in between leave the recorded one's workspaces as it expects them"""
    op, x = _operator(dl, dr, sites, "fp64_tc")
    ref = op(x).numpy()
    first, second = _captured(op, x)
    assert np.array_equal(first, ref) and np.array_equal(second, 2.0 * ref)
    assert np.array_equal(op(x).numpy(), ref)
    _check(op, x)
