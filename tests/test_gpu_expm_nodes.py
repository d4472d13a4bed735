"""Krylov exponentials at many nodes at once (fmpt_expm_nodes): more nodes than a grid axis holds.
With 8 vectors of an 8-dimensional space the projection is exact: each node is exp(s t H) x of the
dense matrix, to 1e-12 (|t H| below 1, 8 vectors orthogonal to 1e-15)."""

import ctypes

import numpy as np
import pytest
import scipy.linalg

import finitemptools_gb300 as fm
from finitemptools_gb300 import DeviceTensor as DT
from finitemptools_gb300._native import lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nnodes", [1, 65535, 65536, 131500])
def test_many_nodes(nnodes):
    rng = np.random.default_rng(5)
    a, b = (m + m.T for m in (rng.standard_normal((4, 4)), rng.standard_normal((2, 2))))
    L, R = DT.from_numpy(0.2 * a[:, None, :]), DT.from_numpy(0.2 * b[:, None, :])
    op = fm.HeffOp("c", L, R, dtype=np.float64)
    x = rng.standard_normal((4, 2))
    dx = DT.from_numpy(x)
    nodes = np.linspace(0.0, 1.0, nnodes) if nnodes > 1 else np.array([0.7])
    out = DT((nnodes,) + x.shape, np.float64, op.h)
    err = ctypes.c_double()
    op.h.check(lib().fmpt_expm_nodes(op.ptr, -0.5, 0.0, dx.ptr, 8, nnodes,
                                     nodes.ctypes.data_as(ctypes.POINTER(ctypes.c_double)),
                                     out.ptr, ctypes.byref(err)))
    y = out.numpy().reshape(-1, order="F").reshape(nnodes, 8)        # one vector after another
    H = 0.04 * np.kron(b, a)                              # column-major (a', b')
    for q in {0, nnodes // 2, min(65534, nnodes - 1), min(65535, nnodes - 1), nnodes - 1}:
        ref = scipy.linalg.expm(-0.5 * nodes[q] * H) @ x.reshape(-1, order="F")
        assert np.linalg.norm(y[q] - ref) <= 1e-12 * np.linalg.norm(ref)
