"""Several host threads, each with a handle of its own, use the tensor-core kernels for the first
time in a process at once: kernel attributes and resident clusters are looked up once per device
under a lock.  Every thread gets the result of the same operator on one thread, bit for bit."""

import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

PROGRAM = """
import threading
import numpy as np
import finitemptools_gb300 as fm
from finitemptools_gb300 import DeviceTensor as DT

FORMS = [("tf32x3", 96), ("bf16", 300), ("fp64_tc", 200), ("tf32", 1100), ("fp64_tc", 129)]


def run(k, out):
    h = fm.Handle()
    res = []
    for precision, D in FORMS[k % 5:] + FORMS[:k % 5]:
        rng = np.random.default_rng(D)
        L, R, x = (DT.from_numpy(rng.standard_normal(s), h) for s in ((D, 2, D), (D, 2, D), (D, D)))
        op = fm.HeffOp("c", L, R, precision=precision, dtype=np.float64)
        y = op(x).numpy()
        E, v, _, _ = op.lanczos(x, 3, 1e-12)
        res.append((precision, D, y, E, v.numpy()))
        del op, L, R, x, v
    out[k] = sorted(res, key=lambda r: r[:2])


out = {}
threads = [threading.Thread(target=run, args=(k, out)) for k in range(5)]
for t in threads:
    t.start()
for t in threads:
    t.join()
run(5, out)
for k in range(5):
    for a, b in zip(out[k], out[5]):
        assert a[:2] == b[:2] and a[3] == b[3], (k, a[:2])
        assert np.array_equal(a[2], b[2]) and np.array_equal(a[4], b[4]), (k, a[:2])
print("ok")
"""


def test_first_use_from_many_threads():
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    run = subprocess.run([sys.executable, "-c", PROGRAM], cwd=root, capture_output=True, text=True,
                         timeout=300)
    assert run.returncode == 0 and run.stdout.strip() == "ok", run.stderr[-2000:]
