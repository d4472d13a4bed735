"""Cases for measuring the framework: what a DMRG / TDVP program has it do, through the
package's public entry points, from the smallest bonds near the ends of a chain to the
largest of the two-site H_eff*x benchmark.

Kinds (the values of a case's "kind"):
  heff      one application of a prepared effective Hamiltonian (HeffOp.__call__), one or two
            sites, real or complex, in one of the precisions of the contraction
  solve     the eigenproblem of one DMRG2 bond: a new operator on the bond's environments and
            the Lanczos solve on it (simple_lanczos_solver)
  exp       the evolution of one TDVP1 site: a new one-site operator and its Krylov exponential
  env       the environment updates of one site in both directions (updateleft, updateright)
  u1        one application of the block-sparse (U(1)) two-site operator at a centre bond
  split     the truncated split of a two-site tensor by the density matrix (dm_split)
  gradient  one TDVP1 step and its reverse pass (tdvp1_gradient)

All inputs have the structure of a chain's: Hermitian environments whose identity channel is
the identity and whose other channels are projected operators of norm about 1 (the last one
a block energy), and states whose entries fall off along both bonds as Schmidt values do.
Device data is FP64 (complex: real plane, then imaginary plane), column-major.
"""

import math

import numpy as np
import torch

import finitemptools_gb300 as fm
from finitemptools_gb300 import adjoint
from finitemptools_gb300.auxiliary import dm_split, gemm

CHANNELS = {"tfi": 3, "xxz": 5, "j1j2": 8}


# ------------------------------------------------------------------ cases
def listed():
    return [
        # a bond near the end of a chain (bond dimension 2^5): latency and launches
        _heff("small bond, fp64", 32, 32, "xxz", 2, "fp64"),
        # the benchmark's H_eff*x: its headline form and size
        _heff("benchmark bond, fp64_tc", 2048, 2048, "xxz", 2, "fp64_tc"),
        # a truncated J1-J2 bond: odd dimensions, the wider MPO
        _heff("ragged j1j2 bond, fp64_tc", 683, 701, "j1j2", 2, "fp64_tc"),
        # an ordinary bond of the FP64-accurate form
        _heff("ordinary bond, fp64_tc", 256, 256, "xxz", 2, "fp64_tc"),
        # the lowest precision of the precision table
        _heff("large bond, bf16", 1024, 1024, "xxz", 2, "bf16"),
        # the solve of a D = 64 chain's bond (the FP64 DMRG2 of the benchmark)
        {"name": "bond solve, fp64", "kind": "solve", "dl": 64, "dr": 64, "model": "xxz",
         "precision": "fp64", "vectors": 20, "reorth": False},
        # the solve of the mixed-precision sweep
        {"name": "bond solve, tf32x3", "kind": "solve", "dl": 256, "dr": 256, "model": "xxz",
         "precision": "tf32x3", "vectors": 20, "reorth": True},
        # one site of the TDVP1 benchmark (transverse-field Ising chain, complex state)
        {"name": "site exponential", "kind": "exp", "dl": 64, "dr": 64, "model": "tfi",
         "vectors": 20, "dt": 0.05},
        # the environments of a D = 1024 site
        {"name": "environments, fp64_tc", "kind": "env", "dl": 1024, "dr": 1024, "model": "xxz",
         "precision": "fp64_tc", "complex": False},
        # the centre bond of a long Sz = 0 chain
        {"name": "u1 centre bond", "kind": "u1", "length": 64, "dim": 512},
        # the split of a D = 128 bond's two-site tensor
        {"name": "bond split", "kind": "split", "dl": 128, "dr": 128, "keep": 128, "side": 0,
         "complex": False},
        # forward and reverse pass of the differentiable TDVP1
        {"name": "tdvp1 gradient", "kind": "gradient", "length": 8, "dim": 16, "dt": 0.05},
    ]


def _heff(name, dl, dr, model, sites, precision, cplx=False):
    return {"name": name, "kind": "heff", "dl": dl, "dr": dr, "model": model, "sites": sites,
            "precision": precision, "complex": cplx}


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def pair(lo, hi):
        dl = size(lo, hi)
        return dl, max(lo, min(hi, int(round(dl * rng.uniform(0.6, 1.4)))))

    kind = rng.choice(["heff", "heff", "heff", "solve", "exp", "env", "u1", "split", "gradient"])
    model = rng.choice(sorted(CHANNELS))
    if kind == "heff":
        precision = rng.choice(["fp64", "fp64_tc", "fp64_tc", "bf16", "tf32", "tf32x3"])
        cplx = precision in ("fp64", "fp64_tc") and rng.random() < 0.3
        hi = {"fp64": 192, "fp64_tc": 1400}.get(precision, 2048)
        dl, dr = pair(8 if precision == "fp64" else 64, hi // 2 if cplx else hi)
        case = _heff(None, dl, dr, model, rng.choice([1, 2, 2]), precision, cplx)
        del case["name"]
        return case
    if kind == "solve":
        precision = rng.choice(["fp64", "fp64_tc", "tf32x3"])
        dl, dr = pair(*{"fp64": (12, 128), "fp64_tc": (64, 400), "tf32x3": (64, 400)}[precision])
        return {"kind": kind, "dl": dl, "dr": dr, "model": model, "precision": precision,
                "vectors": rng.randint(8, 24), "reorth": precision == "tf32x3"}
    if kind == "exp":
        dl, dr = pair(8, 100)
        return {"kind": kind, "dl": dl, "dr": dr, "model": model,
                "vectors": rng.choice([20, 30]), "dt": 0.05}
    if kind == "env":
        precision = rng.choice(["fp64", "fp64_tc"])
        cplx = rng.random() < 0.3
        dl, dr = pair(*((16, 200) if precision == "fp64" else (64, 600 if cplx else 1200)))
        return {"kind": kind, "dl": dl, "dr": dr, "model": model, "precision": precision,
                "complex": cplx}
    if kind == "u1":
        return {"kind": kind, "length": 2 * rng.randint(10, 40), "dim": size(32, 800)}
    if kind == "split":
        dl, dr = pair(8, 200)
        return {"kind": kind, "dl": dl, "dr": dr, "keep": max(2, min(dl, dr) - rng.randint(0, 5)),
                "side": rng.randint(0, 1), "complex": rng.random() < 0.5}
    return {"kind": kind, "length": rng.randint(4, 8), "dim": rng.randint(4, 16),
            "dt": rng.uniform(0.02, 0.05)}


# ------------------------------------------------- MPO tensors and made-up chains
def _mpo(model, field=0.7):
    """Bulk Schur tensor W[wl, s_out, wr, s_in] of a spin chain in the Pauli convention."""
    sp, sm = np.array([[0.0, 0.0], [1.0, 0.0]]), np.array([[0.0, 1.0], [0.0, 0.0]])
    x, z, one = sp + sm, np.diag([-1.0, 1.0]), np.eye(2)
    w = CHANNELS[model]
    W = np.zeros((w, 2, w, 2))
    W[0, :, 0, :] = W[w - 1, :, w - 1, :] = one
    if model == "tfi":
        W[0, :, 1, :], W[0, :, 2, :], W[1, :, 2, :] = -z, -field * x, z
    elif model == "xxz":
        for c, (a, b) in enumerate([(2 * sp, sm), (2 * sm, sp), (z, z)], 1):
            W[0, :, c, :], W[c, :, 4, :] = a, b
    else:
        for c, (a, b) in enumerate([(sp, 2 * sm), (sm, 2 * sp), (z, z)], 1):
            W[0, :, c, :], W[c, :, 7, :], W[c + 3, :, 7, :] = a, b, 0.5 * b
            W[c, :, c + 3, :] = one
    return W


def _random(gen, shape, cplx):
    r = torch.randn(shape, generator=gen, device="cuda", dtype=torch.float64)
    if not cplx:
        return r
    return torch.complex(r, torch.randn(shape, generator=gen, device="cuda", dtype=torch.float64))


def _environment(gen, dim, model, cplx, left):
    """h[a', w, a] of a block: the identity in the channel where nothing has started (left)
    or all has ended (right), raising and lowering operators as adjoint pairs, the others
    Hermitian, the block's energy in the last channel (right: the first)."""
    w = CHANNELS[model]
    h = torch.zeros((dim, w, dim), device="cuda",
                    dtype=torch.complex128 if cplx else torch.float64)
    ident, energy = (0, w - 1) if left else (w - 1, 0)
    pairs = {"tfi": [], "xxz": [(1, 2)], "j1j2": [(1, 2), (4, 5)]}[model]
    h[:, ident, :] = torch.eye(dim, device="cuda", dtype=h.dtype)
    for p, q in pairs:
        m = _random(gen, (dim, dim), cplx) / (2 * math.sqrt(dim))
        h[:, p, :], h[:, q, :] = m, m.mH
    for c in set(range(w)) - {ident} - {c for pq in pairs for c in pq}:
        m = _random(gen, (dim, dim), cplx) / (2 * math.sqrt(dim))
        h[:, c, :] = (m + m.mH) * (5.0 if c == energy else 0.7)
    return h


def _falloff(n):
    return 10.0 ** (-4.0 * torch.arange(n, device="cuda", dtype=torch.float64) / n)


def _state(gen, shape, cplx):
    """A normalised state tensor whose entries fall off along its first and last index."""
    x = _random(gen, shape, cplx)
    x *= _falloff(shape[0]).reshape([-1] + [1] * (len(shape) - 1)) * _falloff(shape[-1])
    return x / torch.linalg.vector_norm(x)


def _isometry(gen, rows, cols, cplx):
    q, _ = torch.linalg.qr(_random(gen, (rows, cols), cplx))
    return q


def _site_tensors(gen, dl, dr, cplx):
    """A left-canonical and a right-canonical site tensor [dl, 2, dr] (isometric as far as
    the dimensions allow)."""
    left = _random(gen, (2 * dl, dr), cplx) / math.sqrt(2 * dl)
    right = _random(gen, (dl, 2 * dr), cplx) / math.sqrt(2 * dr)
    return left.reshape(dl, 2, dr), right.reshape(dl, 2, dr)


# ------------------------------------------------------- device tensors and torch
class _Memory:
    """The memory of a DeviceTensor for torch.as_tensor; keeps the tensor alive."""

    def __init__(self, tensor):
        self.tensor = tensor
        n = tensor.nbytes // 8
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": "<f8", "version": 3,
                                         "data": (tensor.ptr, False)}


def _flat(tensor):
    """A DeviceTensor's FP64 values in place (complex: the two planes)."""
    return torch.as_tensor(_Memory(tensor), device="cuda")


def _planes(t):
    """A torch tensor's values in a DeviceTensor's layout."""
    t = t.permute(*reversed(range(t.ndim))).reshape(-1) if t.ndim > 1 else t.reshape(-1)
    return torch.cat([t.real, t.imag]) if t.is_complex() else t


def _device(handle, t):
    d = fm.DeviceTensor(t.shape, np.complex128 if t.is_complex() else np.float64, handle)
    handle.synchronize()
    _flat(d).copy_(_planes(t))
    torch.cuda.synchronize()
    return d


_handle = None


def _get_handle():
    global _handle
    if _handle is None:
        _handle = fm.default_handle()
    return _handle


# ------------------------------------------------------------------ inputs
def _tensors(case, seed):
    """The inputs of a case as torch tensors on the GPU, from the seed alone."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    kind = case["kind"]
    if kind in ("heff", "solve", "exp"):
        cplx = kind == "exp" or bool(case.get("complex"))
        dl, dr = case["dl"], case["dr"]
        sites = {"solve": 2, "exp": 1}.get(kind) or case["sites"]
        return {"left": _environment(gen, dl, case["model"], cplx, True),
                "right": _environment(gen, dr, case["model"], cplx, False),
                "x": _state(gen, (dl,) + (2,) * sites + (dr,), cplx)}
    if kind == "env":
        cplx, dl, dr = case["complex"], case["dl"], case["dr"]
        a, b = _site_tensors(gen, dl, dr, cplx)
        return {"left": _environment(gen, dl, case["model"], cplx, True),
                "right": _environment(gen, dr, case["model"], cplx, False), "a": a, "b": b}
    if kind == "split":
        m, n = 2 * case["dl"], 2 * case["dr"]
        r = min(m, n)
        s = 10.0 ** (-3.0 * torch.arange(r, device="cuda", dtype=torch.float64) / r)
        u, v = (_isometry(gen, k, r, case["complex"]) for k in (m, n))
        return {"x": (u * s) @ v.mH / torch.linalg.vector_norm(s)}
    if kind == "u1":
        legs = _u1_legs(case)
        out = {}
        for name, leg in (("left", legs[0]), ("right", legs[1])):
            q = torch.tensor(np.repeat(list(leg), list(leg.values())), device="cuda")
            dim = len(q)
            h = _environment(gen, dim, "xxz", False, name == "left")
            mask = q[:, None, None] == q[None, None, :] + torch.tensor(_U1_CHANNELS,
                                                                       device="cuda")[:, None]
            out[name] = h * mask
        out["x"] = _random(gen, (_u1_blocks(legs)[1],), False)
        out["x"] /= torch.linalg.vector_norm(out["x"])
        return out
    length, dims = case["length"], _chain_dims(case)
    rng = np.random.default_rng(seed)
    return {"fields": 0.7 + 0.3 * rng.random(length),
            # a right-canonical complex state
            "sites": [_isometry(gen, 2 * dims[i + 1], dims[i], True).mH.reshape(
                dims[i], 2, dims[i + 1]).contiguous() for i in range(length)]}


def _chain_dims(case):
    n = case["length"]
    return [min(case["dim"], 2 ** i, 2 ** (n - i)) for i in range(n + 1)]


# U(1) legs: charges (up spins) of half filling with the product states' shares of dim
_U1_CHANNELS = [0, 1, -1, 0, 0]


def _u1_legs(case):
    n = case["length"]

    def leg(i):
        caps = {q: min(math.comb(i, q), math.comb(n - i, n // 2 - q))
                for q in range(max(0, n // 2 - (n - i)), min(i, n // 2) + 1)}
        total = sum(caps.values())
        if total <= case["dim"]:
            return caps
        return {q: max(1, min(c, case["dim"] * c // total)) for q, c in caps.items()}

    return leg(n // 2 - 1), leg(n // 2 + 1)


def _u1_blocks(legs):
    """The allowed blocks (row offset, rows, s1, s2, column offset, columns) of the packed
    two-site vector, in its order, and its length."""
    def offsets(leg):
        o, out = 0, []
        for q, d in leg.items():
            out.append((q, o, d))
            o += d
        return out

    blocks, total = [], 0
    for qr, ob, db in offsets(legs[1]):
        for s2 in range(2):
            for s1 in range(2):
                for ql, oa, da in offsets(legs[0]):
                    if ql + s1 + s2 == qr:
                        blocks.append((oa, da, s1, s2, ob, db))
                        total += da * db
    return blocks, total


def prepare(case, seed):
    kind, handle, t = case["kind"], _get_handle(), _tensors(case, seed)
    if kind == "gradient":
        h = [float(f) for f in t["fields"]]
        state = {"mpo": fm.tfi_mpo(h), "dt": case["dt"], "site": (case["length"] + 1) // 2,
                 "psi": fm.FiniteMPS([_device(handle, a) for a in t["sites"]])}
        return dict(state, kind=kind)
    state = {k: _device(handle, v) for k, v in t.items()}
    state["kind"] = kind
    if kind in ("heff", "solve", "exp", "env"):
        state["W"] = _mpo(case["model"])
    if kind == "heff":
        two = case["sites"] == 2
        if case["complex"] and case["precision"] not in ("fp64", "fp64_tc"):
            raise ValueError("the complex cases are FP64")
        state["op"] = fm.HeffOp("ac2" if two else "ac", state["left"], state["right"],
                                W1=state["W"], W2=state["W"] if two else None,
                                precision=case["precision"], dtype=state["x"].dtype)
    elif kind == "u1":
        vl, vr = (fm.U1Space(leg) for leg in _u1_legs(case))
        W = _mpo("xxz")
        state["op"] = fm.U1HeffOp(state["left"], state["right"], W, W, vl, vr, (0, 1), (0, 1),
                                  _U1_CHANNELS, _U1_CHANNELS, _U1_CHANNELS)
    elif kind == "split":
        state.update(m=2 * case["dl"], n=2 * case["dr"], side=case["side"],
                     trunc=fm.MPSTruncation(case["keep"], 1e-10))
    else:
        state.update({k: case[k] for k in ("precision", "vectors", "reorth", "dt") if k in case})
    if kind in ("heff", "u1"):
        # the operator and the output vector stay, as in a solver's loop
        state["y"] = fm.DeviceTensor(state["x"].shape, state["x"].dtype, handle)
        state["out"] = _flat(state["y"])
    torch.cuda.synchronize()
    return state


# -------------------------------------------------------------------- one pass
def run(s):
    kind = s["kind"]
    if kind in ("heff", "u1"):
        s["op"](s["x"], s["y"])
        return s["out"]
    if kind == "solve":
        op = fm.HeffOp("ac2", s["left"], s["right"], W1=s["W"], W2=s["W"],
                       precision=s["precision"], dtype=s["x"].dtype)
        energy, vec, _, _ = op.lanczos(s["x"], s["vectors"], 1e-12, s["reorth"])
        return [energy, _flat(vec)]
    if kind == "exp":
        op = fm.HeffOp("ac", s["left"], s["right"], W1=s["W"], dtype=s["x"].dtype)
        return _flat(op.exponentiate(-0.5j * s["dt"], s["x"], 1e-8 / (0.5 * s["dt"]),
                                     s["vectors"]))
    if kind == "env":
        return [_flat(fm.updateleft(s["left"], s["a"], s["W"], s["a"], s["precision"])),
                _flat(fm.updateright(s["right"], s["b"], s["W"], s["b"], s["precision"]))]
    if kind == "split":
        a, sv, b, _ = dm_split(s["x"], s["m"], s["n"], s["trunc"], s["side"])
        # the kept two-site tensor, as a sweep forms it for its fidelity
        ab = gemm(a, b, (s["m"], s["n"]), s["m"], s["n"], sv.shape[0])
        return [_flat(a), _flat(sv), _flat(b), _flat(ab)]
    value, grads = adjoint.tdvp1_gradient(s["mpo"], s["psi"], -1j * s["dt"], 1, s["site"],
                                          np.diag([-1.0, 1.0]), checkpoint=1)
    return [value, grads]


# ------------------------------------------------------------ work that is needed
def work(case):
    kind = case["kind"]
    f = 4 if case.get("complex") or kind in ("exp", "gradient") else 1    # real FMAs per FMA
    b = 16 if f == 4 else 8
    if kind in ("heff", "solve", "exp"):
        dl, dr, w = case["dl"], case["dr"], CHANNELS[case["model"]]
        p = 2 ** ({"solve": 2, "exp": 1}.get(kind) or case["sites"])
        flops = 2 * f * w * p * dl * dr * (dl + dr)
        data = b * (w * (dl * dl + dr * dr) + 2 * p * dl * dr)
        return {"bytes": data, "flops": flops * case.get("vectors", 1)}
    if kind == "env":
        dl, dr, w = case["dl"], case["dr"], CHANNELS[case["model"]]
        return {"bytes": b * (2 * w * (dl * dl + dr * dr) + 4 * dl * dr),
                "flops": 2 * 2 * f * w * 2 * dl * dr * (dl + dr)}
    if kind == "u1":
        legs = _u1_legs(case)
        blocks, n = _u1_blocks(legs)
        left, right = legs
        flops, data = 0, 0
        # L.x and .R over the allowed channel blocks; the middle leg's charge is the block's
        for _, da, _, _, _, db in blocks:
            flops += 2 * 5 * da * db * (da + db)
        for leg in (left, right):
            data += sum(8 * d * (3 * d + leg.get(q + 1, 0) + leg.get(q - 1, 0))
                        for q, d in leg.items())
        return {"bytes": data + 16 * n, "flops": flops}
    if kind == "split":
        m, n, k = 2 * case["dl"], 2 * case["dr"], case["keep"]
        r = m if case["side"] == 0 else n
        # the Gram matrix, its eigenvectors, the other factor and the kept tensor
        return {"bytes": b * (2 * m * n + (m + n) * k),
                "flops": f * (m * n * r + 9 * r ** 3 + 4 * m * n * k)}
    dims = _chain_dims(case)
    # per site and pass: about 20 Krylov vectors forward (twice: the reverse pass repeats the
    # forward) and two exponentials with 8 quadrature nodes in reverse, on both half sweeps
    per = sum(2 * f * 3 * 2 * a * c * (a + c) for a, c in zip(dims, dims[1:]))
    sites = 16 * sum(2 * a * c for a, c in zip(dims, dims[1:]))
    return {"bytes": 2 * sites + 16 * 12 * case["length"] * 3, "flops": 2 * per * (2 * 20 + 2 * 28)}


# ------------------------------------------------------------ the same in 64 bits
def _apply(W, left, right, x):
    """H_eff x of one or two sites (left [a', w, a], right [b', w, b])."""
    t = torch.tensordot(left, x, ([2], [0]))                       # a' w s.. b
    if x.ndim == 4:
        t = torch.einsum("xwstb,wpms,mqvt->xpqvb", t, W, W)
        return torch.tensordot(t, right, ([3, 4], [1, 2]))
    t = torch.einsum("xwsb,wpvs->xpvb", t, W)
    return torch.tensordot(t, right, ([2, 3], [1, 2]))


def _exp(apply, t, x):
    """exp(t H) x by Taylor series over steps short enough for 1e-17."""
    steps = max(1, math.ceil(abs(t) * 30.0))
    for _ in range(steps):
        term = x
        for k in range(1, 40):
            term = (t / steps / k) * apply(term)
            x = x + term
    return x


def _update_left(h, a, W, conj):
    return torch.einsum("xwa,asb,wpvs,xpy->yvb", h, a, W, conj)


def _exact_lanczos(apply, x, vectors):
    v, prev = x / torch.linalg.vector_norm(x), None
    alpha, beta = [], []
    for _ in range(vectors):
        y = apply(v)
        alpha.append(float((v * y).sum()))
        y = y - alpha[-1] * v - (beta[-1] * prev if beta else 0)
        beta.append(float(torch.linalg.vector_norm(y)))
        prev, v = v, y / beta[-1]
    return float(np.linalg.eigvalsh(np.diag(alpha) + np.diag(beta[:-1], 1) +
                                    np.diag(beta[:-1], -1))[0])


def exact(case, seed):
    kind, t = case["kind"], _tensors(case, seed)
    if kind == "gradient":
        return _exact_gradient(case, t)
    if kind == "split":
        u, s, v = torch.linalg.svd(t["x"], full_matrices=False)
        k = case["keep"]
        # the factors' phases are the eigensolver's
        return [None, s[:k].contiguous(), None, _planes((u[:, :k] * s[:k]) @ v[:k])]
    cplx = t["left"].is_complex()
    W = torch.tensor(_mpo(case.get("model", "xxz")), device="cuda",
                     dtype=torch.complex128 if cplx else torch.float64)
    if kind == "heff":
        return _planes(_apply(W, t["left"], t["right"], t["x"]))
    if kind == "solve":
        return [_exact_lanczos(lambda v: _apply(W, t["left"], t["right"], v), t["x"],
                               case["vectors"]), None]
    if kind == "exp":
        return _planes(_exp(lambda v: _apply(W, t["left"], t["right"], v), -0.5j * case["dt"],
                            t["x"]))
    if kind == "env":
        def update(h, x, conj):
            y = torch.tensordot(h, x, ([2], [0]))                  # x w s b
            y = torch.einsum("xwsb,wpvs->xpvb", y, W)
            return torch.tensordot(conj, y, ([0, 1], [0, 1]))      # y v b
        left = update(t["left"], t["a"], t["a"].conj())
        y = torch.tensordot(t["b"], t["right"], ([2], [2]))        # a s y v
        y = torch.einsum("asyv,wpvs->ypwa", y, W)
        right = torch.tensordot(t["b"].conj(), y, ([2, 1], [0, 1]))
        return [_planes(left), _planes(right)]
    blocks, _ = _u1_blocks(_u1_legs(case))
    dense = torch.zeros((len(t["left"]), 2, 2, len(t["right"])), device="cuda",
                        dtype=torch.float64)
    o = 0
    for oa, da, s1, s2, ob, db in blocks:
        dense[oa:oa + da, s1, s2, ob:ob + db] = t["x"][o:o + da * db].reshape(db, da).T
        o += da * db
    y = _apply(W, t["left"], t["right"], dense)
    return torch.cat([y[oa:oa + da, s1, s2, ob:ob + db].T.reshape(-1)
                      for oa, da, s1, s2, ob, db in blocks])


def _exact_gradient(case, t):
    """One TDVP1 sweep written out, with the gradient by torch's own reverse mode."""
    n, dt = case["length"], -1j * case["dt"]
    Ws = [torch.tensor(_mpo("tfi", float(f)), device="cuda", dtype=torch.complex128)
          .requires_grad_() for f in t["fields"]]
    a = list(t["sites"])

    def end(c):
        e = torch.zeros((1, 3, 1), device="cuda", dtype=torch.complex128)
        e[0, c, 0] = 1
        return e

    def update_right(h, x, W):
        return torch.einsum("yvb,asb,wpvs,xpy->xwa", h, x, W, x.conj())

    def c_apply(left, right):
        return lambda c: torch.einsum("xwa,ab,ywb->xy", left, c, right)

    left, right = [end(0)], [end(2)]
    for i in range(n - 1, 0, -1):
        right.append(update_right(right[-1], a[i], Ws[i]))
    right = right[::-1]                      # right[i]: the environment right of site i
    for i in range(n - 1):
        x = _exp(lambda v: _apply(Ws[i], left[i], right[i], v), dt / 2, a[i])
        q, r = torch.linalg.qr(x.reshape(-1, x.shape[2]))
        a[i] = q.reshape(x.shape[0], 2, -1)
        left.append(_update_left(left[i], a[i], Ws[i], a[i].conj()))
        r = _exp(c_apply(left[i + 1], right[i]), -dt / 2, r)
        a[i + 1] = torch.tensordot(r, a[i + 1], 1)
    a[n - 1] = _exp(lambda v: _apply(Ws[n - 1], left[n - 1], right[n - 1], v), dt, a[n - 1])
    for i in range(n - 2, -1, -1):
        x = a[i + 1]
        q, r = torch.linalg.qr(x.reshape(x.shape[0], -1).mH)
        a[i + 1] = q.mH.reshape(-1, 2, x.shape[2])
        right[i] = update_right(right[i + 1], a[i + 1], Ws[i + 1])
        c = _exp(c_apply(left[i + 1], right[i]), -dt / 2, r.mH)
        a[i] = torch.tensordot(a[i], c, 1)
        a[i] = _exp(lambda v: _apply(Ws[i], left[i], right[i], v), dt / 2, a[i])
    z = torch.diag(torch.tensor([-1.0, 1.0], device="cuda", dtype=torch.complex128))
    h1 = h0 = torch.ones((1, 1), device="cuda", dtype=torch.complex128)
    for i in range(n):
        o = z if i == (n + 1) // 2 - 1 else torch.eye(2, device="cuda", dtype=torch.complex128)
        h1 = torch.einsum("xa,asb,ps,xpy->yb", h1, a[i], o, a[i].conj())
        h0 = torch.einsum("xa,asb,xsy->yb", h0, a[i], a[i].conj())
    value = (h1 / h0).real.sum()
    grads = torch.autograd.grad(value, Ws)
    return [float(value), [g.cpu().numpy() for g in grads]]
