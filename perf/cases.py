"""Performance cases of the framework: whole solves of Hessenberg-triangular
pencils, batches of small pencils, and the steps either side of a solve
(balancing, Hessenberg-triangular reduction, reordering), each through the
entry point that a program calls.

Inputs.  "dense" pencils have the distribution of the Hessenberg-triangular
form of a dense Gaussian pair: normal entries, chi-distributed diagonal of T
and subdiagonal of H, which is what a solve meets after a QR factorisation
and the reduction.  "infinite" sets 5 % of T's diagonal to zero; "graded"
scales rows and columns by 10**u, u ~ U(-1, 1).  Matrices are column-major
(what every entry point takes), held as torch tensors X with X[j, i] the
entry (i, j), so a tensor is the transpose of the matrix.

Outputs.  Q, Z and the triangular factors of a generalized Schur form are not
determined by the pencil: the order in which eigenvalues deflate, signs, and
a rotation inside each complex block are free, so two correct solves of one
pencil differ in every entry.  What is determined comes back whole: the
products Q S Z^T and Q P Z^T (the pencil the factors stand for), Q^T Q and
Z^T Z, the parts of S and P that have to be zero, and all eigenvalues as
points of the Riemann sphere (finite and infinite alike) in order of modulus.
Reductions and balancing, whose results are determined, return them as they
are.
"""
import ctypes
import importlib.util
import math
import os
import random
import sys

import numpy as np
import torch

_DEV = "cuda"
_F64 = torch.float64


def _package():
    """The framework's package (its folder's name is not an identifier)."""
    name = "gevp_pdhgeqz_b200"
    if name not in sys.modules:
        root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
        path = os.path.join(root, "gevp-pdhgeqz_b200", "__init__.py")
        spec = importlib.util.spec_from_file_location(name, path)
        mod = importlib.util.module_from_spec(spec)
        sys.modules[name] = mod
        spec.loader.exec_module(mod)
    return sys.modules[name]


def listed():
    """Twelve cases: six solves from the smallest block to the largest order
    that fits a pass, two batches, and the four steps around a solve."""
    return [
        # one small pencil: a subproblem inside another program's loop; latency
        {"name": "solve_56", "path": "solve", "kind": "dense", "n": 56, "job": "S", "comp": "I"},
        # after gghrd: the given Q, Z are updated (COMPQ = COMPZ = 'V'); odd order
        {"name": "solve_201_v", "path": "solve", "kind": "dense", "n": 201, "job": "S", "comp": "V"},
        # the Fortran drop-in with host arrays, as an unchanged caller uses it
        {"name": "pdhgeqz_400", "path": "host", "kind": "dense", "n": 400, "job": "S", "comp": "I"},
        # eigenvalues only
        {"name": "eigenvalues_901", "path": "solve", "kind": "dense", "n": 901, "job": "E", "comp": "N"},
        # singular T, as in descriptor systems: infinite eigenvalues to deflate first
        {"name": "solve_infinite_700", "path": "solve", "kind": "infinite", "n": 700, "job": "S", "comp": "I"},
        # badly scaled entries: many deflations, few sweeps
        {"name": "solve_graded_2000", "path": "solve", "kind": "graded", "n": 2000, "job": "S", "comp": "I"},
        # the largest ordinary solve: AED, sweeps and far updates all at work
        {"name": "solve_1800", "path": "solve", "kind": "dense", "n": 1800, "job": "S", "comp": "I"},
        # many independent pencils that fit shared memory
        {"name": "batch_small", "path": "batch", "count": 600, "lo": 16, "hi": 80, "mix": 1},
        # uneven batch up to orders that do not fit shared memory
        {"name": "batch_uneven", "path": "batch", "count": 220, "lo": 32, "hi": 300, "mix": 2},
        # dense A, triangular B to Hessenberg-triangular form with Q and Z
        {"name": "gghrd_800", "path": "gghrd", "n": 800},
        # 40 % of the eigenvalues moved to the top, with the projection norms
        {"name": "tgsen_700", "path": "tgsen", "n": 700, "share": 0.4, "ijob": 1},
        # balancing with hidden isolated eigenvalues and bad scaling
        {"name": "ggbal_3000", "path": "ggbal", "n": 3000},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the ranges the listed ones stand for."""
    path = rng.choice(["solve", "solve", "solve", "solve", "host", "batch", "batch", "gghrd", "tgsen", "ggbal"])
    if path == "solve":
        kind = rng.choice(["dense", "dense", "infinite", "graded"])
        job, comp = rng.choice([("S", "I"), ("S", "I"), ("S", "V"), ("E", "N")])
        return {"path": path, "kind": kind, "n": _log_int(rng, 24, 1800), "job": job, "comp": comp}
    if path == "host":
        return {"path": path, "kind": rng.choice(["dense", "graded"]), "n": _log_int(rng, 24, 1000), "job": "S",
                "comp": rng.choice(["I", "V"])}
    if path == "batch":
        lo = rng.randint(8, 48)
        if rng.random() < 0.5:
            return {"path": path, "count": rng.randint(100, 600), "lo": lo, "hi": rng.randint(lo + 8, 80),
                    "mix": rng.randrange(1000)}
        return {"path": path, "count": rng.randint(60, 220), "lo": lo, "hi": rng.randint(100, 300),
                "mix": rng.randrange(1000)}
    if path == "gghrd":
        return {"path": path, "n": _log_int(rng, 48, 800)}
    if path == "tgsen":
        return {"path": path, "n": _log_int(rng, 48, 700), "share": round(rng.uniform(0.1, 0.7), 3),
                "ijob": rng.choice([0, 1])}
    return {"path": path, "n": _log_int(rng, 200, 3000)}


def _sizes(case):
    r = random.Random(case["mix"])
    return [r.randint(case["lo"], case["hi"]) for _ in range(case["count"])]


def work(case):
    """Bytes: each input read once, each output written once.  Flops: for a
    solve with Q and Z about 20 n^3, for eigenvalues alone 8 n^3 (the counts of
    multishift QZ with early deflation on these inputs, not of the classical
    double-shift iteration); reduction 14 n^3 + Q and Z (DGGHRD); reordering
    24 n flops for each of the swaps the selection needs."""
    if case["path"] in ("solve", "host"):
        n = case["n"]
        if case["job"] == "E":
            return {"bytes": 8.0 * (2 * n * n + 3 * n), "flops": 8.0 * n ** 3}
        return {"bytes": 8.0 * ((6 if case["comp"] == "I" else 8) * n * n + 3 * n), "flops": 20.0 * n ** 3}
    if case["path"] == "batch":
        ns = _sizes(case)
        return {"bytes": 8.0 * sum(6 * n * n + 3 * n for n in ns), "flops": 20.0 * sum(float(n) ** 3 for n in ns)}
    n = case["n"]
    if case["path"] == "gghrd":
        return {"bytes": 8.0 * 6 * n * n, "flops": 14.0 * n ** 3}
    if case["path"] == "tgsen":
        swaps = case["share"] * (1 - case["share"]) * n * n / 8
        return {"bytes": 8.0 * 8 * n * n, "flops": 192.0 * n * swaps}
    return {"bytes": 8.0 * 4 * n * n, "flops": 10.0 * n * n}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _gen(seed):
    g = torch.Generator(device=_DEV)
    g.manual_seed(int(seed))
    return g


def _randn(g, *shape):
    return torch.randn(*shape, dtype=_F64, device=_DEV, generator=g)


def _chi(g, dof):
    """Chi-distributed values of the given degrees of freedom (the normal
    approximation with mean sqrt(k - 1/2) and variance 1/2), positive."""
    return (torch.sqrt(dof - 0.5) + math.sqrt(0.5) * _randn(g, dof.numel())).abs() + 1e-3


def _pencil(kind, n, g):
    """(H, T) of order n, transposed (see above)."""
    h = torch.tril(_randn(g, n, n), 1)
    t = torch.tril(_randn(g, n, n))
    k = torch.arange(n, 0, -1, dtype=_F64, device=_DEV)
    d = _chi(g, k)
    if kind == "infinite":
        d[torch.randperm(n, device=_DEV, generator=g)[: max(1, n // 20)]] = 0.0
    t.diagonal().copy_(d)
    if n > 1:
        h.diagonal(1).copy_(_chi(g, k[:-1]))
    if kind == "graded":
        r = 10.0 ** (2.0 * torch.rand(n, dtype=_F64, device=_DEV, generator=g) - 1.0)
        c = 10.0 ** (2.0 * torch.rand(n, dtype=_F64, device=_DEV, generator=g) - 1.0)
        h *= c[:, None] * r[None, :]
        t *= c[:, None] * r[None, :]
    return h, t


def _orthogonal(n, g):
    return torch.linalg.qr(_randn(g, n, n))[0]


def _schur_form(case, g, seed):
    """A generalized real Schur form with the entries of a dense Gaussian
    pair's (normal above the diagonal, blocks of size sqrt(n)), nine in ten
    blocks complex pairs, and the selection."""
    n = case["n"]
    s = torch.tril(_randn(g, n, n), -1).cpu().numpy()
    t = torch.tril(_randn(g, n, n), -1).cpu().numpy()
    r = random.Random(int(seed) + 77)
    select = np.zeros(n, dtype=np.int32)
    j = 0
    while j < n:
        th = 0.5 * math.acos(r.uniform(-1.0, 1.0))
        size = 2 if j + 1 < n and r.random() < 0.9 else 1
        b0 = math.sqrt(n) * math.cos(th) + 1e-3
        if size == 2:
            ph, d, b1 = math.acos(r.uniform(-0.99, 0.99)), r.uniform(0.5, 2.0), b0 * r.uniform(0.5, 1.0)
            a, b = math.tan(th) * math.cos(ph), math.tan(th) * math.sin(ph)
            s[j, j], s[j + 1, j], s[j, j + 1], s[j + 1, j + 1] = b0 * a, b0 * b * d, -b1 * b / d, b1 * a
            t[j, j], t[j + 1, j], t[j + 1, j + 1] = b0, 0.0, b1
        else:
            s[j, j], t[j, j] = r.choice([-1.0, 1.0]) * math.sqrt(n) * math.sin(th), b0
        if r.random() < case["share"]:
            select[j:j + size] = 1
        j += size
    return torch.from_numpy(s).to(_DEV), torch.from_numpy(t).to(_DEV), select


def _balance_pencil(n, g):
    """Block-triangular pencil with 64 isolatable rows and columns under a
    random permutation, graded over six decades."""
    k = min(64, n // 4)
    a, b = _randn(g, n, n), _randn(g, n, n)
    for m in (a, b):
        # transposed storage: row index of the tensor is the matrix column
        for lo, hi in ((0, k), (n - k, n)):
            m[lo:hi, lo:hi] = torch.triu(m[lo:hi, lo:hi].T).T
        m[:k, k:] = 0.0
        m[:n - k, n - k:] = 0.0
    d = 10.0 ** (6.0 * torch.rand(2, n, dtype=_F64, device=_DEV, generator=g) - 3.0)
    p = torch.randperm(n, device=_DEV, generator=g)
    return tuple((m * d[0][:, None] * d[1][None, :])[p][:, p].contiguous() for m in (a, b))


def _inputs(case, seed):
    """The case's inputs, from the seed alone."""
    g = _gen(seed)
    path = case["path"]
    if path in ("solve", "host"):
        x = {"h": None, "t": None}
        x["h"], x["t"] = _pencil(case["kind"], case["n"], g)
        if case["comp"] == "V":
            x["q"], x["z"] = _orthogonal(case["n"], g), _orthogonal(case["n"], g)
        return x
    if path == "batch":
        pen = [_pencil("dense", n, g) for n in _sizes(case)]
        return {"h": torch.cat([p[0].reshape(-1) for p in pen]), "t": torch.cat([p[1].reshape(-1) for p in pen])}
    n = case["n"]
    if path == "gghrd":
        h, t = _randn(g, n, n), torch.tril(_randn(g, n, n))
        t.diagonal().copy_(_chi(g, torch.arange(n, 0, -1, dtype=_F64, device=_DEV)))
        return {"h": h, "t": t}
    if path == "tgsen":
        s, t, select = _schur_form(case, g, seed)
        return {"h": s, "t": t, "q": _orthogonal(n, g), "z": _orthogonal(n, g), "select": select}
    a, b = _balance_pencil(n, g)
    return {"h": a, "t": b}


def _padding(ns):
    """Positions of every pencil's entries in a stack padded to the largest
    order (the identity's diagonal fills the rest)."""
    top = max(ns)
    where = []
    for p, n in enumerate(ns):
        i = torch.arange(n, device=_DEV)
        where.append(((p * top + i[:, None]) * top + i[None, :]).reshape(-1))
    return top, torch.cat(where)


def prepare(case, seed):
    """Inputs, work buffers and the solver context that a program keeps."""
    pkg = _package()
    x = _inputs(case, seed)
    st = {"case": case, "pkg": pkg, "in": x, "solver": pkg.Solver(0)}
    path = case["path"]
    if path == "host":
        st["host"] = {k: np.asfortranarray(v.cpu().numpy().T) for k, v in x.items()}
        st["buf"] = {k: np.zeros((case["n"], case["n"]), order="F") for k in ("h", "t", "q", "z")}
        return st
    st["buf"] = {k: torch.zeros_like(x["h"]) for k in ("h", "t", "q", "z")}
    if path == "batch":
        ns = _sizes(case)
        st["batch"] = pkg.Batch(ns)
        st["pad"] = _padding(ns)
        st["eig"] = torch.zeros(3, sum(ns), dtype=_F64, device=_DEV)
        st["info"] = torch.zeros(len(ns), dtype=torch.int32, device=_DEV)
        st["pencil_of"] = torch.repeat_interleave(torch.arange(len(ns), device=_DEV),
                                                  torch.tensor(ns, device=_DEV)).to(_F64)
    else:
        st["eig"] = torch.zeros(3, case["n"], dtype=_F64, device=_DEV)
    torch.cuda.synchronize()
    return st


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def _sphere(ar, ai, be, group=None):
    """Eigenvalues (ar + i ai) / be as points of the Riemann sphere, the
    imaginary part by its absolute value (conjugates coincide), in order of
    modulus (within each group)."""
    m = torch.hypot(ar, ai)
    d = m * m + be * be
    points = torch.stack([2 * ar * be / d, 2 * (ai * be).abs() / d, (m * m - be * be) / d])
    order = torch.argsort(torch.log(m) - torch.log(be.abs()), stable=True)
    if group is not None:
        order = order[torch.argsort(group[order], stable=True)]
    return points[:, order]


def _factored(s, p, q, z):
    """What a generalized Schur form stands for (transposed storage: the
    tensor of Q S Z^T is Z~^T S~ Q~); works on stacks too."""
    zt = z.transpose(-1, -2)
    qt = q.transpose(-1, -2)
    return {"QSZt": zt @ s @ q, "QPZt": zt @ p @ q, "QtQ": q @ qt, "ZtZ": z @ zt,
            "below_S": torch.triu(s, 2), "below_P": torch.triu(p, 1)}


def _check(rc):
    if rc != 0:
        raise RuntimeError("the call returned %d" % rc)


def run(st):
    """One pass: the inputs copied to the buffers that the call overwrites
    (it works in place), the call, and its results."""
    case, pkg, x, b, solver = st["case"], st["pkg"], st["in"], st["buf"], st["solver"]
    path = case["path"]
    if path == "host":
        h = st["host"]
        for k, v in h.items():
            b[k][...] = v
        ar, ai, be, info = pkg.pdhgeqz(case["job"], case["comp"], case["comp"], b["h"], b["t"], b["q"], b["z"])
        _check(info)
        s, p, q, z = (torch.from_numpy(b[k].T).to(_DEV) for k in ("h", "t", "q", "z"))
        out = _factored(s, p, q, z)
        out["eig"] = _sphere(*(torch.from_numpy(v).to(_DEV) for v in (ar, ai, be)))
        return out
    for k in ("h", "t", "q", "z"):
        if k in x:
            b[k].copy_(x[k])
    torch.cuda.current_stream().synchronize()  # the solver works on a stream of its own
    ptr = {k: v.data_ptr() for k, v in b.items()}
    if path == "batch":
        e = st["eig"]
        pkg.solve_batched_device(solver, st["batch"], ptr["h"], ptr["t"], ptr["q"], ptr["z"], e[0].data_ptr(),
                                 e[1].data_ptr(), e[2].data_ptr(), st["info"].data_ptr())
        top, where = st["pad"]
        count = st["batch"].count
        full = []
        for k in ("h", "t", "q", "z"):
            m = torch.zeros(count * top * top, dtype=_F64, device=_DEV)
            m[where] = b[k]
            full.append(m.view(count, top, top))
        out = {k: v.reshape(-1)[where] for k, v in _factored(*full).items()}
        out["eig"] = _sphere(e[0], e[1], e[2], st["pencil_of"])
        out["info"] = st["info"].clone()
        return out
    n = case["n"]
    if path == "solve":
        e = st["eig"]
        comp = case["comp"]
        _check(solver.solve_device(ptr["h"], ptr["t"], ptr["q"], ptr["z"], n, n, e[0].data_ptr(), e[1].data_ptr(),
                                   e[2].data_ptr(), job=case["job"], compq=comp, compz=comp))
        out = _factored(b["h"], b["t"], b["q"], b["z"]) if case["job"] == "S" else {}
        out["eig"] = _sphere(e[0], e[1], e[2])
        return out
    if path == "gghrd":
        _check(solver.gghrd_device(ptr["h"], ptr["t"], ptr["q"], ptr["z"], n, n))
        return {k: b[k] for k in ("h", "t", "q", "z")}
    if path == "tgsen":
        e, sel = st["eig"], x["select"]
        m, info = ctypes.c_int(0), ctypes.c_int(0)
        pl, pr = ctypes.c_double(0.0), ctypes.c_double(0.0)
        counts = (ctypes.c_int * 2)()
        dif = (ctypes.c_double * 2)()
        vp, pint = ctypes.c_void_p, ctypes.POINTER(ctypes.c_int)
        _check(pkg.lib().b200qz_tgsen_dev(
            solver.handle, case["ijob"], 1, 1, sel.ctypes.data_as(pint), n, vp(ptr["h"]), n, vp(ptr["t"]), n,
            vp(ptr["q"]), n, vp(ptr["z"]), n, vp(e[0].data_ptr()), vp(e[1].data_ptr()), vp(e[2].data_ptr()),
            ctypes.byref(m), ctypes.byref(pl), ctypes.byref(pr), dif, ctypes.byref(info), counts))
        _check(info.value)
        out = _factored(b["h"], b["t"], b["q"], b["z"])
        out["m"] = m.value
        if case["ijob"] == 1:
            out["pl_pr"] = np.array([pl.value, pr.value])
        lead = torch.arange(n, device=_DEV) < m.value
        out["eig"] = _sphere(e[0], e[1], e[2], (~lead).to(_F64))  # the selected ones, then the others
        return out
    ilo, ihi, ls, rs, info = solver.ggbal_device(ptr["h"], ptr["t"], n, n, "B")
    _check(info)
    return {"h": b["h"], "t": b["t"], "ilo": ilo, "ihi": ihi, "lscale": ls, "rscale": rs}


# ---------------------------------------------------------------------------
# the same in 64 bits, by torch and numpy alone
# ---------------------------------------------------------------------------
def _sphere_of(lam, group=None):
    be = torch.ones(len(lam), dtype=_F64)
    lam = torch.from_numpy(np.asarray(lam, dtype=np.complex128))
    return _sphere(lam.real.clone(), lam.imag.clone(), be, group)


def _eigenvalues(h, t):
    return np.linalg.eigvals(np.linalg.solve(t, h))


def exact(case, seed):
    """What run() returns, where plain linear algebra gives it: the pencil
    itself for the products, the identity, zeros, and the eigenvalues of
    T^-1 H where T is well conditioned and the order moderate.  None for the
    reduction (its own rotations define it) and for balancing."""
    path = case["path"]
    if path in ("gghrd", "ggbal"):
        return None
    x = _inputs(case, seed)
    if path == "batch":
        ns = _sizes(case)
        eyes = torch.cat([torch.eye(n, dtype=_F64).reshape(-1) for n in ns])
        zero = torch.zeros_like(eyes)
        out = {"QSZt": x["h"], "QPZt": x["t"], "QtQ": eyes, "ZtZ": eyes, "below_S": zero, "below_P": zero}
        parts, o = [], 0
        hh, tt = x["h"].cpu().numpy(), x["t"].cpu().numpy()
        for n in ns:
            parts.append(_sphere_of(_eigenvalues(hh[o:o + n * n].reshape(n, n).T, tt[o:o + n * n].reshape(n, n).T)))
            o += n * n
        out["eig"] = torch.cat(parts, 1)
        out["info"] = torch.zeros(len(ns), dtype=torch.int32)
        return out
    n = case["n"]
    out = {}
    if path == "tgsen" or case["job"] == "S":
        h, t = x["h"], x["t"]
        if "q" in x:
            h, t = (x["z"].T @ m @ x["q"] for m in (h, t))
        eye, zero = torch.eye(n, dtype=_F64), torch.zeros(n, n, dtype=_F64)
        out = {"QSZt": h, "QPZt": t, "QtQ": eye, "ZtZ": eye, "below_S": zero, "below_P": zero}
    if path == "tgsen":
        s, t, sel = x["h"].cpu().numpy().T, x["t"].cpu().numpy().T, x["select"]
        lam = np.zeros(n, dtype=np.complex128)
        j = 0
        while j < n:
            k = 2 if j + 1 < n and s[j + 1, j] != 0.0 else 1
            lam[j:j + k] = _eigenvalues(s[j:j + k, j:j + k], t[j:j + k, j:j + k])
            j += k
        out["m"] = int(sel.sum())
        if case["ijob"] == 1:
            out["pl_pr"] = None
        out["eig"] = _sphere_of(lam, torch.from_numpy(1.0 - sel.astype(np.float64)))
    else:
        out["eig"] = None
        if case["kind"] != "infinite" and n <= 1000:
            out["eig"] = _sphere_of(_eigenvalues(x["h"].cpu().numpy().T, x["t"].cpu().numpy().T))
    return out
