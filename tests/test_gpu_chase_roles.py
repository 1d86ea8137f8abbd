"""The chase kernel where its split changes: fewer, exactly and more bulges
than its warps take at a time (8), windows just below, at and above one and
two columns per lane (32, 64) and the largest, the longest chain; and blocks
that leave the fast reflectors (diagonal T, zero bulge columns, entries far
from 1).  A sweep through one window is an orthogonal equivalence within
50 n eps that returns a Hessenberg-triangular pencil."""
import ctypes

import numpy as np
import pytest
import torch

from conftest import EPS

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def solver(pkg):
    s = pkg.Solver(0)
    yield s
    s.close()


def _chase(pkg, solver, H, T, nb, coef):
    n = H.shape[0]
    bul, tmax = [], 0
    for k in range(nb):
        base, tlo = -3 * k, 3 * k
        thi = (n - 1) - base
        bul += [base, tlo, thi, 1]
        tmax = max(tmax, thi)
    dH, dT = (torch.from_numpy(M.T.copy()).cuda() for M in (H, T))
    dU = torch.zeros(n * n, dtype=torch.float64, device="cuda")
    dV = torch.zeros_like(dU)
    rc = pkg.lib().b200qz_chase_window(solver.handle, dH.data_ptr(), dT.data_ptr(), n, 0, n, n - 1,
                                       (ctypes.c_int * len(bul))(*bul), (ctypes.c_double * len(coef))(*coef), nb,
                                       tmax, dU.data_ptr(), dV.data_ptr())
    assert rc == 0
    return (dH.cpu().numpy().T, dT.cpu().numpy().T, dU.cpu().numpy().reshape(n, n).T,
            dV.cpu().numpy().reshape(n, n).T)


def _check(H, T, out):
    S, P, U, V = out
    n = H.shape[0]
    eye = np.eye(n)
    for A, B in ((H, S), (T, P)):
        m = np.abs(A).max()
        assert np.linalg.norm(U @ (B / m) @ V.T - A / m) <= 50 * n * EPS * np.linalg.norm(A / m)
    assert np.linalg.norm(U.T @ U - eye) <= 50 * n * EPS and np.linalg.norm(V.T @ V - eye) <= 50 * n * EPS
    assert not np.any(np.tril(S, -2)) and not np.any(np.tril(P, -1))


@pytest.mark.parametrize("n,nb", [(5, 1), (12, 1), (31, 7), (32, 8), (33, 9), (40, 8), (63, 16), (64, 17), (65, 8),
                                  (66, 9), (79, 24), (80, 1), (80, 26)])
def test_chase_splits(pkg, solver, n, nb):
    rng = np.random.default_rng(1000 * n + nb)
    H = np.triu(rng.standard_normal((n, n)), -1)
    T = np.triu(rng.standard_normal((n, n)))
    T[np.arange(n), np.arange(n)] += np.sign(T[np.arange(n), np.arange(n)])
    coef = []
    for b in range(nb):
        a, c = rng.standard_normal(2)
        coef += [1.0, 2 * a, a * a + (c * c if b % 2 else -c * c)]
    _check(H, T, _chase(pkg, solver, H, T, nb, coef))


@pytest.mark.parametrize("kind", ["diagonal_t", "zero_sub", "tiny", "huge", "parallel"])
@pytest.mark.parametrize("n,nb", [(24, 3), (64, 9)])
def test_chase_blocks(pkg, solver, n, nb, kind):
    rng = np.random.default_rng(n + len(kind))
    H = np.triu(rng.standard_normal((n, n)), -1)
    T = np.triu(rng.standard_normal((n, n)))
    T[np.arange(n), np.arange(n)] += np.sign(T[np.arange(n), np.arange(n)])
    if kind == "diagonal_t":
        T = np.diag(np.diag(T))
    elif kind == "zero_sub":
        k = np.arange(4, n, 7)
        H[k, k - 1] = 0.0
    elif kind == "tiny":
        H, T = H * 1e-150, T * 1e-150
    elif kind == "huge":
        H, T = H * 1e150, T * 1e150
    elif kind == "parallel":
        # every 3x3 block of T nearly rank one: rows of the bulge blocks nearly parallel
        T = np.triu(np.outer(np.ones(n), 1.0 + 0.1 * rng.standard_normal(n))) + 1e-9 * np.triu(rng.standard_normal((n, n)))
    coef = []
    for b in range(nb):
        a = rng.standard_normal()
        coef += [1.0, 2 * a, a * a + 0.3]
    _check(H, T, _chase(pkg, solver, H, T, nb, coef))
