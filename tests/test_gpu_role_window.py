"""Window QZ with a role per warp, at the window orders where its work split
changes (one or two columns per lane at 32 and 64, one or two rows per
follower thread at 64, the ring of posted steps, the largest window) and on
the inputs that leave its fast rotations: entries whose squares leave the
range, zero bulge columns, zeros on T's diagonal, blocks that split.  Each
is a full small QZ through the window entry: generalized Schur structure,
backward errors and orthogonality within 50 n eps, LAPACK's eigenvalues."""
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


def _pencil(n, kind, seed):
    rng = np.random.default_rng(seed)
    H = np.triu(rng.standard_normal((n, n)), -1)
    T = np.triu(rng.standard_normal((n, n)))
    T[np.arange(n), np.arange(n)] = np.sqrt(np.arange(n, 0, -1)) + 0.1
    if kind == "tiny":
        H *= 1e-160
    elif kind == "huge":
        H, T = H * 1e150, T * 1e150
    elif kind == "zero_t":
        k = rng.choice(n, max(1, n // 8), replace=False)
        T[k, k] = 0.0
    elif kind == "split":
        k = np.arange(3, n, 5)
        H[k, k - 1] = 0.0
    elif kind == "sparse":
        # few entries off the band: reflections of a vector with zeros
        H = np.triu(np.tril(H, 1), -1)
        T = np.diag(np.diag(T))
    elif kind == "graded":
        d = 10.0 ** (-np.linspace(0, 6, n))
        H, T = d[:, None] * H, d[:, None] * T
    return np.asfortranarray(H), np.asfortranarray(T)


def _window_qz(pkg, solver, H, T):
    n = H.shape[0]
    dev = [torch.from_numpy(M.T.copy()).cuda() for M in (H, T)]
    q = torch.zeros(n, n, dtype=torch.float64, device="cuda")
    z = torch.zeros_like(q)
    sh = torch.zeros(3 * n, dtype=torch.float64, device="cuda")
    info = (ctypes.c_int * 3)()
    rc = pkg.lib().b200qz_aed_window(solver.handle, dev[0].data_ptr(), dev[1].data_ptr(), n, 0, 0, n - 1,
                                     q.data_ptr(), z.data_ptr(), sh.data_ptr(), info)
    assert rc == 0 and info[1] == 0, (rc, list(info))
    return [np.asfortranarray(t.cpu().numpy().T) for t in (dev[0], dev[1], q, z)], list(info)


@pytest.mark.parametrize("n", [2, 3, 4, 5, 31, 32, 33, 34, 35, 48, 63, 64, 65, 66, 79, 80])
@pytest.mark.parametrize("kind", ["dense", "zero_t", "split"])
def test_window_orders(pkg, lapack, solver, n, kind):
    H, T = _pencil(n, kind, 100 * n + len(kind))
    (S, P, Q, Z), info = _window_qz(pkg, solver, H, T)
    r = lapack.residuals(H, T, S, P, Q, Z)
    for key in ("h", "t", "q", "z"):
        assert r[key] <= 50 * r["neps"], (key, r)
    assert lapack.schur_structure_ok(S, P)
    So, Po, ar, ai, be, _, _, _ = lapack.dhgeqz(H, T)
    ok, ratio, _ = lapack.match_eigenvalues((ar, ai, be), lapack.eig_from_schur(S, P),
                                            lapack.eig_tolerance(So, Po, H, T))
    assert ok, ratio


@pytest.mark.parametrize("n", [3, 33, 48, 80])
@pytest.mark.parametrize("kind", ["tiny", "huge", "sparse", "graded"])
def test_window_ranges(pkg, lapack, solver, n, kind):
    """Backward errors and structure only: far from 1 the oracle's own
    eigenvalues under- and overflow."""
    H, T = _pencil(n, kind, 7 * n + len(kind))
    (S, P, Q, Z), info = _window_qz(pkg, solver, H, T)
    eye = np.eye(n)
    assert np.abs(Q.T @ Q - eye).max() <= 50 * n * EPS and np.abs(Z.T @ Z - eye).max() <= 50 * n * EPS
    for A, B in ((H, S), (T, P)):
        m = np.abs(A).max()
        assert np.linalg.norm(Q @ (B / m) @ Z.T - A / m) <= 50 * n * EPS * np.linalg.norm(A / m)
    assert not np.any(np.tril(S, -2)) and not np.any(np.tril(P, -1))
    sub = np.diag(S, -1) != 0.0
    assert not np.any(sub[1:] & sub[:-1])
