"""Reordering where a swap does not go through, or a block does not stay whole.

A swap is rejected when its blocks are not finite (Inf in the entries between
them): the call returns info 1, and what it has done so far is an equivalence
by orthogonal Q and Z.  A 2x2 block whose eigenvalues are a rounding error away
from real may come out of a swap with real ones: it is carried to its place
as two 1x1 blocks."""
import numpy as np
import pytest

from conftest import EPS

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def solver(pkg):
    s = pkg.Solver(0)
    yield s
    s.close()


def _form(n, seed, off):
    """Generalized Schur form of 2x2 blocks with off-diagonal entries off."""
    rng = np.random.default_rng(seed)
    S = np.triu(rng.standard_normal((n, n)), 1)
    T = np.triu(rng.standard_normal((n, n)), 1)
    for j in range(0, n, 2):
        a = rng.uniform(-3.0, 3.0) + 8.0 * (j % 4)
        S[j, j] = S[j + 1, j + 1] = a
        S[j, j + 1], S[j + 1, j] = off
        T[j, j] = T[j + 1, j + 1] = 1.0
        T[j, j + 1] = 0.0
    return np.asfortranarray(S), np.asfortranarray(T)


@pytest.mark.parametrize("n,at", [(8, 2), (60, 30), (200, 80), (200, 150)])
def test_rejected_swap(solver, n, at):
    """Blocks go in pairs, every second one selected; the entries between the
    block at row `at` and the selected one after it hold an Inf."""
    S, T = _form(n, 3 * n, (1.0, -1.0))
    sel = np.zeros(n, dtype=np.int32)
    sel[2::4] = sel[3::4] = 1
    if sel[at]:
        at -= 2
    S[at, at + 2] = np.inf
    G = [M.copy(order="F") for M in (S, T)] + [np.asfortranarray(np.eye(n)) for _ in range(2)]
    ar, ai, be, m, pl, pr, info, ret = solver.tgsen(*G, sel, ijob=1)
    assert ret == 0 and info == 1
    assert m == int(sel.sum()) and pl == 0.0 and pr == 0.0
    S1, T1, Q, Z = G
    eye = np.eye(n)
    assert np.linalg.norm(Q.T @ Q - eye) <= 50 * n * EPS and np.linalg.norm(Z.T @ Z - eye) <= 50 * n * EPS
    assert np.linalg.norm(Q @ T1 @ Z.T - T) <= 50 * n * EPS * np.linalg.norm(T)
    assert not np.any(np.tril(T1, -1)) and not np.any(np.tril(S1, -2))
    # the blocks stay where they were; standardising them mixes the four
    # entries between them, nothing else
    bad = ~np.isfinite(S1)
    assert bad.any() and bad[at:at + 2, at + 2:at + 4].sum() == bad.sum()


@pytest.mark.parametrize("n", [40, 180])
def test_block_that_turns_real(solver, lapack, n):
    """Eigenvalues a +- 3e-9 i: rounding in a swap makes some pairs real."""
    S, T = _form(n, 5, (1.0, -1e-17))
    sel = np.zeros(n, dtype=np.int32)
    sel[2::4] = sel[3::4] = 1
    G = [M.copy(order="F") for M in (S, T)] + [np.asfortranarray(np.eye(n)) for _ in range(2)]
    ar, ai, be, m, pl, pr, info, ret = solver.tgsen(*G, sel, ijob=1)
    assert ret == 0 and info == 0 and m == int(sel.sum())
    r = lapack.residuals(S, T, *G)
    for key in ("h", "t", "q", "z"):
        assert r[key] <= 50 * r["neps"], (key, r[key] / r["neps"])
    assert lapack.schur_structure_ok(G[0], G[1])
    assert np.count_nonzero(np.diag(G[0], -1)) < n // 2  # (some did)
    # the selected ones lead: their values are near 8 (and 24) + U(-3, 3), the others near 0 (and 16)
    lam = ar / be
    want = np.sort(np.diag(S)[sel != 0])
    assert np.allclose(np.sort(lam[:m]), want, atol=1e-3)
    assert 0.0 < pl <= 1.0 and 0.0 < pr <= 1.0
