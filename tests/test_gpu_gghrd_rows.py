"""The Hessenberg-triangular reduction where its split changes: orders at the
edges of the row warps (32 rows), of a window (hr_win pairs) and of one walk's
groups (16 entries) and stages (64 rotations); zeros in the column of A and on
B's diagonal (exact rotations) and entries outside the range of plain squares
(rotations one after another).  Against LAPACK DGGHRD: the same rotations in
the same order and sign convention, entrywise to rounding."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def solver(pkg):
    s = pkg.Solver(0)
    yield s
    s.close()


def _compare(solver, lapack, A, B, win, scale=1.0):
    n = A.shape[0]
    H0, T0, Q0, Z0, info = lapack.dgghrd(A, B)
    assert info == 0
    H, T = np.array(A, order="F"), np.array(B, order="F")
    Q, Z = np.zeros((n, n), order="F"), np.zeros((n, n), order="F")
    solver.set_param("hr_win", win)
    try:
        assert solver.gghrd(H, T, Q, Z) == 0
    finally:
        solver.set_param("hr_win", 128)
    assert not np.any(np.tril(H, -2)) and not np.any(np.tril(T, -1))
    tol = 1e-12 * n
    assert np.abs(H - H0).max() <= tol * np.abs(H0).max()
    assert np.abs(T - T0).max() <= tol * np.abs(T0).max()
    assert np.abs(Q - Q0).max() <= tol and np.abs(Z - Z0).max() <= tol


def _pencil(n, seed):
    rng = np.random.default_rng(seed)
    return rng.standard_normal((n, n)), np.triu(rng.standard_normal((n, n))) + 4.0 * np.eye(n)


@pytest.mark.parametrize("n,win", [(4, 128), (18, 16), (19, 17), (34, 128), (35, 33), (66, 64), (67, 65), (98, 32),
                                   (99, 31), (130, 128), (131, 129), (163, 160), (260, 160)])
def test_row_splits(solver, lapack, n, win):
    A, B = _pencil(n, n)
    _compare(solver, lapack, A, B, win)


@pytest.mark.parametrize("n", [40, 140])
def test_exact_zeros(solver, lapack, n):
    A, B = _pencil(n, 7 * n)
    A[n // 2:, 0] = 0.0          # identities below a column's middle
    A[n // 3, :2] = 0.0          # a swap of rows
    B[n // 4, n // 4] = 0.0      # no fill: an identity of columns
    B[n - 1, n - 1] = 0.0
    _compare(solver, lapack, A, B, 128)


@pytest.mark.parametrize("scale", [1e-200, 1e200])
def test_out_of_range_squares(solver, lapack, scale):
    n = 70
    A, B = _pencil(n, 3)
    _compare(solver, lapack, A * scale, B, 128)
    _compare(solver, lapack, A, B * scale, 128)
