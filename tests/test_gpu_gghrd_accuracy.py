"""The Hessenberg-triangular reduction's factors are as orthogonal, and its
backward errors as small, as LAPACK DGGHRD's on the same pencil: the same
rotations in the same order, so the same number of roundings."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,seed", [(50, 0), (200, 1), (333, 2)])
def test_errors_against_dgghrd(pkg, lapack, n, seed):
    rng = np.random.default_rng(seed)
    A = rng.standard_normal((n, n))
    B = np.triu(rng.standard_normal((n, n)))
    B[np.arange(n), np.arange(n)] = np.sqrt(np.arange(n, 0, -1))
    ref = lapack.dgghrd(A, B)
    assert ref[4] == 0
    H, T = np.array(A, order="F"), np.array(B, order="F")
    Q, Z = np.zeros((n, n), order="F"), np.zeros((n, n), order="F")
    s = pkg.Solver(0)
    try:
        assert s.gghrd(H, T, Q, Z) == 0
    finally:
        s.close()

    def errors(H, T, Q, Z):
        eye = np.eye(n)
        return (np.linalg.norm(Q.T @ Q - eye), np.linalg.norm(Z.T @ Z - eye),
                np.linalg.norm(Q @ H @ Z.T - A) / np.linalg.norm(A), np.linalg.norm(Q @ T @ Z.T - B) / np.linalg.norm(B))

    for name, mine, theirs in zip("QZHT", errors(H, T, Q, Z), errors(*ref[:4])):
        assert mine <= theirs, (name, mine, theirs)
