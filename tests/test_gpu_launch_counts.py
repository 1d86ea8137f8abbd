"""Kernel launches that a reduction and a reordering report, which the bench
lines state: counted against what the call consists of."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def solver(pkg):
    s = pkg.Solver(0)
    yield s
    s.close()


@pytest.mark.parametrize("n,win", [(2, 128), (3, 128), (40, 128), (150, 128), (150, 32)])
def test_reduction(solver, n, win):
    """Q and Z set, B's lower part cleared, a launch per window and two per
    column, the last column's factors on Q and Z."""
    rng = np.random.default_rng(n)
    A, B = np.asfortranarray(rng.standard_normal((n, n))), np.asfortranarray(np.triu(rng.standard_normal((n, n))))
    Q, Z = np.zeros((n, n), order="F"), np.zeros((n, n), order="F")
    solver.set_param("hr_win", win)
    try:
        assert solver.gghrd(A, B, Q, Z) == 0
    finally:
        solver.set_param("hr_win", 128)
    windows = sum(-(-(n - 2 - jc) // win) for jc in range(n - 2))
    assert solver.stats()["launches"] == 3 + windows + 2 * (n - 2) + (1 if n > 2 else 0)


def test_reordering(solver, lapack, pkg):
    """Signs and eigenvalues; with one window over the whole form also its
    launch, the status after it and the update of Q and Z."""
    n = 30
    H, T = pkg.pencils.random_ht(n, 4, 0.0)
    S, P, ar, ai, be, Q, Z, info = lapack.dhgeqz(H, T)
    assert info == 0
    for select, launches in ((np.zeros(n), 2), (np.ones(n), 2), (np.arange(n) >= n // 2, 5)):
        G = [np.array(M, order="F", copy=True) for M in (S, P, Q, Z)]
        *_, info, ret = solver.tgsen(*G, np.asarray(select, dtype=np.int32))
        assert ret == 0 and info == 0
        assert solver.stats()["launches"] == launches
