"""Batched pencils at the orders where the one-CTA solve's tables change: the
early deflation window (600, 1200), the shifts of a sweep and its chains (590),
the spike test (750), each side, and with zeros on T's diagonal.  Backward
error and orthogonality within 50 n eps, Schur structure, eigenvalues against
LAPACK; on the largest, where LAPACK takes minutes, against the single solve."""
import numpy as np
import pytest

from test_gpu_batched import _check_pencil, _run_batch

pytestmark = pytest.mark.gpu


def _parts(b, p, hh, tt, qq, zz, ee):
    n, e0 = int(b.n[p]), int(b.eoff[p])
    return ([b.unpack(x, p) for x in (hh, tt, qq, zz)],
            [ee[k * b.neig + e0:k * b.neig + e0 + n] for k in range(3)])


@pytest.mark.parametrize("sizes,zeros", [([589, 591], 0.0), ([599, 600], 0.0), ([650], 0.02), ([749, 751], 0.0)])
def test_orders(pkg, lapack, sizes, zeros):
    mats, b, hh, tt, qq, zz, ee, info = _run_batch(pkg, sizes, seed=57 + sizes[0], zero_frac=zeros)
    assert (info == 0).all(), info
    for p in range(b.count):
        factors, eig = _parts(b, p, hh, tt, qq, zz, ee)
        _check_pencil(lapack, *mats[p], *factors, *eig)


def test_largest_window(pkg, lapack):
    n = 1201
    mats, b, hh, tt, qq, zz, ee, info = _run_batch(pkg, [n], seed=60, zero_frac=0.0)
    assert info[0] == 0
    H, T = mats[0]
    (S, P, Q, Z), (ar, ai, be) = _parts(b, 0, hh, tt, qq, zz, ee)
    r = lapack.residuals(H, T, S, P, Q, Z)
    for key in ("h", "t", "q", "z"):
        assert r[key] <= 50 * r["neps"], (key, r[key] / r["neps"])
    assert lapack.schur_structure_ok(S, P)
    S1, P1, Q1, Z1, ar1, ai1, be1, info1 = pkg.solve(H, T)
    assert info1 == 0
    ok, ratio, _ = lapack.match_eigenvalues((ar1, ai1, be1), (ar, ai, be), lapack.eig_tolerance(S1, P1, H, T))
    assert ok, ratio
