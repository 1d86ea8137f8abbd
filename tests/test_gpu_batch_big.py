"""Batched pencils above the shared-memory window (order 80), each solved by
one CTA's windowed iteration: just above the window, around the tile and
window sizes of the updates (96, 128, 144), orders where the active block
splits, zeros on T's diagonal at the top, inside and at the bottom; and mixed
with pencils of the shared-memory kernel.  Backward error and orthogonality
within 50 n eps, Schur structure, eigenvalues against LAPACK."""
import numpy as np
import pytest

from test_gpu_batched import _check_pencil, _run_batch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes,zeros", [
    ([81, 82, 95, 96, 97, 112, 113], 0.0),
    ([127, 128, 129, 143, 144, 145, 161], 0.02),
    ([193, 80, 255, 12, 320], 0.01),
    ([100, 100, 160], 0.3),
])
def test_big_pencils(pkg, lapack, sizes, zeros):
    mats, b, hh, tt, qq, zz, ee, info = _run_batch(pkg, sizes, seed=31 + len(sizes), zero_frac=zeros)
    assert (info == 0).all(), info
    for p in range(b.count):
        n, e0 = int(b.n[p]), int(b.eoff[p])
        _check_pencil(lapack, mats[p][0], mats[p][1], b.unpack(hh, p), b.unpack(tt, p), b.unpack(qq, p),
                      b.unpack(zz, p), ee[e0:e0 + n], ee[b.neig + e0:b.neig + e0 + n],
                      ee[2 * b.neig + e0:2 * b.neig + e0 + n])


@pytest.mark.parametrize("where", [[0], [1], [99], [0, 50, 99], [40, 41, 42]])
def test_infinite_positions(pkg, lapack, where, monkeypatch):
    n = 100
    H, T = pkg.pencils.random_ht(n, 77, 0.0)
    for k in where:
        T[k, k] = 0.0
    monkeypatch.setattr(pkg.pencils, "random_ht", lambda *a: (H.copy(order="F"), T.copy(order="F")))
    mats, b, hh, tt, qq, zz, ee, info = _run_batch(pkg, [n], seed=1)
    assert info[0] == 0
    S, P = b.unpack(hh, 0), b.unpack(tt, 0)
    _check_pencil(lapack, H, T, S, P, b.unpack(qq, 0), b.unpack(zz, 0), ee[:n], ee[n:2 * n], ee[2 * n:])
    assert np.count_nonzero(ee[2 * n:] == 0.0) >= 1  # (zeros of T count as one rank lost or more)


def test_non_finite_is_reported(pkg):
    import torch
    n = 120
    H, T = pkg.pencils.random_ht(n, 5, 0.0)
    H[60, 60] = np.nan
    b = pkg.Batch([n])
    dev = torch.device("cuda:0")
    h, t = (torch.from_numpy(b.pack([M])).to(dev) for M in (H, T))
    q, z = torch.zeros_like(h), torch.zeros_like(h)
    e = torch.zeros(3 * n, dtype=torch.float64, device=dev)
    info = torch.zeros(1, dtype=torch.int32, device=dev)
    s = pkg.Solver(0)
    try:
        pkg.solve_batched_device(s, b, h.data_ptr(), t.data_ptr(), q.data_ptr(), z.data_ptr(), e.data_ptr(),
                                 e.data_ptr() + 8 * n, e.data_ptr() + 16 * n, info.data_ptr())
        torch.cuda.synchronize()
    finally:
        s.close()
    assert int(info[0]) != 0
