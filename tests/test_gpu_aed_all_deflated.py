"""An early deflation that deflates its whole window.  The window's first row
is then a converged block, and the entry H(kwtop, kwtop-1) that joined it to
the rest, negligible by the spike test but not by the scan's test of its two
neighbours, has to be zero: left as it is, the output would hold a 2x2 block
that is none.  For the window entry, a single solve and the batch's one-CTA
solve."""
import ctypes

import numpy as np
import pytest
import torch

from test_gpu_batched import _check_pencil

pytestmark = pytest.mark.gpu

NW = 24  # the early deflation window of these orders


def _pencil(n, seed):
    """The entry left of the trailing window's first row is far below the
    window's eigenvalues and above eps times its diagonal neighbours."""
    rng = np.random.default_rng(seed)
    H = np.triu(rng.standard_normal((n, n)), -1)
    T = np.triu(rng.standard_normal((n, n)))
    k = np.arange(n)
    T[k, k] = np.sqrt(np.arange(n, 0, -1)) + 0.5
    w = n - NW
    H[w, w] = H[w - 1, w - 1] = 1e-6
    H[w, w - 1] = 1e-20
    return np.asfortranarray(H), np.asfortranarray(T), w


def test_window(pkg):
    H, T, w = _pencil(100, 3)
    n = H.shape[0]
    s = pkg.Solver(0)
    try:
        h, t = (torch.from_numpy(M.T.copy()).cuda() for M in (H, T))
        q, z = (torch.zeros(NW, NW, dtype=torch.float64, device="cuda") for _ in range(2))
        sh = torch.zeros(3 * NW, dtype=torch.float64, device="cuda")
        info = (ctypes.c_int * 3)()
        torch.cuda.synchronize()
        rc = pkg.lib().b200qz_aed_window(s.handle, h.data_ptr(), t.data_ptr(), n, 0, w, n - 1, q.data_ptr(),
                                         z.data_ptr(), sh.data_ptr(), info)
    finally:
        s.close()
    assert rc == 0 and list(info) == [0, 0, 1]  # nothing left undeflated
    assert h[w - 1, w].item() == 0.0


@pytest.mark.parametrize("n", [100, 200])
def test_solve(pkg, lapack, n):
    H, T, w = _pencil(n, 7)
    S, P, Q, Z, ar, ai, be, info = pkg.solve(H, T)
    assert info == 0
    assert S[w, w - 1] == 0.0
    _check_pencil(lapack, H, T, S, P, Q, Z, ar, ai, be)


def test_batch(pkg, lapack, monkeypatch):
    from test_gpu_batched import _run_batch
    H, T, w = _pencil(100, 7)
    monkeypatch.setattr(pkg.pencils, "random_ht", lambda *a: (H.copy(order="F"), T.copy(order="F")))
    mats, b, hh, tt, qq, zz, ee, info = _run_batch(pkg, [100], seed=1)
    assert info[0] == 0
    n, S = 100, b.unpack(hh, 0)
    assert S[w, w - 1] == 0.0
    _check_pencil(lapack, H, T, S, b.unpack(tt, 0), b.unpack(qq, 0), b.unpack(zz, 0), ee[:n], ee[n:2 * n], ee[2 * n:])
