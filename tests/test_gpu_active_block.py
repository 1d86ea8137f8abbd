"""A solve of rows ILO..IHI goes by the order of that block, not by the
matrix's: the block alone and inside a larger matrix takes the same number of
early deflations, sweeps and windows."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _counts(pkg, H, T, ilo, ihi):
    n = H.shape[0]
    s = pkg.Solver(0)
    try:
        out = [torch.from_numpy(M.T.copy()).cuda() for M in (H, T)]
        out += [torch.zeros(n, n, dtype=torch.float64, device="cuda") for _ in range(2)]
        e = torch.zeros(3, n, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        assert s.solve_device(*(x.data_ptr() for x in out), n, n, *(v.data_ptr() for v in e), ilo=ilo, ihi=ihi) == 0
        st = s.stats()
    finally:
        s.close()
    return [st[k] for k in ("aeds", "aed_deflations", "sweeps", "windows", "shifts")], e[:, ilo - 1:ihi].cpu()


@pytest.mark.parametrize("m,n", [(300, 1000), (700, 760), (760, 1100)])
def test_block_alone_and_inside(pkg, m, n):
    H0, T0 = pkg.pencils.random_ht(m, 5, 0.0)
    rng = np.random.default_rng(1)
    H, T = (np.asfortranarray(np.triu(rng.standard_normal((n, n)))) for _ in range(2))
    lo = (n - m) // 2
    H[lo:lo + m, lo:lo + m], T[lo:lo + m, lo:lo + m] = H0, T0
    alone, e0 = _counts(pkg, H0, T0, 1, m)
    inside, e1 = _counts(pkg, H, T, lo + 1, lo + m)
    assert inside == alone
    assert torch.equal(e0, e1)
