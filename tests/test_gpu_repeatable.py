"""A solve repeats itself bit for bit.  The window QZ overlaps its warps
through flags in shared memory; what a warp reads before another has written
it shows as two runs of one input that differ.  Windows with many deflations
(each moves the end of the active block, and with it the entries the next
shift is formed from), whole solves and batches, each several times: every
output equal in every bit."""
import ctypes

import pytest
import torch

from test_gpu_role_window import _pencil

pytestmark = pytest.mark.gpu

RUNS = 12


@pytest.fixture(scope="module")
def solver(pkg):
    s = pkg.Solver(0)
    yield s
    s.close()


def _same(a, b):
    """Equal bits (NaN equals itself)."""
    return torch.equal(a.contiguous().view(torch.int64), b.contiguous().view(torch.int64))


def _window(pkg, solver, H, T):
    n = H.shape[0]
    out = [torch.from_numpy(M.T.copy()).cuda() for M in (H, T)]
    out += [torch.zeros(n, n, dtype=torch.float64, device="cuda") for _ in range(2)]
    out.append(torch.zeros(3 * n, dtype=torch.float64, device="cuda"))
    torch.cuda.synchronize()
    info = (ctypes.c_int * 3)()
    rc = pkg.lib().b200qz_aed_window(solver.handle, out[0].data_ptr(), out[1].data_ptr(), n, 0, 0, n - 1,
                                     out[2].data_ptr(), out[3].data_ptr(), out[4].data_ptr(), info)
    assert rc == 0 and info[1] == 0, (rc, list(info))
    return out, list(info)


@pytest.mark.parametrize("n", [33, 48, 56, 65, 80])
@pytest.mark.parametrize("kind", ["dense", "zero_t", "split", "graded"])
def test_window(pkg, solver, n, kind):
    H, T = _pencil(n, kind, 11 * n + len(kind))
    first, info = _window(pkg, solver, H, T)
    for run in range(RUNS):
        again, info2 = _window(pkg, solver, H, T)
        assert info2 == info, run
        for k, (a, b) in enumerate(zip(first, again)):
            assert _same(a, b), (run, k)


def _solve(solver, H, T):
    n = H.shape[0]
    out = [torch.from_numpy(M.T.copy()).cuda() for M in (H, T)]
    out += [torch.zeros(n, n, dtype=torch.float64, device="cuda") for _ in range(2)]
    e = torch.zeros(3, n, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    rc = solver.solve_device(*(x.data_ptr() for x in out), n, n, e[0].data_ptr(), e[1].data_ptr(), e[2].data_ptr())
    assert rc == 0
    return out + [e]


@pytest.mark.parametrize("n,zeros", [(70, 0.0), (201, 0.0), (300, 0.05), (950, 0.0)])
def test_solve(pkg, solver, n, zeros):
    H, T = pkg.pencils.random_ht(n, 40 + n, zeros)
    first = _solve(solver, H, T)
    for run in range(3):
        for k, (a, b) in enumerate(zip(first, _solve(solver, H, T))):
            assert _same(a, b), (run, k)


def test_batch(pkg, solver):
    sizes = [80, 79, 66, 65, 64, 49, 48, 33, 32, 17, 5, 2, 150, 120, 97, 81] * 4
    b = pkg.Batch(sizes)
    mats = [pkg.pencils.random_ht(n, 900 + i, 0.03) for i, n in enumerate(sizes)]
    h0, t0 = (torch.from_numpy(b.pack([m[k] for m in mats])).cuda() for k in (0, 1))
    ref = None
    for run in range(4):
        h, t = h0.clone(), t0.clone()
        q, z = torch.zeros_like(h), torch.zeros_like(h)
        e = torch.zeros(3 * b.neig, dtype=torch.float64, device="cuda")
        info = torch.zeros(b.count, dtype=torch.int32, device="cuda")
        torch.cuda.synchronize()
        pkg.solve_batched_device(solver, b, *(x.data_ptr() for x in (h, t, q, z)), e.data_ptr(),
                                 e.data_ptr() + 8 * b.neig, e.data_ptr() + 16 * b.neig, info.data_ptr())
        torch.cuda.synchronize()
        assert not info.any()
        if ref is None:
            ref = [h, t, q, z, e]
        for k, (x, y) in enumerate(zip(ref, [h, t, q, z, e])):
            assert _same(x, y), (run, k)
