"""A tunable that was changed can be set back: with every tunable set to another
value and then to its default, by name or by b200qz_set_params, a solve takes
the same path as in a fresh context (the same counts) and gives the same
bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu

# name: (another value, the default)
TUNABLES = {
    "nw_max": (40, 0), "w_chase": (48, 64), "nmin": (64, 80), "ns_max": (20, 0), "maxit_factor": (20, 30),
    "aed_nskip": (2, -1), "max_wave": (2, 8), "stall_limit": (100, 300), "aed_limit": (0, -1),
    "upd_persist": (0, 1), "split": (8, 0), "aed_threads": (128, 256), "aed_swap_fail": (1, 0), "aed_ms": (1, 0),
}


def _solve(pkg, H, T, setup):
    n = H.shape[0]
    s = pkg.Solver(0)
    try:
        setup(s)
        out = [torch.from_numpy(M.T.copy()).cuda() for M in (H, T)]
        out += [torch.zeros(n, n, dtype=torch.float64, device="cuda") for _ in range(2)]
        e = torch.zeros(3, n, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        assert s.solve_device(*(x.data_ptr() for x in out), n, n, *(v.data_ptr() for v in e)) == 0
        st = s.stats()
    finally:
        s.close()
    return out + [e], {k: st[k] for k in ("aeds", "sweeps", "windows", "launches", "chains", "shifts")}


def _by_name(names):
    def setup(s):
        for k in names:
            s.set_param(k, TUNABLES[k][0])
        for k in names:
            s.set_param(k, TUNABLES[k][1])
    return setup


def _by_params(s):
    s.set_params(nw_max=40, w_chase=48, nmin=64, ns_max=20, maxit_factor=20)
    s.set_params(nw_max=0, w_chase=64, nmin=80, ns_max=0, maxit_factor=30)


@pytest.fixture(scope="module")
def fresh(pkg):
    """A pencil whose sweeps have more than eight bulges to place."""
    H, T = pkg.pencils.random_ht(950, 12, 0.0)
    out, counts = _solve(pkg, H, T, lambda s: None)
    assert 2 * counts["sweeps"] <= counts["chains"]  # a sweep has two chains
    return H, T, out, counts


@pytest.mark.parametrize("name", list(TUNABLES) + ["all"])
def test_set_back_by_name(pkg, fresh, name):
    H, T, want, counts = fresh
    out, got = _solve(pkg, H, T, _by_name(list(TUNABLES) if name == "all" else [name]))
    assert got == counts
    assert all(torch.equal(a, b) for a, b in zip(want, out))


def test_set_back_by_params(pkg, fresh):
    H, T, want, counts = fresh
    out, got = _solve(pkg, H, T, _by_params)
    assert got == counts
    assert all(torch.equal(a, b) for a, b in zip(want, out))


def test_out_of_range_stays_refused(pkg):
    s = pkg.Solver(0)
    try:
        for name, v in (("nw_max", 3), ("nw_max", -1), ("nw_max", 81), ("w_chase", 11), ("w_chase", 81)):
            with pytest.raises(ValueError):
                s.set_param(name, v)
        with pytest.raises(ValueError):
            s.set_params(nw_max=81)
    finally:
        s.close()


def test_trace_leaves_the_solver_as_it_was(pkg, fresh):
    H, T, want, counts = fresh

    def trace(s):
        Ht, Tt = pkg.pencils.clustered_ht(300, 5)
        assert len(pkg.learned.trace_pencil(s, Ht, Tt, decisions=(0,), horizon=1)) == 1

    out, got = _solve(pkg, H, T, trace)
    assert got == counts
    assert all(torch.equal(a, b) for a, b in zip(want, out))
