"""The learned policy's idea of the fixed table is the solver's: the AED window
by order, also in what traces record and compare with."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def tables(tmp_path_factory):
    lib = str(tmp_path_factory.mktemp("tables") / "libtables.so")
    subprocess.run(["g++", "-O1", "-shared", "-fPIC", "-std=c++17", "-Wno-unknown-pragmas", "-I",
                    os.path.join(HERE, "..", "gevp-pdhgeqz_b200", "csrc"), os.path.join(HERE, "solver_tables.cpp"),
                    "-o", lib], check=True, capture_output=True, timeout=300)
    return ctypes.CDLL(lib)


def test_window_and_shifts_are_the_solvers(pkg, tables):
    lrn = pkg.learned
    for n in list(range(30, 700, 7)) + [599, 600, 1199, 1200, 2999, 3000, 5000, 6000, 9000]:
        assert lrn.table_window(n) == tables.table_window(n), n
        if n < 6000:
            nw, nsf = lrn.table_choice(n, lrn.table_window(n))
            assert nw == min(n, tables.table_window(n))
            assert nsf == min(1.0, tables.table_shifts(n) / nw), n


class _Solver:
    """Records the tunables a trace sets; no decision point is ever reached."""

    def __init__(self):
        self.set = {"nw_max": 0, "ns_max": 0, "aed_limit": -1}

    def set_param(self, name, value):
        self.set[name] = value

    def solve_device(self, *a, **k):
        return 0

    def stats(self):
        return {"stop_ktop": 0, "stop_kbot": 0, "remaining": 0, "last_aed_fraction": 0.0, "seconds": 0.0}


def test_trace_leaves_the_defaults(pkg, monkeypatch):
    import torch
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 0)
    monkeypatch.setattr(torch, "device", lambda *a: "cpu")
    s = _Solver()
    assert pkg.learned.trace_pencil(s, np.eye(4), np.eye(4)) == []
    assert s.set == {"nw_max": 0, "ns_max": 0, "aed_limit": -1}


def test_gain_with_a_window_per_sample(pkg):
    """One window for all samples, and the same one given per sample."""
    lrn = pkg.learned
    rng = np.random.default_rng(2)
    k = 9
    X = rng.random((k, lrn.NIN)).astype(np.float32)
    scores = rng.random((k, len(lrn.GRID_NW), len(lrn.GRID_NSF))) + 0.5
    nh = rng.integers(300, 8000, k)
    P = lrn.init_params(4)
    one = lrn.offline_gain(P, X, scores, nh, (lrn.GRID_NW, lrn.GRID_NSF, 56))
    each = lrn.offline_gain(P, X, scores, nh, (lrn.GRID_NW, lrn.GRID_NSF, np.full(k, 56)))
    assert one == each
    tr = {"grid_nw": np.array(lrn.GRID_NW), "grid_nsf": np.array(lrn.GRID_NSF), "table_nw": np.full(k, 48)}
    assert np.array_equal(lrn.trace_grid(tr)[2], np.full(k, 48))
