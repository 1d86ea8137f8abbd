"""The window QZ with a role per warp, its device source run on the host as a
thread block of fibers (tests/warp_emu.h), with the order of the warps chosen
by the test.  What a warp reads before another has written it shows as a
result that depends on that order: every order has to give the same bits."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from test_cpu_host_algorithms import _check

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "..", "gevp-pdhgeqz_b200", "csrc")
_pd = ctypes.POINTER(ctypes.c_double)
RIGHT, Q, Z = 0x06, 0x28, 0xC0  # warps of the right transformations, of Q and of Z


def _build(out):
    """Host build of qz_roles.cuh without its PTX; the polls after which a wait
    gives up are a variable."""
    with open(os.path.join(CSRC, "qz_roles.cuh")) as f:
        text = f.read()
    a = text.index("__device__ __forceinline__ int role_ld")
    b = text.index("// Sums of squares outside")
    assert "asm" not in text[:a].split("#ifdef __CUDACC__")[1] and "asm" not in text[b:]
    text = (text[:a] + text[b:]).replace("#ifdef __CUDACC__", "#if 1")
    assert "constexpr int kRoleSpin" in text
    text = text.replace("constexpr int kRoleSpin", "inline int kRoleSpin")
    with open(os.path.join(out, "roles_host.inc"), "w") as f:
        f.write(text)
    lib = os.path.join(out, "libemu.so")
    subprocess.run(["g++", "-O2", "-ffp-contract=off", "-shared", "-fPIC", "-std=c++17", "-Wno-unknown-pragmas",
                    "-I", out, "-I", CSRC, "-I", HERE, os.path.join(HERE, "emu_roles.cpp"), "-o", lib],
                   check=True, capture_output=True, timeout=300)
    L = ctypes.CDLL(lib)
    L.emu_role_qz.argtypes = [ctypes.c_int] + [_pd] * 4 + [ctypes.c_uint, ctypes.c_int]
    return L


@pytest.fixture(scope="module")
def emu(tmp_path_factory):
    return _build(str(tmp_path_factory.mktemp("emu")))


def _pencil(n, kind, seed):
    rng = np.random.default_rng(seed)
    H = np.triu(rng.standard_normal((n, n)), -1)
    T = np.triu(rng.standard_normal((n, n)))
    T[np.arange(n), np.arange(n)] = np.sqrt(np.arange(n, 0, -1)) + 0.1
    if kind == "zero_t":
        k = rng.choice(n, max(1, n // 8), replace=False)
        T[k, k] = 0.0
    elif kind == "split":
        k = np.arange(3, n, 5)
        H[k, k - 1] = 0.0
    return np.asfortranarray(H), np.asfortranarray(T)


def _run(L, H, T, slow, spin=1 << 22):
    n = H.shape[0]
    out = [H.copy(order="F"), T.copy(order="F"), np.zeros((n, n), order="F"), np.zeros((n, n), order="F")]
    rc = L.emu_role_qz(n, *(a.ctypes.data_as(_pd) for a in out), slow, spin)
    return rc, out


@pytest.mark.parametrize("n,kind,seed", [(9, "dense", 1), (20, "dense", 2), (20, "split", 3), (24, "zero_t", 4),
                                         (34, "dense", 5)])
def test_any_order_of_the_warps(emu, lapack, n, kind, seed):
    H, T = _pencil(n, kind, seed)
    rc, first = _run(emu, H, T, 0)
    assert rc == 0
    _check(lapack, H, T, *first)
    for slow in (RIGHT, RIGHT | Q | Z):
        rc, out = _run(emu, H, T, slow)
        assert rc == 0, slow
        for k, (a, b) in enumerate(zip(first, out)):
            assert np.array_equal(a.view(np.int64), b.view(np.int64)), (slow, k, np.abs(a - b).max())


def test_wait_orders_every_lane(emu):
    """Only some lanes poll the counts that a wait is for, but all of them read
    what the counts stand for: each lane has to be ordered behind the polls."""
    assert emu.emu_wait_done(7) == 32


def test_a_wait_that_gives_up_is_reported(emu):
    """Waits limited to a few polls, with the core and some followers held
    back, so that other followers give up at every point of the solve, after
    its last step among them: either the result is right or the status says
    that it is not."""
    H, T = _pencil(6, "dense", 8)
    rc, good = _run(emu, H, T, 0)
    assert rc == 0
    gave_up = 0
    for slow in (0x01, 0x01 | RIGHT, 0x01 | RIGHT | Q, 0x01 | Q | Z):
        for spin in range(1, 60):
            rc, out = _run(emu, H, T, slow, spin)
            gave_up += rc != 0
            assert rc != 0 or all(np.array_equal(a.view(np.int64), b.view(np.int64)) for a, b in zip(good, out)), \
                (slow, spin)
    assert gave_up > 0
