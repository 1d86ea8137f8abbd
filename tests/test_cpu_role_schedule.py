"""The window QZ, the early deflation and the chase with a role per warp, their
device source run on the host as a thread block of fibers (tests/warp_emu.h),
with the order of the warps chosen by the test.  What a warp reads before another has written it shows as a
result that depends on that order: every order has to give the same bits."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from conftest import EPS
from test_cpu_host_algorithms import _check

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "..", "gevp-pdhgeqz_b200", "csrc")
_pd = ctypes.POINTER(ctypes.c_double)
RIGHT, Q, Z = 0x06, 0x28, 0xC0  # warps of the right transformations, of Q and of Z


def _host_headers(out):
    """qz_roles.cuh and qz_chase_roles.cuh for the host: without their PTX, the
    polls after which a wait gives up a variable."""
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
    with open(os.path.join(CSRC, "qz_chase_roles.cuh")) as f:
        text = f.read()
    bar = [line for line in text.splitlines() if "asm" in line]
    assert len(bar) == 1 and "void chase_bar()" in bar[0]
    text = text.replace(bar[0], "").replace("#ifdef __CUDACC__", "#if 1").replace("qz_roles.cuh", "roles_host.inc")
    with open(os.path.join(out, "chase_host.inc"), "w") as f:
        f.write(text)


def _build(out):
    _host_headers(out)
    lib = os.path.join(out, "libemu.so")
    subprocess.run(["g++", "-O2", "-U_FORTIFY_SOURCE", "-ffp-contract=off", "-shared", "-fPIC", "-std=c++17", "-Wno-unknown-pragmas",
                    "-I", out, "-I", CSRC, "-I", HERE, os.path.join(HERE, "emu_roles.cpp"), "-o", lib],
                   check=True, capture_output=True, timeout=300)
    L = ctypes.CDLL(lib)
    L.emu_role_qz.argtypes = [ctypes.c_int] + [_pd] * 4 + [ctypes.c_uint, ctypes.c_int]
    L.emu_aed.argtypes = [ctypes.c_int] + [_pd] * 4 + [ctypes.c_double, ctypes.c_int, _pd, ctypes.POINTER(ctypes.c_int),
                                                       ctypes.c_uint]
    L.emu_aed.restype = None
    L.emu_chase.argtypes = [ctypes.c_int] + [_pd] * 4 + [_pd, ctypes.c_int, ctypes.c_uint]
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
                                         (34, "split", 5), (34, "dense", 6), (66, "split", 7)])
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
        for spin in range(1, 40, 2):
            rc, out = _run(emu, H, T, slow, spin)
            gave_up += rc != 0
            assert rc != 0 or all(np.array_equal(a.view(np.int64), b.view(np.int64)) for a, b in zip(good, out)), \
                (slow, spin)
    assert gave_up > 0


def _same(a, b):
    return all(np.array_equal(x.view(np.int64), y.view(np.int64)) for x, y in zip(a, b))


@pytest.mark.parametrize("nskip", [0, 4])
def test_early_deflation_in_any_order(emu, nskip):
    """Window of 20 with a spike that deflates some blocks: swaps of several
    moves at once, then the re-reduction, whose column rotations go from warp
    0 to the others."""
    n, s = 20, 1e-9
    H, T = _pencil(n, "dense", 17)
    first = None
    for slow in (0, 0x01, 0xFE, 0x0F, 0xAA):
        out = [H.copy(order="F"), T.copy(order="F"), np.zeros((n, n), order="F"), np.zeros((n, n), order="F"),
               np.zeros(3 * n)]
        info = (ctypes.c_int * 3)()
        emu.emu_aed(n, *(a.ctypes.data_as(_pd) for a in out[:4]), s, nskip, out[4].ctypes.data_as(_pd), info, slow)
        assert info[1] == 0 and 2 < info[0] < n and info[2] == 1, list(info)
        m = info[0]
        if first is None:
            first = out
            S, P, Q, Z = out[:4]
            for A, B in ((H, S), (T, P)):
                assert np.linalg.norm(Q @ B @ Z.T - A) <= 50 * n * EPS * np.linalg.norm(A)
            assert not np.any(np.tril(S[:m, :m], -2)) and not np.any(np.tril(P, -1))
        assert _same(first, out), slow


@pytest.mark.parametrize("n,nb", [(12, 1), (30, 4), (38, 9)])
def test_chase_in_any_order(emu, n, nb):
    """The coefficient warp, the chase warps or the factor warps (behind the
    ring, and up to its length behind) held back; more bulges than warps."""
    H, T = _pencil(n, "dense", n)
    rng = np.random.default_rng(n)
    coef = np.concatenate([[1.0, 2 * a, a * a + 0.3] for a in rng.standard_normal(nb)])
    first = None
    chase = sum(1 << w for w in range(16) if w % 4 in (1, 2))
    factor = sum(1 << w for w in range(16) if w % 4 == 3)
    for slow in (0, 0x0001, chase, factor, factor | 0x0006):
        out = [H.copy(order="F"), T.copy(order="F"), np.zeros((n, n), order="F"), np.zeros((n, n), order="F")]
        assert emu.emu_chase(n, *(a.ctypes.data_as(_pd) for a in out), coef.ctypes.data_as(_pd), nb, slow) == 0
        if first is None:
            first = out
            S, P, U, V = out
            for A, B in ((H, S), (T, P)):
                assert np.linalg.norm(U @ B @ V.T - A) <= 50 * n * EPS * np.linalg.norm(A)
            assert not np.any(np.tril(S, -2)) and not np.any(np.tril(P, -1))
        assert _same(first, out), slow
