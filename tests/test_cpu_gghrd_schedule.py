"""The Hessenberg-triangular reduction's kernels, their device source run on the
host (tests/warp_emu.h, tests/emu_hessred.cpp) with the launch sequence of the
host code: against LAPACK DGGHRD, and the same bits whichever blocks of a
launch come first and whichever warps of a block are held back.  The blocks of
a launch take parts of the matrices that no other one of it touches, and the
row warps of a window wait for each other's rotations."""
import ctypes
import os
import re
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "..", "gevp-pdhgeqz_b200", "csrc")
_pd = ctypes.POINTER(ctypes.c_double)


def _source():
    """hessred.cu for the host."""
    with open(os.path.join(CSRC, "hessred.cu")) as f:
        text = f.read()
    text = re.sub(r'#include "(hessred\.cuh|kernels\.h|qz_roles\.cuh)"\n', "", text)
    text, k = re.subn(r'asm volatile\("cp\.async\.ca\.shared\.global.*?;\n', "*dst = *src;\n", text, flags=re.S)
    text, w = re.subn(r'asm volatile\("cp\.async\.wait_all;.*?;(?= })', "", text)
    assert (k, w) == (1, 1) and "asm" not in text
    text, k = re.subn(r"extern __shared__ __align__\(16\) double (\w+)\[\];", r"double* const \1 = emu_shared();", text)
    text, w = re.subn(r"__shared__ __align__\(16\) double (\w+)\[[^\n]*\];", r"double* const \1 = emu_shared();", text)
    assert k >= 1 and w >= 1 and "__shared__" not in text
    text, k = re.subn(r"(k_hr_\w+)<<<(.*?)>>>\((.*?)\);", r"emu_launch([&]() { \1(\3); }, \2);", text, flags=re.S)
    assert k >= 5 and "<<<" not in text
    return text


@pytest.fixture(scope="module")
def emu(tmp_path_factory):
    from test_cpu_role_schedule import _host_headers
    out = str(tmp_path_factory.mktemp("emuhr"))
    _host_headers(out)
    with open(os.path.join(out, "hessred_host.inc"), "w") as f:
        f.write(_source())
    with open(os.path.join(out, "cuda_runtime.h"), "w") as f:
        f.write("#pragma once\n")
    lib = os.path.join(out, "libemuhr.so")
    subprocess.run(["g++", "-O2", "-U_FORTIFY_SOURCE", "-ffp-contract=off", "-shared", "-fPIC", "-std=c++17", "-Wno-unknown-pragmas",
                    "-I", out, "-I", CSRC, "-I", HERE, os.path.join(HERE, "emu_hessred.cpp"), "-o", lib],
                   check=True, capture_output=True, timeout=300)
    L = ctypes.CDLL(lib)
    L.emu_gghrd.argtypes = [ctypes.c_int] * 3 + [_pd] * 4 + [ctypes.c_int] * 6 + [ctypes.c_uint]
    return L


def _run(L, A, B, W, ilo=0, ihi=None, qrows=0, sms=4, order=0, slow=0):
    n = A.shape[0]
    out = [A.copy(order="F"), B.copy(order="F"), np.zeros((n, n), order="F"), np.zeros((n, n), order="F")]
    rc = L.emu_gghrd(n, ilo, n - 1 if ihi is None else ihi, *(a.ctypes.data_as(_pd) for a in out), W, 2, 2, qrows,
                     sms, order, slow)
    assert rc == 0
    return out


def _pencil(n, seed):
    rng = np.random.default_rng(seed)
    return (np.asfortranarray(rng.standard_normal((n, n))),
            np.asfortranarray(np.triu(rng.standard_normal((n, n))) + 4.0 * np.eye(n)))


# orders and windows: one row warp, its last row, two and three warps of a
# window, a window's remainder, more helper blocks than items
@pytest.mark.parametrize("n,W,sms", [(3, 128, 4), (9, 4, 3), (20, 16, 4), (34, 128, 2), (37, 33, 9), (70, 66, 4)])
def test_any_order(emu, lapack, n, W, sms):
    A, B = _pencil(n, n)
    first = _run(emu, A, B, W, sms=sms)
    H0, T0, Q0, Z0, info = lapack.dgghrd(A, B)
    assert info == 0
    for M, M0 in zip(first, (H0, T0, Q0, Z0)):
        assert np.abs(M - M0).max() <= 1e-12 * n * np.abs(M0).max()
    orders = [(1, 0)] if n > 60 else [(1, 0), (0, 0x0001), (1, 0x003E), (0, 0xFFC0)]
    for order, slow in orders:
        out = _run(emu, A, B, W, sms=sms, order=order, slow=slow)
        for k, (a, b) in enumerate(zip(first, out)):
            assert np.array_equal(a.view(np.int64), b.view(np.int64)), (order, slow, k)


@pytest.mark.parametrize("ilo,ihi", [(0, 14), (5, 21), (4, 17), (6, 7)])
def test_inner_block_and_transposed_q(emu, lapack, ilo, ihi):
    n = 22
    A, B = _pencil(n, 3)
    for j in range(n):  # upper triangular outside the block
        A[max(j + 1, ihi + 1):, j] = 0.0
        if j < ilo:
            A[j + 1:, j] = 0.0
    A = np.asfortranarray(A)
    H, T, Q, Z = _run(emu, A, B, 8, ilo, ihi)
    assert np.abs(Q @ H @ Z.T - A).max() <= 1e-12 and np.abs(Q @ T @ Z.T - B).max() <= 1e-12
    assert not np.any(np.tril(H, -2)) and not np.any(np.tril(T, -1))
    Hq, Tq, Qq, Zq = _run(emu, A, B, 8, ilo, ihi, qrows=1)
    assert np.array_equal(H, Hq) and np.array_equal(T, Tq) and np.array_equal(Z, Zq)
    assert np.abs(Qq.T - Q).max() <= 1e-13
