"""The one-CTA solve of a batched pencil above order 80, its device source run
on the host as a block of fibers (tests/warp_emu.h): early deflations by half
of the warps, chases by another split, updates by two groups of eight warps.
Shared memory begins as NaN; whichever warps are held back, the same bits."""
import ctypes
import os
import re
import subprocess

import numpy as np
import pytest

from test_cpu_host_algorithms import _check
from test_cpu_role_schedule import CSRC, HERE, _host_headers, _pd, _pencil, _same


@pytest.fixture(scope="module")
def emu(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("emubig"))
    _host_headers(out)
    with open(os.path.join(CSRC, "batch_big.cuh")) as f:
        text = f.read()
    text, a = re.subn(r'asm volatile\("bar\.sync 2, %0;".*?;(?= })', "emu::named_barrier(2, kRoleThreads);", text)
    text, b = re.subn(r'asm volatile\("bar\.sync %0, 256;".*?;(?= })', "emu::named_barrier(3 + grp, 256);", text)
    text, c = re.subn(r"extern __shared__ double smem\[\];", "double* const smem = (double*)emu::block()->arena;", text)
    assert (a, b, c) == (1, 1, 2) and "asm" not in text
    text = text.replace("#ifdef __CUDACC__", "#if 1").replace("qz_chase_roles.cuh", "chase_host.inc")
    with open(os.path.join(out, "batch_big_host.inc"), "w") as f:
        f.write(text)
    lib = os.path.join(out, "libemubig.so")
    subprocess.run(["g++", "-O2", "-U_FORTIFY_SOURCE", "-ffp-contract=off", "-shared", "-fPIC", "-std=c++17", "-Wno-unknown-pragmas",
                    "-I", out, "-I", CSRC, "-I", HERE, os.path.join(HERE, "emu_batch_big.cpp"), "-o", lib],
                   check=True, capture_output=True, timeout=300)
    L = ctypes.CDLL(lib)
    L.emu_big.argtypes = [ctypes.c_int] + [_pd] * 4 + [ctypes.c_uint]
    return L


@pytest.mark.parametrize("n,kind,seed,orders", [(84, "split", 1, (0x00FF, 0xFF00, 0x5555)),
                                                (86, "dense", 2, (0x0006, 0xFF00)), (90, "zero_t", 3, (0x8888,))])
def test_any_order_of_the_warps(emu, lapack, n, kind, seed, orders):
    H, T = _pencil(n, kind, seed)
    first = None
    for slow in (0,) + orders:
        out = [H.copy(order="F"), T.copy(order="F"), np.zeros((n, n), order="F"), np.zeros((n, n), order="F")]
        assert emu.emu_big(n, *(a.ctypes.data_as(_pd) for a in out), slow) == 0
        if first is None:
            first = out
            _check(lapack, H, T, *out)
        assert _same(first, out), hex(slow)
