"""role_rsqrt and role_rcp, from which the window kernels form their rotations
and reflectors, against 80-bit arithmetic over the range they are used in.

Bounds, in units of rounding u = 2^-53.  The hardware's approximations are
good to 2^-20, so e = 1 - x y^2 (or 1 - x y) is at most about 2^-19.
role_rsqrt: the rounding of x y enters e as u and the result as u / 2, the
last operation rounds to u, and the series stops at 5/16 e^3 < 0.03 u: 1.6 u
with room for the products' own roundings (u e).  role_rcp: after one Newton
step e is below 2^-38, the second one's e is exact to u e, and the last
operation rounds to u: 1.01 u."""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
U = 2.0 ** -53


@pytest.fixture(scope="module")
def math(tmp_path_factory):
    lib = str(tmp_path_factory.mktemp("math") / "librolemath.so")
    nvcc = "/usr/local/cuda/bin/nvcc" if os.path.exists("/usr/local/cuda/bin/nvcc") else shutil.which("nvcc")
    subprocess.run([nvcc, "-shared", "-Xcompiler", "-fPIC", "-std=c++17", "-O3", "--expt-relaxed-constexpr",
                    "-gencode", "arch=compute_100a,code=sm_100a", "-I",
                    os.path.join(HERE, "..", "gevp-pdhgeqz_b200", "csrc"), "-o", lib,
                    os.path.join(HERE, "role_math.cu")], check=True, capture_output=True, timeout=300)
    return ctypes.CDLL(lib)


def _run(math, x):
    import torch
    d = torch.from_numpy(x).cuda()
    root, inv = torch.zeros_like(d), torch.zeros_like(d)
    torch.cuda.synchronize()
    assert math.role_math(*(ctypes.c_void_p(t.data_ptr()) for t in (d, root, inv)), x.size) == 0
    return root.cpu().numpy(), inv.cpu().numpy()


@pytest.mark.parametrize("lo,hi", [(1.0, 4.0), (0.5e-290, 1e-240), (1e-240, 1e-3), (1e-3, 1e3), (1e3, 1e240),
                                   (1e240, 1e280)])
def test_error(math, lo, hi):
    rng = np.random.default_rng(int(abs(np.log10(hi))) + 1)
    x = np.exp(rng.uniform(np.log(lo), np.log(hi), 1 << 20))
    # powers of two and their neighbours
    p = 2.0 ** np.arange(np.ceil(np.log2(lo)), np.floor(np.log2(hi)) + 1)
    x = np.concatenate([x, p, np.nextafter(p, 0.0), np.nextafter(p, np.inf)])
    root, inv = _run(math, x)
    xl = x.astype(np.longdouble)
    exact = 1 / np.sqrt(xl)
    assert np.max(np.abs((root - exact) / exact)) <= 1.6 * U
    if lo >= 1e-240 and hi <= 1e240:  # scale factors: entries in role_in_range
        assert np.max(np.abs((inv - 1 / xl) * xl)) <= 1.01 * U
