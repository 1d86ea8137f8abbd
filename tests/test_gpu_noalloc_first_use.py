"""The batched solve that allocates nothing, in a process of its own: after the
first call, which sets the device up whatever its pencils are, no call takes
device memory, the first one with pencils above order 80 included (they run in
a kernel of their own, with a larger stack per thread)."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))

CHILD = """
import torch
from conftest import load_package
from test_zz_no_alloc import _buffers, _noalloc
pkg = load_package()
taken = []
for sizes in ([5, 20, 60], [5, 20, 60], [100, 81], [200, 3]):
    b = pkg.Batch(sizes)
    mats = [pkg.pencils.random_ht(n, 1 + i, 0.0) for i, n in enumerate(sizes)]
    h, t = (torch.from_numpy(b.pack([m[k] for m in mats])).cuda() for k in (0, 1))
    bufs = _buffers(torch, b, h, t)
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    assert _noalloc(pkg, b, *bufs, stream=torch.cuda.current_stream().cuda_stream) == 0
    torch.cuda.synchronize()
    taken.append(free - torch.cuda.mem_get_info()[0])
    assert not bufs[5].any()
print("taken", *taken)
"""


def test_no_memory_after_the_first_call():
    r = subprocess.run([sys.executable, "-c", CHILD], cwd=HERE, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    taken = [int(v) for v in r.stdout.split("taken")[1].split()]
    assert taken[1:] == [0, 0, 0], taken
