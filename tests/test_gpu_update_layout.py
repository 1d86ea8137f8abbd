"""The update kernels' two ways of staging (16-byte pieces where every run of
the slab or factor starts on 16 bytes, 8-byte ones elsewhere): even and odd
leading dimensions and origins, factors inside a larger matrix, orders that
are no multiple of the 16-row slices, slabs that end inside a tile, against
the FP64 product to 8 k eps of |W| |M|, nothing outside the slab touched."""
import numpy as np
import pytest
import torch

from conftest import EPS

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("side", ["L", "R"])
@pytest.mark.parametrize("k,length,r0,c0,pad,ldw", [(64, 64, 4, 2, 0, 64), (64, 65, 4, 3, 1, 64), (64, 31, 3, 2, 2, 66),
                                                    (63, 100, 2, 2, 0, 64), (17, 33, 0, 0, 1, 17), (128, 40, 6, 1, 2, 128),
                                                    (2, 1, 0, 0, 0, 2), (50, 500, 2, 4, 0, 51)])
def test_update_layouts(pkg, side, k, length, r0, c0, pad, ldw):
    rng = np.random.default_rng(k + length + r0)
    W = rng.standard_normal((ldw, k))
    rows, cols = (r0 + k, c0 + length + 3) if side == "L" else (r0 + length, c0 + k + 3)
    ld = rows + (rows & 1) + pad  # even, or odd with pad 1
    M = rng.standard_normal((ld, cols))
    dM = torch.from_numpy(M.T.copy()).cuda()
    dW = torch.from_numpy(W.T.copy()).cuda()
    s = pkg.Solver(0)
    try:
        assert pkg.lib().b200qz_update(s.handle, side.encode(), dM.data_ptr(), ld, r0, c0, length, dW.data_ptr(), ldw,
                                       k) == 0
    finally:
        s.close()
    out = dM.cpu().numpy().T
    Wk = W[:k]
    ref = M.copy()
    if side == "L":
        sl = (slice(r0, r0 + k), slice(c0, c0 + length))
        ref[sl] = Wk.T @ M[sl]
        scale = np.abs(Wk.T) @ np.abs(M[sl])
    else:
        sl = (slice(r0, r0 + length), slice(c0, c0 + k))
        ref[sl] = M[sl] @ Wk
        scale = np.abs(M[sl]) @ np.abs(Wk)
    assert np.all(np.abs(out[sl] - ref[sl]) <= 8 * k * EPS * scale)
    mask = np.ones(M.shape, dtype=bool)
    mask[sl] = False
    assert np.array_equal(out[mask], M[mask])
