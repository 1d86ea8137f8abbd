"""The plan of a reordering (reorder_plan.h), built for the host: its swaps,
applied in order, give the stable partition of the blocks by selection with
exactly as many swaps as the one-block-at-a-time reordering needs (the
inversions); every window holds whole blocks in at most 80 rows, windows of a
phase and swaps of a round are disjoint, and no round has more swaps than the
kernel has room for."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
SRC = r'''
#include "reorder_plan.h"
using namespace qz;
static ReoPlan P;
extern "C" int plan(int nb, const int* sz, const int* sel, int* counts) {
  P = ReoPlan();
  std::vector<int> s(sz, sz + nb), e(sel, sel + nb);
  reorder_plan(s, e, P);
  counts[0] = (int)P.phase.size(); counts[1] = (int)P.win.size(); counts[2] = (int)P.round.size();
  counts[3] = (int)P.swap.size(); counts[4] = P.most;
  return kReoPairs;
}
extern "C" void fetch(int* phase, int* win, int* round, int* swap) {
  for (auto& f : P.phase) { *phase++ = f.first; *phase++ = f.count; }
  for (auto& w : P.win) { *win++ = w.w0; *win++ = w.wk; *win++ = w.r0; *win++ = w.rounds; }
  for (int r : P.round) *round++ = r;
  for (int k : P.swap) *swap++ = k;
}
'''
_pi = ctypes.POINTER(ctypes.c_int)


@pytest.fixture(scope="module")
def planner(tmp_path_factory):
    d = tmp_path_factory.mktemp("plan")
    src, out = str(d / "p.cpp"), str(d / "libplan.so")
    with open(src, "w") as f:
        f.write(SRC)
    inc = os.path.join(HERE, "..", "gevp-pdhgeqz_b200", "csrc")
    subprocess.run(["g++", "-O2", "-shared", "-fPIC", "-std=c++17", "-I", inc, src, "-o", out], check=True,
                   capture_output=True, timeout=120)
    return ctypes.CDLL(out)


def _plan(L, sz, sel):
    sz, sel = (np.ascontiguousarray(v, dtype=np.int32) for v in (sz, sel))
    c = (ctypes.c_int * 5)()
    pairs = L.plan(len(sz), sz.ctypes.data_as(_pi), sel.ctypes.data_as(_pi), c)
    ph, wi, ro, sw = (np.zeros(max(1, k), dtype=np.int32) for k in (2 * c[0], 4 * c[1], c[2], c[3]))
    L.fetch(*(v.ctypes.data_as(_pi) for v in (ph, wi, ro, sw)))
    return ph[:2 * c[0]].reshape(-1, 2), wi[:4 * c[1]].reshape(-1, 4), ro[:c[2]], sw[:c[3]], c[4], pairs


@pytest.mark.parametrize("nb,share,ones,seed", [(1, 1.0, 0.5, 0), (2, 0.5, 0.0, 1), (39, 0.5, 0.0, 2),
                                                 (40, 0.3, 0.0, 3), (78, 0.5, 1.0, 4), (80, 0.5, 1.0, 5),
                                                 (200, 0.4, 0.1, 6), (500, 0.05, 0.3, 7), (500, 0.95, 0.7, 8),
                                                 (90, 0.0, 0.5, 9), (90, 1.0, 0.5, 10)])
def test_plan_is_the_stable_partition(planner, nb, share, ones, seed):
    rng = np.random.default_rng(seed)
    sz = np.where(rng.random(nb) < ones, 1, 2)
    sel = (rng.random(nb) < share).astype(int)
    if seed in (2, 5):  # the worst order: every unselected block first
        sel = np.sort(sel)
    phases, wins, rounds, swaps, most, room = _plan(planner, sz, sel)
    ids, size = list(range(nb)), list(sz)
    inv = sum(int(np.sum(sel[k + 1:])) for k in range(nb) if not sel[k])
    assert len(swaps) == inv and (len(phases) == 0 or most == phases[:, 1].max())
    for first, count in phases:
        used = set()
        for w0, wk, r0, nr in wins[first:first + count]:
            assert 2 <= wk <= 80
            rows = set(range(w0, w0 + wk))
            assert not rows & used
            used |= rows
            starts = np.concatenate([[0], np.cumsum(size)])
            assert w0 in starts and w0 + wk in starts
            for r in range(r0, r0 + nr):
                mine = set()
                assert 0 < rounds[r + 1] - rounds[r] <= room
                for s in swaps[rounds[r]:rounds[r + 1]]:
                    j, n1, n2 = int(s) & 255, (int(s) >> 8) & 15, int(s) >> 12
                    cells = set(range(j, j + n1 + n2))
                    assert not cells & mine and max(cells) < wk
                    mine |= cells
                    b = int(np.searchsorted(np.concatenate([[0], np.cumsum(size)]), w0 + j))
                    assert (size[b], size[b + 1]) == (n1, n2)
                    assert not sel[ids[b]] and sel[ids[b + 1]]
                    ids[b], ids[b + 1] = ids[b + 1], ids[b]
                    size[b], size[b + 1] = size[b + 1], size[b]
    assert ids == [k for k in range(nb) if sel[k]] + [k for k in range(nb) if not sel[k]]
