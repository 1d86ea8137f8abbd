// Which blocks a reordering swaps, where and when (host code).
//
// The selected blocks have to lead, selected and unselected ones each in
// their old order: a stable 0/1 sort of the diagonal blocks by adjacent
// swaps, as many as there are (unselected, selected) inversions whatever
// their order.  Windows on a grid of row intervals of kReoStride, shifted by
// half an interval every other phase, each sort what they hold; the windows of a
// phase are disjoint, so a phase is one launch with a CTA per window and two
// batched updates.  When no window of either grid has an inversion, no two
// neighbours have one.  Inside a window the swaps go by rounds of an
// odd-even transposition sort, whose pairs are disjoint.
#pragma once
#include <cstdint>
#include <utility>
#include <vector>

namespace qz {

constexpr int kReoStride = 78;        // rows of a grid interval (even)
constexpr int kReoWin = 80;           // largest window: kReoStride and a 2x2 block that starts on its last row
constexpr int kReoPairs = kReoWin / 2;  // most swaps of a round

struct ReoWindow {
  int w0, wk;     // first row, rows
  int r0, rounds; // its rounds in ReoPlan::round (rounds + 1 entries: first swap of each, then the end)
};
struct ReoPhase {
  int first, count;  // its windows in ReoPlan::win
};
struct ReoPlan {
  std::vector<ReoPhase> phase;
  std::vector<ReoWindow> win;
  std::vector<int> round;
  std::vector<int> swap;  // row inside the window | size of the first block << 8 | of the second << 12
  int64_t swaps = 0;
  int most = 0;           // windows of the largest phase
};

// sz, sel: sizes (1, 2) and selection of the diagonal blocks in order; left
// in the order after the plan.
inline void reorder_plan(std::vector<int>& sz, std::vector<int>& sel, ReoPlan& P) {
  const int nb = (int)sz.size();
  int idle = 0;  // phases in a row without an inversion
  for (int ph = 0; idle < 2; ++ph) {
    ReoPhase F{(int)P.win.size(), 0};
    const int off = (ph & 1) ? kReoStride / 2 : 0;
    int b = 0, row = 0;
    while (b < nb) {
      // blocks that start in the interval of this row
      const int end = row < off ? off : off + ((row - off) / kReoStride + 1) * kReoStride;
      int e = b, r = row;
      bool inv = false, seen = false;
      while (e < nb && r < end) {
        if (!sel[e]) seen = true;
        else if (seen) inv = true;
        r += sz[e++];
      }
      if (inv) {
        // from the first unselected block to the last selected one
        int lo = b, lrow = row, hi = e;
        while (sel[lo]) lrow += sz[lo++];
        while (!sel[hi - 1]) --hi;
        ReoWindow W{lrow, 0, (int)P.round.size(), 0};
        for (int k = lo; k < hi; ++k) W.wk += sz[k];
        int quiet = 0;
        for (int par = 0; quiet < 2; par ^= 1) {
          const int s0 = (int)P.swap.size();
          int pos = 0;
          for (int k = lo; k < hi; ++k) {
            if (((k - lo) & 1) == par && k + 1 < hi && !sel[k] && sel[k + 1]) {
              P.swap.push_back(pos | sz[k] << 8 | sz[k + 1] << 12);
              std::swap(sz[k], sz[k + 1]);
              std::swap(sel[k], sel[k + 1]);
              pos += sz[k] + sz[k + 1];
              ++k;
            } else {
              pos += sz[k];
            }
          }
          if ((int)P.swap.size() > s0) {
            P.round.push_back(s0);
            ++W.rounds;
            quiet = 0;
          } else {
            ++quiet;
          }
        }
        P.round.push_back((int)P.swap.size());
        P.win.push_back(W);
        ++F.count;
      }
      b = e;
      row = r;
    }
    if (F.count == 0) { ++idle; continue; }
    idle = 0;
    P.phase.push_back(F);
    if (F.count > P.most) P.most = F.count;
  }
  P.swaps = (int64_t)P.swap.size();
}

}  // namespace qz
