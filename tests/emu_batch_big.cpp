// The one-CTA solve of a batched pencil (batch_big.cuh), run as a thread block
// on the host (warp_emu.h).  batch_big_host.inc is that header with its named
// barriers turned into emu::named_barrier and its shared memory into the
// emulated block's; the tensor-core product is below.
#include <algorithm>
#include <cfloat>

#include "emu_prims.h"

inline int atomicMax(int* p, int v) {
  const int old = *p;
  *p = std::max(old, v);
  return old;
}
inline int atomicAdd(int* p, int v) {
  const int old = *p;
  *p += v;
  return old;
}

namespace qz {
using std::max;
using std::min;
inline void chase_bar();
// mma.m8n8k4: lane l holds A(l / 4, l % 4), B(l % 4, l / 4), C(l / 4, 2 (l % 4) + {0, 1})
inline void dmma_8x8x4(double& d0, double& d1, double a, double b) {
  double A[32], B[32];
  const std::vector<uint64_t>& va = emu::meet(emu_bits(a));
  for (int i = 0; i < 32; ++i) A[i] = emu_double(va[i]);
  const std::vector<uint64_t>& vb = emu::meet(emu_bits(b));
  for (int i = 0; i < 32; ++i) B[i] = emu_double(vb[i]);
  const int row = emu::lane_id() / 4, col = 2 * (emu::lane_id() % 4);
  for (int k = 0; k < 4; ++k) {
    d0 = fma(A[4 * row + k], B[4 * col + k], d0);
    d1 = fma(A[4 * row + k], B[4 * (col + 1) + k], d1);
  }
}
}  // namespace qz
#include "chase_host.inc"
namespace qz {
inline void chase_bar() { emu::named_barrier(1, kChaseMain); }
}  // namespace qz
#include "batch_big_host.inc"

using namespace qz;

// H, T (n x n) in place, Q, Z; returns the status.
extern "C" int emu_big(int n, double* H, double* T, double* Q, double* Z, unsigned slow) {
  std::vector<double> mem(kBigSmem / sizeof(double) + 8);
  memset(mem.data(), 0xff, mem.size() * sizeof(double));
  double hs = 0.0, ts = 0.0;
  for (int k = 0; k < n * n; ++k) {
    hs += H[k] * H[k];
    ts += T[k] * T[k];
    Q[k] = Z[k] = k % (n + 1) == 0 ? 1.0 : 0.0;
  }
  int status = -1;
  emu::run(kBigThreads, slow, (char*)mem.data(), [&](int tid) {
    BigPencil p{H, T, Q, Z, n, {}};
    p.tol.safmin = DBL_MIN;
    p.tol.ulp = DBL_EPSILON;
    p.tol.smlnum = DBL_MIN * ((double)n / DBL_EPSILON);
    p.tol.htol = fmax(DBL_MIN, DBL_EPSILON * sqrt(hs));
    p.tol.ttol = fmax(DBL_MIN, DBL_EPSILON * sqrt(ts));
    const int r = big_solve(p, mem.data(), 30 * n);
    if (tid == 0) status = r;
  });
  return status;
}
