// The window QZ and the early deflation with a role per warp (qz_roles.cuh),
// and the chase (qz_chase_roles.cuh), run as thread blocks on the host
// (warp_emu.h).  roles_host.inc and chase_host.inc are those headers with
// their flag loads, flag stores, predicated stores and named barrier, which
// are PTX, left out: they are in emu_prims.h and below.
#include <algorithm>
#include <cfloat>

#include "emu_prims.h"

namespace qz {
inline void chase_bar();
}  // namespace qz
#include "chase_host.inc"
namespace qz {
inline void chase_bar() { emu::named_barrier(1, kChaseMain); }
}  // namespace qz

using namespace qz;

namespace {
struct EmuExec {
  int tid, nt;
  int* si;
  double* sd;
  void sync() { emu::block_barrier(); }
  void stamp(int) {}
  void count(int) {}
};
}  // namespace

extern "C" {
// Window QZ of (H, T) (n x n, in place), Q, Z its factors.  slow: warps that
// run only when the others cannot get on; spin: polls before a wait gives up.
// Returns the status.
int emu_role_qz(int n, double* H, double* T, double* Q, double* Z, unsigned slow, int spin) {
  kRoleSpin = spin;
  const int ld = n % 2 == 0 ? n + 1 : n;
  std::vector<double> mem((size_t)4 * n * ld + kRoleDoubles + 3 * n + 8, NAN);  // (as uninitialised)
  double* const m = mem.data();
  std::vector<int> si(64, -1);
  double hs = 0.0, ts = 0.0;
  for (int j = 0; j < n; ++j)
    for (int i = 0; i < n; ++i) {
      hs += H[i + j * n] * H[i + j * n];
      ts += T[i + j * n] * T[i + j * n];
      m[i + j * ld] = H[i + j * n];
      m[n * ld + i + j * ld] = T[i + j * n];
      m[2 * n * ld + i + j * ld] = m[3 * n * ld + i + j * ld] = i == j ? 1.0 : 0.0;
    }
  RoleBuf* const rb = (RoleBuf*)(m + 4 * n * ld);
  int status = -1;
  emu::run(kRoleThreads, slow, (char*)m, [&](int tid) {
    EmuExec x{tid, kRoleThreads, si.data(), (double*)(rb + 1)};
    WinState w;
    w.n = n;
    w.H = MatV{m, ld};
    w.T = MatV{m + n * ld, ld};
    w.Q = MatV{m + 2 * n * ld, ld};
    w.Z = MatV{m + 3 * n * ld, ld};
    w.wantq = w.wantz = true;
    w.tol.safmin = DBL_MIN;
    w.tol.ulp = DBL_EPSILON;
    w.tol.smlnum = DBL_MIN * ((double)n / DBL_EPSILON);
    w.tol.htol = fmax(DBL_MIN, DBL_EPSILON * sqrt(hs));
    w.tol.ttol = fmax(DBL_MIN, DBL_EPSILON * sqrt(ts));
    const int r = cta_role_qz(x, w, 30 * n, rb);
    if (r == 0) cta_std_all(x, w, x.sd);
    if (tid == 0) status = r;
  });
  for (int j = 0; j < n; ++j)
    for (int i = 0; i < n; ++i) {
      H[i + j * n] = m[i + j * ld];
      T[i + j * n] = m[n * ld + i + j * ld];
      Q[i + j * n] = m[2 * n * ld + i + j * ld];
      Z[i + j * n] = m[3 * n * ld + i + j * ld];
    }
  return status;
}

// Early deflation of a window (n x n, in place) with spike entry s (k_aed_win);
// out3: undeflated, status, changed; shifts: 3 n.
void emu_aed(int n, double* H, double* T, double* Q, double* Z, double s, int nskip, double* shifts, int* out3,
             unsigned slow) {
  kRoleSpin = 1 << 22;
  const int ld = n % 2 == 0 ? n + 1 : n;
  std::vector<double> mem((size_t)4 * n * ld + kRoleDoubles + 64 + 4 * n + 8, NAN);
  double* const m = mem.data();
  std::vector<int> si(64, -1);
  for (int j = 0; j < n; ++j)
    for (int i = 0; i < n; ++i) {
      m[i + j * ld] = H[i + j * n];
      m[n * ld + i + j * ld] = T[i + j * n];
      m[2 * n * ld + i + j * ld] = m[3 * n * ld + i + j * ld] = i == j ? 1.0 : 0.0;
    }
  RoleBuf* const rb = (RoleBuf*)(m + 4 * n * ld);
  emu::run(kRoleThreads, slow, (char*)m, [&](int tid) {
    EmuExec x{tid, kRoleThreads, si.data(), (double*)rb + kRoleDoubles};
    WinState w;
    w.n = n;
    w.H = MatV{m, ld};
    w.T = MatV{m + n * ld, ld};
    w.Q = MatV{m + 2 * n * ld, ld};
    w.Z = MatV{m + 3 * n * ld, ld};
    w.wantq = w.wantz = true;
    w.tol.safmin = DBL_MIN;
    w.tol.ulp = DBL_EPSILON;
    w.tol.smlnum = DBL_MIN * ((double)n / DBL_EPSILON);
    w.tol.htol = w.tol.ttol = DBL_EPSILON * n;
    const int qz = cta_role_qz(x, w, 30 * n, rb);
    if (qz == 0) cta_std_all(x, w, x.sd + 64);
    cta_aed_deflate(
        x, w, s, shifts, shifts + n, shifts + 2 * n, qz, [&]() { return cta_role_spike(x, w, s, nskip, false, rb); },
        [&](int mm) { return cta_role_hessred(x, w, mm, rb); });
  });
  for (int k = 0; k < 3; ++k) out3[k] = si[8 + k];
  for (int j = 0; j < n; ++j)
    for (int i = 0; i < n; ++i) {
      H[i + j * n] = m[i + j * ld];
      T[i + j * n] = m[n * ld + i + j * ld];
      Q[i + j * n] = m[2 * n * ld + i + j * ld];
      Z[i + j * n] = m[3 * n * ld + i + j * ld];
    }
}

// Chase of nb bulges (polynomials coef, 3 each) through a window that ends its
// block: introduced at the top, pushed off at the bottom (k_chase_win).
// Returns 0, or 1 if a wait gave up.
int emu_chase(int n, double* H, double* T, double* U, double* V, const double* coef, int nb, unsigned slow) {
  kRoleSpin = 1 << 22;
  const int ld = n % 2 == 0 ? n + 1 : n;
  const size_t ring = 4 * (size_t)n * ld;
  std::vector<double> mem(ring + chase_ring_doubles(nb) + 8, NAN);
  double* const m = mem.data();
  std::vector<Bulge> bl(nb);
  ChaseShare share{};
  int tmax = 0;
  for (int k = 0; k < nb; ++k) {
    bl[k] = Bulge{-3 * k, 3 * k, n - 1 + 3 * k, 1, coef[3 * k], coef[3 * k + 1], coef[3 * k + 2]};
    tmax = std::max(tmax, bl[k].thi);
  }
  for (int j = 0; j < n; ++j)
    for (int i = 0; i < n; ++i) {
      m[i + j * ld] = H[i + j * n];
      m[n * ld + i + j * ld] = T[i + j * n];
      m[2 * n * ld + i + j * ld] = m[3 * n * ld + i + j * ld] = i == j ? 1.0 : 0.0;
    }
  bool ok = false;
  emu::run(kChaseRoleThreads, slow, (char*)m, [&](int tid) {
    const bool r = cta_chase_roles(n, n - 1, MatV{m, ld}, MatV{m + n * ld, ld}, MatV{m + 2 * n * ld, ld},
                                   MatV{m + 3 * n * ld, ld}, bl.data(), nb, tmax, m + ring, &share);
    if (tid == 0) ok = r;
  });
  for (int j = 0; j < n; ++j)
    for (int i = 0; i < n; ++i) {
      H[i + j * n] = m[i + j * ld];
      T[i + j * n] = m[n * ld + i + j * ld];
      U[i + j * n] = m[2 * n * ld + i + j * ld];
      V[i + j * n] = m[3 * n * ld + i + j * ld];
    }
  return ok ? 0 : 1;
}

// role_wait_done by warp 0 while warps 1 and 2 post their counts up to v:
// lanes of warp 0 whose later reads are ordered behind both counts.
int emu_wait_done(int v) {
  kRoleSpin = 1 << 22;
  std::vector<double> mem(kRoleDoubles, 0.0);
  RoleBuf* const rb = (RoleBuf*)mem.data();
  int lanes = 0;
  emu::run(
      96, 0, (char*)mem.data(),
      [&](int tid) {
        const int warp = tid / 32, lane = tid % 32;
        if (warp != 0) {
          for (int k = 1; k <= v; ++k) {
            __syncwarp();
            if (lane == 0) role_st(&rb->done[warp], k);
          }
          return;
        }
        if (!role_wait_done(rb, kRoleRight, v, lane)) return;
        auto& s = emu::block()->seen[tid];
        if (s[&rb->done[1]] >= v && s[&rb->done[2]] >= v) ++lanes;
      },
      true);
  return lanes;
}
}
