// Hessenberg-triangular reduction on the device: the launch sequence of
// the windowed Givens form in hessred.cuh, with the chain split by rows.
//
// Per column jc: one launch per window, from the bottom of the column up.
// CTA 0 runs the window.  A warp owns 32 rows of the window's block of B, a
// row per lane, and carries each row's entry through the column rotations in
// a register: first those of the window below (walk (a)), then, as other
// warps publish them, those of the pairs below its own rows, then it runs its
// own 32 pairs, where the carries are what the pairs read.  The row rotations
// need the column of A alone, whose carried entries are running norms: a warp
// forms 32 at a time from a scan of squares.  G on the block's own columns is
// left to the walks (f) (Z's of later windows do not reach those entries).
// The other CTAs apply the previous window's rotations elsewhere (walks (e),
// (f), (g)) on entries CTA 0 does not touch, and the pairs of the window's
// rows of the previous column's factors to Q and Z (two sets of rotation
// records).  After the column's last window, one launch applies that window's
// walks and one the column's G to A.
//
// Walks along rows (a lane per row, loads of 32 rows coalesced, 16 ahead of
// the carry) take the Z's and Q; walks down columns (a warp per column, 32
// rotations per affine scan of the carried value) the G's.
//
// Bounds: the chain, a dependent sequence of one reciprocal square root per
// pair on one SM (about n^2/2 pairs): 270 cycles a pair (mostly instruction
// issue of a lone warp), 760 with a barrier per pair; then a window's loads
// and stores through that SM, 16 bytes a cycle.  All in, n = 800 with Q and
// Z: 272 ms then, 86 now (windows of 64 to 160 pairs within 7 % of that);
// n = 2000: 1.79 s then, 0.53 now.
#include "hessred.h"

#include <algorithm>

#include "hessred.cuh"
#include "kernels.h"
#include "qz_roles.cuh"

namespace qz {
namespace {

constexpr int kHrThreads = 512;
constexpr int kHrWarps = kHrThreads / 32;
constexpr int kHrGroups = (kHrMaxWin + 31) / 32;  // row warps of a window
constexpr int kHrSpin = 1 << 22;                  // polls before a wait gives up
constexpr int kHrStage = 64;                      // rotations a row walk stages at a time (a power of two)
constexpr int kHrChunk = 16;                      // entries a row walk reads ahead

__device__ void cp_async8(double* dst, const double* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}
__device__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

__global__ void __launch_bounds__(kHrThreads) k_hr_zero_lower(double* B, int64_t ldb, int n) {
  const int64_t total = (int64_t)n * n;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
    const int r = (int)(i % n), c = (int)(i / n);
    if (r > c) B[r + c * ldb] = 0.0;
  }
}

// Warp walks: the 32 lanes take 32 consecutive rotations of a walk at once.
// The carried value follows a first-order linear recurrence, carry ->
// a carry + b per rotation, so the carries of the 32 steps come from one
// warp scan of the affine maps (five shuffle rounds) instead of 32
// dependent steps, and the 32 loads of a chunk are in flight together.
// The results differ from the one-thread walks only by rounding.
constexpr unsigned kFull = 0xffffffffu;

__device__ void affine_scan(double& a, double& b, int lane) {
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const double ap = __shfl_up_sync(kFull, a, off), bp = __shfl_up_sync(kFull, b, off);
    if (lane >= off) {
      b = a * bp + b;
      a = a * ap;
    }
  }
}

// hr_walk_g by a warp: entries (J-1, J), carry = entry J side; the next 64
// entries and rotations are read ahead.
__device__ void hr_wwalk_g(double* v, int64_t st, int Jhi, int Jlo, const double* rot, int lane) {
  double y = v[(int64_t)Jhi * st], x0, c0, s0, x1, c1, s1;
  auto fetch = [&](double& x, double& c, double& s, int J) {
    x = 0.0; c = 1.0; s = 0.0;
    if (J >= Jlo) {
      x = v[(int64_t)(J - 1) * st];
      const double2 r = *(const double2*)(rot + 4 * (int64_t)J);
      c = r.x;
      s = r.y;
    }
  };
  fetch(x0, c0, s0, Jhi - lane);
  fetch(x1, c1, s1, Jhi - 32 - lane);
  for (int J0 = Jhi; J0 >= Jlo; J0 -= 32) {
    const int J = J0 - lane;
    const bool act = J >= Jlo;
    const double xc = x0, cc = c0, sc = s0;
    x0 = x1; c0 = c1; s0 = s1;
    fetch(x1, c1, s1, J - 64);
    double a = act ? sc : 1.0, b = act ? cc * xc : 0.0;
    affine_scan(a, b, lane);
    const double ynew = a * y + b;
    double yprev = __shfl_up_sync(kFull, ynew, 1);
    if (lane == 0) yprev = y;
    if (act) v[(int64_t)J * st] = -sc * xc + cc * yprev;
    y = __shfl_sync(kFull, ynew, 31);
  }
  if (lane == 0) v[(int64_t)(Jlo - 1) * st] = y;
}

// Rotations Jhi..Jlo along 32 rows, a lane each (element j at row[j * st]):
// hr_walk_z, or hr_walk_g with kG.  Returns the carry, which belongs at
// element Jlo-1.  stage: 2 kHrStage doubles of the warp's own; lanes without
// a row (on false) read the given row and store nothing.
template <bool kG>
__device__ double hr_rows(double* row, int64_t st, int Jhi, int Jlo, const double* rot, double* stage, int lane,
                          bool on) {
  double w = row[(int64_t)Jhi * st];
  double2 r0, r1;
  auto rots = [&](int J) {
    r0 = r1 = make_double2(1.0, 0.0);
    if (J - lane >= Jlo) r0 = *(const double2*)(rot + 4 * (int64_t)(J - lane) + (kG ? 0 : 2));
    if (J - 32 - lane >= Jlo) r1 = *(const double2*)(rot + 4 * (int64_t)(J - 32 - lane) + (kG ? 0 : 2));
  };
  double e[kHrChunk], f[kHrChunk];
  const int64_t stb = -8 * st;
  const char* ld = (const char*)(row + (int64_t)(Jhi - 1) * st);  // next to read
  char* out = (char*)(row + (int64_t)Jhi * st);                   // next to store
  // whole groups without predicates: a walk's rate is that of one warp's
  // instructions
  auto fetch = [&](int J) {
    if (J - (kHrChunk - 1) >= Jlo) {
#pragma unroll
      for (int i = 0; i < kHrChunk; ++i) {
        e[i] = *(const double*)ld;
        ld += stb;
      }
    } else {
#pragma unroll
      for (int i = 0; i < kHrChunk; ++i) e[i] = J - i >= Jlo ? *(const double*)(ld + i * stb) : 0.0;
    }
  };
  rots(Jhi);
  fetch(Jhi);
#pragma unroll 1
  for (int J = Jhi; J >= Jlo; J -= kHrChunk) {
    const int q = (Jhi - J) & (kHrStage - 1);
    if (q == 0) {
      __syncwarp();
      ((double2*)stage)[lane] = r0;
      ((double2*)stage)[lane + 32] = r1;
      __syncwarp();
      rots(J - kHrStage);
    }
#pragma unroll
    for (int i = 0; i < kHrChunk; ++i) f[i] = e[i];
    fetch(J - kHrChunk);
    const double2* const rs = (const double2*)stage + q;
    auto step = [&](int i) {
      const double2 r = rs[i];
      const double cz = r.x, sz = kG ? -r.y : r.y, v = cz * w + sz * f[i];
      w = -sz * w + cz * f[i];
      if (on) *(double*)out = v;
      out += stb;
    };
    if (J - (kHrChunk - 1) >= Jlo) {
#pragma unroll
      for (int i = 0; i < kHrChunk; ++i) step(i);
    } else {
#pragma unroll
      for (int i = 0; i < kHrChunk; ++i)
        if (J - i >= Jlo) step(i);
    }
  }
  return w;
}
template <bool kG>
__device__ void hr_rows_item(double* M, int64_t ld, int r0, int rows, int Jhi, int Jlo, const double* rot,
                             double* stage, int lane) {
  const bool on = r0 + lane < rows;
  double* const row = M + (on ? r0 + lane : rows - 1);
  const double w = hr_rows<kG>(row, ld, Jhi, Jlo, rot, stage, lane, on);
  if (on) row[(int64_t)(Jlo - 1) * ld] = w;
}

// The walks of window (plo, phi) outside the blocks, a warp each: (e) Z on
// rows [0, e_end) of B and (g) on rows 0..ihi of A, 32 at a time, (f) G on
// the columns of B right of column plo (a column of the block takes the
// pairs above its own).
__host__ __device__ int hr_win_warps(const HrArgs& a, int e_end, int plo) {
  return (e_end + 31) / 32 + (a.ihi + 32) / 32 + (a.n - 1 - plo);
}
__device__ void hr_win_warp(const HrArgs& a, int i, int e_end, int plo, int phi, double* stage, int lane) {
  const int ne = (e_end + 31) / 32, ng = (a.ihi + 32) / 32;
  if (i < ne) {
    hr_rows_item<false>(a.B, a.ldb, 32 * i, e_end, phi, plo, a.rot, stage, lane);
  } else if (i < ne + ng) {
    hr_rows_item<false>(a.A, a.lda, 32 * (i - ne), a.ihi + 1, phi, plo, a.rot, stage, lane);
  } else {
    const int t = plo + 1 + i - ne - ng;
    hr_wwalk_g(a.B + (int64_t)t * a.ldb, 1, t - 1 < phi ? t - 1 : phi, plo, a.rot, lane);
  }
}
// Pairs Jhi..Jlo of a column's factors on Q and Z, a warp each.
__host__ __device__ int hr_qz_warps(const HrArgs& a) {
  const int rw = (a.n + 31) / 32;
  return (a.wantq ? (a.qrows ? a.n : rw) : 0) + (a.wantz ? rw : 0);
}
__device__ void hr_qz_warp(const HrArgs& a, int i, int Jhi, int Jlo, const double* rot, double* stage, int lane) {
  const int nq = a.wantq ? (a.qrows ? a.n : (a.n + 31) / 32) : 0;
  if (i < nq) {
    if (a.qrows) hr_wwalk_g(a.Q + (int64_t)i * a.ldq, 1, Jhi, Jlo, rot, lane);
    else hr_rows_item<true>(a.Q, a.ldq, 32 * i, a.n, Jhi, Jlo, rot, stage, lane);
  } else {
    hr_rows_item<false>(a.Z, a.ldz, 32 * (i - nq), a.n, Jhi, Jlo, rot, stage, lane);
  }
}

// Row rotations of a window by one warp: pairs J = m-1 .. 1 of the column
// entries acol (hr_g_chain).  Published rotations: (c, s) in gbuf[4J..].
// The carried entry of a pair is the norm of the entries below with the sign
// of the last one: 32 pairs from a scan of squares, each rotation then normed
// by itself.  Entries outside the range of plain squares: one after another.
__device__ void hr_g_warp(int m, double* acol, double* gbuf, int* ready, int lane) {
  bool ok = true;
  for (int i = lane; i < m; i += 32) {
    const double v = fabs(acol[i]);
    ok = ok && (v == 0.0 || (v > kSafeLo && v < kSafeHi));
  }
  if (!__all_sync(kFull, ok)) {
    if (lane == 0) hr_g_chain(m, acol, gbuf, ready);
    __syncwarp();
    return;
  }
  double y = acol[m - 1];
  for (int J0 = m - 1; J0 >= 1; J0 -= 32) {
    const int J = J0 - lane;
    const double f = J >= 1 ? acol[J - 1] : 0.0;
    double q = f * f;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const double t = __shfl_up_sync(kFull, q, off);
      if (lane >= off) q += t;
    }
    const double nrm = sqrt(y * y + q);
    double r = f < 0.0 ? -nrm : nrm;
    double g = __shfl_up_sync(kFull, r, 1);
    if (lane == 0) g = y;
    double c, s, rr;
    hr_lartg(f, g, c, s, rr);
    if (J >= 1) {
      gbuf[4 * J] = c;
      gbuf[4 * J + 1] = s;
    }
    const int last = J0 < 32 ? J0 - 1 : 31;
    y = __shfl_sync(kFull, rr, last);
  }
  __syncwarp();
  for (int i = lane; i < m; i += 32) acol[i] = i == 0 ? y : 0.0;
  __syncwarp();
}

// shared memory of CTA 0 (windows of up to W pairs); the others use its start
// for their walks' rotations
struct HrWinSmem {
  double* Tw;     // m x hr_ldw(m)
  double* gbuf;   // 4 m: (c, s, cz, sz) by pair
  double* acol;   // m
  double* diag;   // kHrGroups: T(J, J) handed from a warp's last pair to the next warp
  double* stage;  // 2 kHrStage per row warp
  int* count;     // pairs published; row rotations published (by hr_g_chain)
};
__host__ __device__ size_t hr_win_doubles(int W) {
  const size_t m = W + 1, own = (m * hr_ldw(W + 1) + 1) / 2 * 2 + 4 * m + m + kHrGroups + 2 + 2 * kHrStage * kHrGroups + 2;
  const size_t other = 2 * kHrStage * kHrWarps;
  return own > other ? own : other;
}
__device__ __forceinline__ HrWinSmem hr_win_smem(double* sm, int W) {
  const int m = W + 1;
  HrWinSmem L;
  L.Tw = sm;
  L.gbuf = sm + (m * hr_ldw(m) + 1) / 2 * 2;
  L.stage = L.gbuf + 4 * m;
  L.acol = L.stage + 2 * kHrStage * kHrGroups;
  L.diag = L.acol + m;
  L.count = (int*)(L.diag + kHrGroups);
  return L;
}

// squares of a pair's rotation in range: high words of 1e-280 and 1e280
constexpr unsigned kHrSquareLo = 0x05E00000u, kHrSquareHi = 0x7A100000u;
// exact cases and entries out of range (a function of its own: the pairs' loop
// stays short)
__device__ __noinline__ void hr_pair_rare(double f, double g, double& c, double& s, double& r) {
  hr_lartg(f, g, c, s, r);
}

// Row warp g of a window: its rows' carries w (lane l: row jh-1-l) through
// the published pairs, then its own pairs jh..jl.  Tw: the block, in
// place (with global stores in flight a publishing store took 500 cycles).
__device__ __forceinline__ void hr_chain_warp(const HrWinSmem L, int m, int ldw, int g, double w, int lane, int* err) {
  const int jh = m - 1 - 32 * g, jl = jh > 32 ? jh - 31 : 1, row = jh - 1 - lane;
  const bool on = row >= 0;
  double* const Tr = L.Tw + (on ? row : 0);
  const unsigned gz = role_sm(L.gbuf + 2);
  const double2* rz = (const double2*)(L.gbuf + 4 * (m - 1) + 2);
  double* col = Tr + (m - 1) * ldw;
  int avail = 0;
  for (int k = 0; k < 32 * g;) {
    if (avail <= k) {
      for (int it = 0; it < kHrSpin; ++it) {
        avail = hr_ld_acq(L.count);
        if (avail > k) break;
      }
      if (avail <= k) {
        if (lane == 0) atomicExch(err, 1);
        avail = 32 * g;  // no wait any more: the result is reported as lost
      }
      if (avail > 32 * g) avail = 32 * g;
    }
#pragma unroll 1
    for (; k < avail; ++k) {
      const double2 r = *rz;
      const double y = *(col - ldw);
      if (on) *col = r.x * w + r.y * y;
      w = -r.y * w + r.x * y;
      col -= ldw;
      rz -= 2;
    }
  }
  // the lane's own pair J = jh - lane: its row rotation and what that makes of
  // T(J-1, J-1), which no column rotation has reached
  const int own = jh - lane >= 1 ? jh - lane : 1;
  const double2 cs = *(const double2*)(L.gbuf + 4 * own);
  const double d = L.Tw[(own - 1) * (ldw + 1)];
  const double u00 = cs.x * d, u10own = -cs.y * d;
  const unsigned tw = role_sm(L.Tw), tr = role_sm(Tr);
  double t11 = g == 0 ? L.Tw[(m - 1) + (m - 1) * ldw] : L.diag[g];
  double y = Tr[(jh - 1) * ldw];
  // running addresses: the column after the next, the column stored, and
  // lanes 0..2's cz, sz, rz
  const double* ahead = Tr + (jh > 1 ? jh - 2 : 0) * ldw;
  unsigned pt = tr + 8 * jh * ldw, pv = lane == 2 ? tw + 8 * jh * (ldw + 1) : gz + 32 * jh + 8 * lane;
  const unsigned dt = 8 * ldw, dv = lane == 2 ? 8 * (ldw + 1) : 32;
  auto step = [&](int J) {
    const int l = jh - J;
    const bool mine = lane == l;
    const double yn = *ahead;
    if (J > 2) ahead -= ldw;
    // row J of the 2x2 block after the pair's G, from the lane of row J-1,
    // which goes on with row J-1 of it
    const double u11own = cs.x * t11 - cs.y * w;
    const double u11 = __shfl_sync(kFull, u11own, l), u10 = __shfl_sync(kFull, u10own, l);
    const double u01 = cs.x * w + cs.y * t11;
    w = mine ? u01 : w;
    y = mine ? u00 : y;
    // every row's two entries: numerators formed beside the root
    const double q = u11 * u11 + u10 * u10;
    const double no = u11 * w + u10 * y, nw = u11 * y - u10 * w;
    const double inv = role_rsqrt(q);
    const double si = __hiloint2double(__double2hiint(inv) | (__double2hiint(u11) & 0x80000000), __double2loint(inv));
    double out = no * si, wn = nw * si;
    // lanes 0..2: cz, sz, rz
    double v = (lane == 0 ? u11 : lane == 1 ? u10 : q) * si;
    const unsigned hq = (unsigned)__double2hiint(q);
    if (hq - kHrSquareLo >= kHrSquareHi - kHrSquareLo || u10 == 0.0 || u11 == 0.0) {
      double cz, sz, rz;
      hr_pair_rare(u11, u10, cz, sz, rz);
      out = cz * w + sz * y;
      wn = -sz * w + cz * y;
      v = lane == 0 ? cz : lane == 1 ? sz : rz;
    }
    role_put(lane < 3, pv, v);
    role_put(on && lane >= l, pt, out);
    pv -= dv;
    pt -= dt;
    t11 = __shfl_sync(kFull, wn, l);
    w = wn;
    y = yn;
  };
  auto publish = [&](int J) {
    if (J == jl && lane == 0) {
      if (g + 1 < kHrGroups) L.diag[g + 1] = t11;
      if (jl == 1) L.Tw[0] = t11;
    }
    __syncwarp();
    if (lane == 0) hr_st_rel(L.count, m - J);
  };
  // eight pairs between the branches (a taken branch costs a lone warp more
  // than the arithmetic between two of them)
  int J = jh;
#pragma unroll 1
  for (; J - 7 >= jl; J -= 8) {
#pragma unroll
    for (int u = 0; u < 8; ++u) step(J - u);
    publish(J - 7);
  }
#pragma unroll 1
  for (; J >= jl; --J) {
    step(J);
    publish(J);
  }
}

// CTA 0 of a window launch: window (lo, hi) of column jc, previous window
// (plo, phi) of the column (plo < 0: none).
__device__ __forceinline__ void hr_window_cta(const HrArgs& a, int jc, int lo, int hi, int plo, int phi, double* sm, int wmax) {
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int o = lo - 1, m = hi - lo + 2, ldw = hr_ldw(m), groups = (m + 30) / 32;
  const HrWinSmem L = hr_win_smem(sm, wmax);
  double* const Bo = a.B + o + (int64_t)o * a.ldb;
  double w = 0.0;
  if (tid == 0) L.count[0] = L.count[1] = 0;
  if (warp < groups) {
    // the carries: column hi of the lane's row, after (a)
    const int row = m - 2 - 32 * warp - lane;
    const bool on = row >= 0;
    double* const r = a.B + o + (on ? row : 0);
    w = plo >= 0 ? hr_rows<false>(r, a.ldb, phi, plo, a.rot, L.stage + 2 * kHrStage * warp, lane, on)
                 : r[(int64_t)hi * a.ldb];
  } else if (warp == kHrGroups) {
    for (int i = lane; i < m; i += 32) L.acol[i] = a.A[(o + i) + (int64_t)jc * a.lda];
    __syncwarp();
    hr_g_warp(m, L.acol, L.gbuf, L.count + 1, lane);
    for (int i = lane; i < m; i += 32) a.A[(o + i) + (int64_t)jc * a.lda] = L.acol[i];
  } else if (warp > kHrGroups) {
    for (int j = warp - kHrGroups - 1; j < m; j += kHrWarps - kHrGroups - 1)
      for (int i = lane; i <= j; i += 32) cp_async8(&L.Tw[i + j * ldw], Bo + i + (int64_t)j * a.ldb);
    cp_async_wait_all();
  }
  __syncthreads();
  if (warp < groups) hr_chain_warp(L, m, ldw, warp, w, lane, a.err);
  __syncthreads();
  // The records, normed to first order: c and s of a pair are rounded
  // separately, c^2 + s^2 is off by 1.2 units of rounding (root mean square;
  // 0.65 so), and every pair multiplies that into whole rows of Q and Z.
  for (int i = 2 + tid; i < 2 * m; i += kHrThreads) {
    double2 r = ((const double2*)L.gbuf)[i];
    const double h = 0.5 * fma(-r.y, r.y, fma(-r.x, r.x, 1.0));
    r.x = fma(r.x, h, r.x);
    r.y = fma(r.y, h, r.y);
    ((double2*)(a.rot + 4 * (int64_t)o))[i] = r;
  }
  for (int j = warp; j < m; j += kHrWarps)
    for (int i = lane; i <= j; i += 32) Bo[i + (int64_t)j * a.ldb] = L.Tw[i + j * ldw];
}

// Window (lo, hi) of column jc; (plo, phi): the previous window of the
// column (plo < 0: none).  CTA 0 runs the window, the others the previous
// window's walks and, of the previous column's factors on Q and Z (its
// records: prev; null: none), the pairs of this window's rows.  (All of them
// in a column's first launch took 98 us of it at n = 2000, where a window
// takes 39.)
__global__ void __launch_bounds__(kHrThreads) k_hr_win(HrArgs a, int jc, int lo, int hi, int plo, int phi, int wmax,
                                                       const double* prev) {
  extern __shared__ __align__(16) double sm[];
  if (blockIdx.x > 0) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, n = gridDim.x - 1;
    double* const stage = sm + 2 * kHrStage * warp;
    const int wins = plo >= 0 ? hr_win_warps(a, lo - 1, plo) : 0, items = wins + (prev ? hr_qz_warps(a) : 0);
    // column jc - 1 has one pair more, the topmost
    const int qlo = lo == jc + 2 ? jc + 1 : lo;
    for (int i = (blockIdx.x - 1) + warp * n; i < items; i += n * kHrWarps) {
      if (i < wins) hr_win_warp(a, i, lo - 1, plo, phi, stage, lane);
      else hr_qz_warp(a, i - wins, hi, qlo, prev, stage, lane);
    }
    return;
  }
  hr_window_cta(a, jc, lo, hi, plo, phi, sm, wmax);
}

// The walks of a column's last window (plo, phi).
__global__ void __launch_bounds__(kHrThreads) k_hr_flush(HrArgs a, int plo, int phi) {
  __shared__ __align__(16) double stage[2 * kHrStage * kHrWarps];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, items = hr_win_warps(a, plo - 1, plo);
  for (int i = blockIdx.x + warp * gridDim.x; i < items; i += gridDim.x * kHrWarps)
    hr_win_warp(a, i, plo - 1, plo, phi, stage + 2 * kHrStage * warp, lane);
}

// Column jc's G on columns jc+1..n-1 of A.
__global__ void __launch_bounds__(kHrThreads) k_hr_colend(HrArgs a, int jc) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, items = a.n - 1 - jc;
  for (int i = blockIdx.x + warp * gridDim.x; i < items; i += gridDim.x * kHrWarps)
    hr_wwalk_g(a.A + (int64_t)(jc + 1 + i) * a.lda, 1, a.ihi, jc + 2, a.rot, lane);
}

// The last column's factors on Q and Z.
__global__ void __launch_bounds__(kHrThreads) k_hr_qz(HrArgs a, int jc) {
  __shared__ __align__(16) double stage[2 * kHrStage * kHrWarps];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, items = hr_qz_warps(a);
  for (int i = blockIdx.x + warp * gridDim.x; i < items; i += gridDim.x * kHrWarps)
    hr_qz_warp(a, i, a.ihi, jc + 2, a.rot, stage + 2 * kHrStage * warp, lane);
}

int blocks_for(int items) { return std::max(1, (items + kHrThreads - 1) / kHrThreads); }
// warp items over the SMs, one CTA each at most
int item_blocks(int items, int sms) { return std::max(1, std::min(items, sms)); }

}  // namespace

cudaError_t gghrd_device(cudaStream_t st, int icompq, int icompz, bool qrows, int n, int ilo, int ihi, double* A,
                         int64_t lda, double* B, int64_t ldb, double* Q, int64_t ldq, double* Z, int64_t ldz, int wmax,
                         GghrdOut* out) {
  if (out) *out = GghrdOut{};
  if (icompq == 2) launch_identity(st, Q, ldq, n);
  if (icompz == 2) launch_identity(st, Z, ldz, n);
  if (n > 1) k_hr_zero_lower<<<std::min(1184, blocks_for(n * n)), kHrThreads, 0, st>>>(B, ldb, n);
  int64_t launches = (icompq == 2) + (icompz == 2) + (n > 1), pairs = 0;
  if (out) out->launches = launches;
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess || n <= 1 || ihi - ilo < 2) return e;
  const int W = std::max(2, std::min(wmax, kHrMaxWin));
  const size_t smem = hr_win_doubles(W) * sizeof(double);
  e = cudaFuncSetAttribute(k_hr_win, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  int dev = 0, sms = 0;
  e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (e != cudaSuccess) return e;
  // two sets of rotation records: a column's and the one's before it
  double* rot = nullptr;
  e = cudaMallocAsync(&rot, sizeof(double) * (8 * (size_t)n + 1), st);
  if (e != cudaSuccess) return e;
  int* err = (int*)(rot + 8 * (size_t)n);
  e = cudaMemsetAsync(err, 0, sizeof(int), st);
  if (e != cudaSuccess) return e;
  HrArgs a{A, lda, B, ldb, Q, ldq, Z, ldz, rot, err, n, ihi, icompq != 0, icompz != 0, qrows};
  const int qz = hr_qz_warps(a);
  for (int jc = ilo; jc <= ihi - 2 && e == cudaSuccess; ++jc) {
    a.rot = rot + 4 * (size_t)n * ((jc - ilo) & 1);
    const double* prev = jc > ilo ? rot + 4 * (size_t)n * ((jc - ilo + 1) & 1) : nullptr;
    int plo = -1, phi = -1;
    for (int hi = ihi; hi >= jc + 2;) {
      const int lo = hr_win_lo(jc, hi, W);
      const int items = (plo >= 0 ? hr_win_warps(a, lo - 1, plo) : 0) + (prev ? qz : 0);
      const int helpers = std::min(items, std::max(1, sms - 1));
      k_hr_win<<<1 + helpers, kHrThreads, smem, st>>>(a, jc, lo, hi, plo, phi, W, prev);
      ++launches;
      pairs += hi - lo + 1;
      plo = lo;
      phi = hi;
      hi = lo - 1;
    }
    k_hr_flush<<<item_blocks(hr_win_warps(a, plo - 1, plo), sms), kHrThreads, 0, st>>>(a, plo, phi);
    k_hr_colend<<<item_blocks(n - 1 - jc, sms), kHrThreads, 0, st>>>(a, jc);
    launches += 2;
    e = cudaGetLastError();
  }
  if (e == cudaSuccess && qz > 0) {
    // (a.rot: the last column's records)
    k_hr_qz<<<item_blocks(qz, sms), kHrThreads, 0, st>>>(a, ihi - 2);
    ++launches;
    e = cudaGetLastError();
  }
  int herr = 0;
  if (e == cudaSuccess) e = cudaMemcpyAsync(&herr, err, sizeof(int), cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  const cudaError_t ef = cudaFreeAsync(rot, st);
  if (e == cudaSuccess) e = ef;
  if (e == cudaSuccess && herr != 0) e = cudaErrorLaunchTimeout;
  if (out) { out->launches = launches; out->pairs = pairs; }
  return e;
}

}  // namespace qz
