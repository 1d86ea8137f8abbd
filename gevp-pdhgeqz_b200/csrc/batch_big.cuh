// Solve of one pencil that does not fit shared memory by one CTA (device):
// the iteration of qz_solver.h (deflation scan, zero chasing, aggressive
// early deflation, chains of bulges, endgame) with the window routines of the
// single-pencil kernels and the updates between them, for the batched solver.
//
// Windows live in shared memory; a window's factors update the rest of H and
// T, Q and Z in 32-wide slab tiles on the FP64 tensor cores (two groups of
// eight warps, a tile each).  What bounds it, at n = 300 with every SM
// occupied (about 80 ms a pencil): the early deflations, 45 % (52 of 1.3M
// cycles: serial chains of rotations), the updates, 30 % (300 of 160k
// cycles, 2.4 times the tensor rate, as 148 pencils' matrices do not stay in
// L2), and the chases, 22 % (115k cycles each: a serial chain of reflectors).
#pragma once
#include "qz_chase_roles.cuh"
#include "qz_solver.h"
#include "update.cuh"

namespace qz {

constexpr int kBigThreads = kChaseRoleThreads;  // 512
constexpr int kBigChase = 64;                   // chase window, 8 bulges per chain
constexpr int kBigBulges = kChaseWarps;
constexpr int kBigEnd = 80;                     // active blocks this small are one window
constexpr int kBigShifts = kBigEnd;             // most shifts of an AED
static_assert(kBigEnd <= kRoleMax, "endgame window");

// odd leading dimension (kernels.h smem_ld)
__host__ __device__ constexpr int big_ld(int n) { return (n % 2 == 0) ? n + 1 : n; }

// shared state behind the window matrices
struct BigShare {
  Bulge bl[kBigBulges];
  double poly[3 * (kBigShifts / 2)];
  double shift[3 * kBigShifts];
  ChaseShare chase;
  int scan[4];  // ktop, count of zeros, lowest zero, bad
  int si[64];
  int npoly;
};
// doubles: four 80 x 81 windows (or chase windows and slab tiles), the role
// buffer or the chase ring, the AED's scratch
constexpr int kBigWin = kBigEnd * (kBigEnd + 1);
constexpr int kBigRing = kRoleDoubles > kChaseSlots * kBigBulges * kChaseRecDoubles
                             ? kRoleDoubles : kChaseSlots * kBigBulges * kChaseRecDoubles;
constexpr int kBigScratch = 64 + 4 * kBigEnd;
constexpr size_t kBigSmem = (size_t)(4 * kBigWin + kBigRing + kBigScratch) * sizeof(double) + sizeof(BigShare);

#ifdef __CUDACC__

// the first kRoleThreads threads of the CTA
struct BigExec {
  int tid, nt;
  int* si;
  double* sd;
  __device__ void sync() { asm volatile("bar.sync 2, %0;" ::"n"(kRoleThreads) : "memory"); }
  __device__ void stamp(int) {}
  __device__ void count(int) {}
};
// all of them
struct BigExecAll {
  int tid, nt;
  int* si;
  double* sd;
  __device__ void sync() { __syncthreads(); }
  __device__ void stamp(int) {}
  __device__ void count(int) {}
};

struct BigPencil {
  double *H, *T, *Q, *Z;
  int n;
  Tol tol;
};

// shared-memory carve-up (all threads hold the same)
struct BigMem {
  double* win;   // 4 kBigWin
  double* ring;
  double* sd;
  BigShare* sh;
};
__device__ inline BigMem big_mem(double* smem) {
  BigMem m;
  m.win = smem;
  m.ring = smem + 4 * kBigWin;
  m.sd = m.ring + kBigRing;
  m.sh = (BigShare*)(m.sd + kBigScratch);
  return m;
}

__device__ inline void big_load(const BigPencil& p, int w, int wk, double* Hs, double* Ts, double* Us, double* Vs,
                                int ld, int ldu) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = kBigThreads / 32;
  for (int j = warp; j < wk; j += nw)
    for (int i = lane; i < wk; i += 32) {
      const size_t g = (size_t)(w + i) + (size_t)(w + j) * p.n;
      Hs[i + j * ld] = p.H[g];
      Ts[i + j * ld] = p.T[g];
      Us[i + j * ldu] = i == j ? 1.0 : 0.0;
      Vs[i + j * ldu] = i == j ? 1.0 : 0.0;
    }
  __syncthreads();
}
__device__ inline void big_store(const BigPencil& p, int w, int wk, const double* Hs, const double* Ts, int ld) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = kBigThreads / 32;
  __syncthreads();
  for (int j = warp; j < wk; j += nw)
    for (int i = lane; i < wk; i += 32) {
      const size_t g = (size_t)(w + i) + (size_t)(w + j) * p.n;
      p.H[g] = Hs[i + j * ld];
      p.T[g] = Ts[i + j * ld];
    }
  __syncthreads();
}

// A tile of an update: M(w:w+k, o:o+len) <- W^T M (left) or M(o:o+len, w:w+k)
// <- M W (right), at most 32 of the other dimension.
struct BigTile {
  double* M;
  const double* W;
  int o, len;
};
constexpr int kBigSlabLd = kBigEnd + 4;                 // left slab tile
constexpr int kBigSlab = kBigEnd * kUpdRightLd;         // doubles of a group's tile
constexpr int kBigHold = 3 * (kUpdTile / 8);            // elements of a tile per thread
static_assert(kBigSlabLd * kUpdTile <= kBigSlab, "slab tile");
static_assert(kBigEnd <= 96 && kBigEnd <= 8 * kBigHold, "elements held");

// The thread's elements of a tile, zero outside it.  Left: rows lane,
// lane + 32, lane + 64 of columns warp, warp + 8, ..; right: row lane of
// columns warp, warp + 8, ..
template <bool kLeft>
__device__ __forceinline__ void big_fetch(const BigTile& t, int n, int w, int k, double (&v)[kBigHold]) {
  const int warp = (threadIdx.x & 255) >> 5, lane = threadIdx.x & 31;
#pragma unroll
  for (int e = 0; e < kBigHold; ++e) {
    const int i = kLeft ? lane + 32 * (e % 3) : lane, j = warp + 8 * (kLeft ? e / 3 : e);
    const bool in = kLeft ? (i < k && j < t.len) : (i < t.len && j < k);
    v[e] = in ? t.M[kLeft ? (size_t)(w + i) + (size_t)(t.o + j) * n : (size_t)(t.o + i) + (size_t)(w + j) * n] : 0.0;
  }
}
template <bool kLeft>
__device__ __forceinline__ void big_put(double* X, int kp, const double (&v)[kBigHold]) {
  const int warp = (threadIdx.x & 255) >> 5, lane = threadIdx.x & 31;
#pragma unroll
  for (int e = 0; e < kBigHold; ++e) {
    const int i = kLeft ? lane + 32 * (e % 3) : lane, j = warp + 8 * (kLeft ? e / 3 : e);
    if (kLeft ? i < kp : j < kp) X[kLeft ? i + j * kBigSlabLd : i + j * kUpdRightLd] = v[e];
  }
}

// The tiles t = grp, grp + 2, .. below count, by the 256 threads of group
// grp; W in shared memory.  The next tile's elements are read while this
// one's product runs: with the reads waited for, the updates of a window of
// 64 rows at n = 320 took 199k cycles, with them ahead 156k (24 tiles, 2.0k
// cycles each at the SM's FP64 tensor rate, on two groups).
template <bool kLeft, class TileOf>
__device__ __forceinline__ void big_tiles(const TileOf& tile_of, int count, int n, int w, int k, int ldw, double* X,
                                          int grp) {
  const int warp = (threadIdx.x & 255) >> 5, lane = threadIdx.x & 31, lr = lane >> 2, lc = lane & 3;
  const int kp = (k + 15) & ~15, half = warp & 1;
  auto bar = [&]() { asm volatile("bar.sync %0, 256;" ::"r"(3 + grp) : "memory"); };
  double v[kBigHold];
  BigTile t{};
  if (grp < count) {
    t = tile_of(grp);
    big_fetch<kLeft>(t, n, w, k, v);
  }
  for (int q = grp; q < count; q += 2) {
    bar();  // the last product has read the slab
    big_put<kLeft>(X, kp, v);
    bar();
    const BigTile now = t;
    if (q + 2 < count) {
      t = tile_of(q + 2);
      big_fetch<kLeft>(t, n, w, k, v);
    }
    for (int sl = warp >> 1; sl < kp / 16; sl += 4) {
      double acc[2][2][2] = {};
      for (int kk = 0; kk < kp; kk += 4) {
        double wf[2], xf[2];
#pragma unroll
        for (int a = 0; a < 2; ++a) {
          const int i = kk + lc, j = sl * 16 + a * 8 + lr;
          wf[a] = (i < k && j < k) ? now.W[i + j * ldw] : 0.0;
          xf[a] = kLeft ? X[i + (half * 16 + a * 8 + lr) * kBigSlabLd] : X[half * 16 + a * 8 + lr + i * kUpdRightLd];
        }
#pragma unroll
        for (int a = 0; a < 2; ++a)
#pragma unroll
          for (int b = 0; b < 2; ++b)
            dmma_8x8x4(acc[a][b][0], acc[a][b][1], kLeft ? wf[a] : xf[a], kLeft ? xf[b] : wf[b]);
      }
#pragma unroll
      for (int a = 0; a < 2; ++a)
#pragma unroll
        for (int b = 0; b < 2; ++b)
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const int x = a * 8 + lr, y = b * 8 + lc * 2 + e;
            const int i = kLeft ? sl * 16 + x : half * 16 + x, j = kLeft ? half * 16 + y : sl * 16 + y;
            if (kLeft ? (i < k && j < now.len) : (i < now.len && j < k))
              now.M[kLeft ? (size_t)(w + i) + (size_t)(now.o + j) * n : (size_t)(now.o + i) + (size_t)(w + j) * n] =
                  acc[a][b][e];
          }
    }
  }
}

// The window's factors on the rest: H, T right of it, then H, T above it and
// Q, Z.  X: two slab tiles.
__device__ inline void big_update(const BigPencil& p, int w, int wk, const double* U, const double* V, int ldu,
                                  double* X) {
  const int grp = threadIdx.x >> 8, n = p.n;
  double* const Xg = X + grp * kBigSlab;
  const int right = n - (w + wk), tr = (right + kUpdTile - 1) / kUpdTile;
  big_tiles<true>(
      [&](int t) {
        const int c = (t < tr ? t : t - tr) * kUpdTile;
        return BigTile{t < tr ? p.H : p.T, U, w + wk + c, right - c};
      },
      2 * tr, n, w, wk, ldu, Xg, grp);
  __syncthreads();
  const int ta = (w + kUpdTile - 1) / kUpdTile, tq = (n + kUpdTile - 1) / kUpdTile;
  big_tiles<false>(
      [&](int t) {
        if (t < 2 * ta) {
          const int r = (t < ta ? t : t - ta) * kUpdTile;
          return BigTile{t < ta ? p.H : p.T, V, r, w - r};
        }
        const int u = t - 2 * ta, r = (u < tq ? u : u - tq) * kUpdTile;
        return BigTile{u < tq ? p.Q : p.Z, u < tq ? U : V, r, n - r};
      },
      2 * ta + 2 * tq, n, w, wk, ldu, Xg, grp);
  __syncthreads();
}
// slab tiles: behind the used part of the windows, or in the H and T windows
// (stored by then) of the larger ones
__device__ inline double* big_slab(const BigMem& m, int used) {
  return used + 2 * kBigSlab <= 4 * kBigWin ? m.win + used : m.win;
}
// with U at 2 wk ld: the largest window whose slab tiles do not fit behind is
// at least this wide, and H and T hold them
static_assert(4 * 70 * 71 + 2 * kBigSlab <= 4 * kBigWin && 2 * kBigSlab <= 2 * 70 * 71, "slab tiles");

// deflation scan: ktop, zeros on T's diagonal (k_scan)
__device__ inline void big_scan(const BigPencil& p, int ifirst, int kbot, BigShare* sh) {
  const int n = p.n;
  __syncthreads();
  if (threadIdx.x == 0) { sh->scan[0] = ifirst; sh->scan[1] = 0; sh->scan[2] = -1; sh->scan[3] = 0; }
  __syncthreads();
  for (int k = ifirst + (int)threadIdx.x; k <= kbot; k += kBigThreads) {
    const double* h = p.H + k + (size_t)k * n;
    const double a = h[0], b = p.T[k + (size_t)k * n], c = k > ifirst ? h[-n] : 0.0;
    if (!isfinite(a) || !isfinite(b) || !isfinite(c)) sh->scan[3] = 1;
    if (k > ifirst && negligible_sub(c, h[-n - 1], a, p.tol)) atomicMax(&sh->scan[0], k);
  }
  __syncthreads();
  const int ktop = sh->scan[0];
  if (threadIdx.x == 0 && ktop > ifirst) p.H[ktop + (size_t)(ktop - 1) * n] = 0.0;
  for (int k = ktop + (int)threadIdx.x; k <= kbot; k += kBigThreads) {
    double& t = p.T[k + (size_t)k * n];
    if (fabs(t) <= p.tol.ttol) {
      t = 0.0;
      atomicAdd(&sh->scan[1], 1);
      atomicMax(&sh->scan[2], k);
    }
  }
  __syncthreads();
}

// pair_shifts of qz_solver.h by one thread: polynomials of up to ns shifts
// from (sr, si, sb)[0..m), the lowest first
__device__ inline int big_pairs(const double* sr, const double* si, const double* sb, int m, int ns, double* poly) {
  int np = 0, jr = m - 1, jc = m - 1;  // next candidates, walking up
  auto is_pair = [&](int j) { return si[j] != 0.0 && j > 0 && si[j - 1] == -si[j]; };
  while (2 * np < ns) {
    // the lowest complex pair at or above jc
    while (jc >= 0 && !is_pair(jc)) --jc;
    // the two lowest real shifts at or above jr (skipping pairs)
    int r0 = jr;
    while (r0 >= 0 && si[r0] != 0.0) r0 -= is_pair(r0) ? 2 : 1;
    int r1 = r0 - 1;
    while (r1 >= 0 && si[r1] != 0.0) r1 -= is_pair(r1) ? 2 : 1;
    if (r1 < 0) r0 = -1;
    if (r0 < 0 && jc < 0) break;
    double c2, c1, c0;
    if (jc >= r0) {
      const int a = jc - 1;
      const double b = sb[a];
      c2 = b * b; c1 = 2.0 * sr[a] * b; c0 = sr[a] * sr[a] + si[a] * si[a];
      jc -= 2;
    } else {
      c2 = sb[r0] * sb[r1]; c1 = sr[r0] * sb[r1] + sr[r1] * sb[r0]; c0 = sr[r0] * sr[r1];
      jr = r1 - 1;
    }
    const double mx = fmax(fabs(c2), fmax(fabs(c1), fabs(c0)));
    if (!(mx > 0.0) || !isfinite(mx)) continue;
    poly[3 * np] = c2 / mx; poly[3 * np + 1] = c1 / mx; poly[3 * np + 2] = c0 / mx;
    ++np;
  }
  return np;
}

// The window phases are functions of their own, which take the shared memory
// by itself (not through pointers, whose accesses would be generic): inlined,
// the solve's state on top of theirs made it spill more of the 128 registers
// that 512 threads leave (220 pencils of order 32 to 300: 106 ms, 96 so).

// window QZ and early deflation of the loaded window of order n (k_aed_win),
// by the first kRoleThreads threads
static __device__ __noinline__ void big_aed(int n, Tol tol, double s, int nskip) {
  extern __shared__ double smem[];
  const BigMem m = big_mem(smem);
  const int ld = big_ld(n);
  BigExec x{(int)threadIdx.x, kRoleThreads, m.sh->si, m.sd};
  RoleBuf* const rb = (RoleBuf*)m.ring;
  WinState w;
  w.n = n;
  w.H = MatV{m.win, ld};
  w.T = MatV{m.win + n * ld, ld};
  w.Q = MatV{m.win + 2 * n * ld, ld};
  w.Z = MatV{m.win + 3 * n * ld, ld};
  w.wantq = w.wantz = true;
  w.tol = tol;
  const int qz = cta_role_qz(x, w, 30 * n, rb);
  if (qz == 0) cta_std_all(x, w, m.sd + 64);
  double* const sr = m.sh->shift;
  cta_aed_deflate(
      x, w, s, sr, sr + kBigShifts, sr + 2 * kBigShifts, qz,
      [&]() { return cta_role_spike(x, w, s, nskip, false, rb); },
      [&](int mm) { return cta_role_hessred(x, w, mm, rb); });
}

// chase of the loaded window of order wk (k_chase_win)
static __device__ __noinline__ bool big_chase(int wk, int last, int ld, int ldu, int nb, int tmax) {
  extern __shared__ double smem[];
  const BigMem m = big_mem(smem);
  return cta_chase_roles(wk, last, MatV{m.win, ld}, MatV{m.win + wk * ld, ld}, MatV{m.win + 2 * wk * ld, ldu},
                         MatV{m.win + wk * (2 * ld + ldu), ldu}, m.sh->bl, nb, tmax, m.ring, &m.sh->chase);
}

// The whole solve; 0, or the 1-based row where it stopped.
__device__ inline int big_solve(const BigPencil& p, double* smem, int maxit) {
  const BigMem m = big_mem(smem);
  BigShare* const sh = m.sh;
  const int tid = threadIdx.x, n = p.n;
  const int nw_aed = nw_table(n);
  int ifirst = 0, kbot = n - 1, stall = 0, last_kbot = -1, last_ktop = -1;
  for (int it = 0; it < maxit; ++it) {
    if (kbot < ifirst) return 0;
    big_scan(p, ifirst, kbot, sh);
    const int ktop = sh->scan[0], ninf = sh->scan[1], jlow = sh->scan[2];
    if (sh->scan[3]) return kbot + 1;
    if (kbot != last_kbot || ktop != last_ktop) stall = 0;
    else if (++stall > 300) return kbot + 1;
    last_kbot = kbot;
    last_ktop = ktop;
    if (ktop == kbot) { kbot -= 1; continue; }
    if (ninf > 0) {
      int jz = jlow;
      if (jz == ktop) {
        // rotation of rows f, f+1 (k_inf_top)
        const int f = ktop;
        double c, s, r;
        lartg(p.H[f + (size_t)f * n], p.H[f + 1 + (size_t)f * n], c, s, r);
        __syncthreads();
        for (int j = f + 1 + tid; j < n; j += kBigThreads) {
          rot_vec(c, s, p.H + f + (size_t)j * n, 1);
          rot_vec(c, s, p.T + f + (size_t)j * n, 1);
        }
        for (int i = tid; i < n; i += kBigThreads) rot_vec(c, s, p.Q + i + (size_t)f * n, n);
        if (tid == 0) { p.H[f + (size_t)f * n] = r; p.H[f + 1 + (size_t)f * n] = 0.0; }
        __syncthreads();
        continue;
      }
      for (;;) {
        const int w = ktop > jz - 1 ? ktop : jz - 1, wk = kbot - w + 1 < kBigChase ? kbot - w + 1 : kBigChase;
        const int stop = w + wk - 1, ld = big_ld(wk);
        double *Hs = m.win, *Ts = Hs + wk * ld, *Us = Ts + wk * ld, *Vs = Us + wk * ld;
        big_load(p, w, wk, Hs, Ts, Us, Vs, ld, ld);
        BigExecAll x{tid, kBigThreads, sh->si, m.sd};
        cta_inf_window(x, wk, ktop >= w ? ktop - w : -1, jz - w, stop - w, stop == kbot, MatV{Hs, ld}, MatV{Ts, ld},
                       MatV{Us, ld}, MatV{Vs, ld});
        big_store(p, w, wk, Hs, Ts, ld);
        big_update(p, w, wk, Us, Vs, ld, big_slab(m, 4 * wk * ld));
        if (stop == kbot) break;
        jz = stop;
      }
      kbot -= 1;
      continue;
    }
    const int nh = kbot - ktop + 1;
    const bool whole = nh <= kBigEnd;
    const int nw = whole ? nh : nw_aed, kwtop = kbot - nw + 1;
    // ---- AED, or the whole active block ----
    {
      const int ld = big_ld(nw);
      double *Hs = m.win, *Ts = Hs + nw * ld, *Us = Ts + nw * ld, *Vs = Us + nw * ld;
      big_load(p, kwtop, nw, Hs, Ts, Us, Vs, ld, ld);
      const double s = whole ? 0.0 : p.H[kwtop + (size_t)(kwtop - 1) * n];
      if (tid < kRoleThreads) big_aed(nw, p.tol, s, whole ? 0 : nskip_table(n));
      __syncthreads();
      const int mu = sh->si[8], status = sh->si[9], changed = sh->si[10];
      if (status == 0 && changed) {
        // (as k_aed_win stores it)
        if (!whole && tid == 0) p.H[kwtop + (size_t)(kwtop - 1) * n] = mu > 0 ? s * Us[0] : 0.0;
        big_store(p, kwtop, nw, Hs, Ts, ld);
        big_update(p, kwtop, nw, Us, Vs, ld, big_slab(m, 4 * nw * ld));
      }
      if (whole) {
        if (status != 0) return kbot + 1;
        kbot = ktop - 1;
        continue;
      }
      const int nd = status == 0 && changed ? nw - mu : 0;
      kbot -= nd;
      if (kbot < ktop) continue;
      if (status == 0 && 100 * nd > nibble_table(nh) * nw) continue;
      const int ns = min(ns_table(nh), mu - (mu & 1));
      if (tid == 0) {
        int np = ns >= 2 ? big_pairs(sh->shift, sh->shift + kBigShifts, sh->shift + 2 * kBigShifts, mu, ns, sh->poly) : 0;
        if (stall > 0 && stall % 40 == 0) {
          // no deflation for a while: exceptional shifts
          double mag = 0.0;
          for (int i = 0; i < mu; ++i)
            if (sh->shift[2 * kBigShifts + i] != 0.0)
              mag = fmax(mag, fabs(sh->shift[i] / sh->shift[2 * kBigShifts + i]));
          if (!(mag > 0.0) || !isfinite(mag)) mag = 1.0;
          for (int k = 0; k < np; ++k) {
            const double a = mag * sin(1.0 + 2.0 * k + 0.37 * stall), b = mag * cos(0.5 + 3.0 * k);
            const double mx = fmax(1.0, fmax(fabs(a + b), fabs(a * b)));
            sh->poly[3 * k] = 1.0 / mx; sh->poly[3 * k + 1] = (a + b) / mx; sh->poly[3 * k + 2] = a * b / mx;
          }
        }
        sh->npoly = np;
      }
      __syncthreads();
    }
    const int np = sh->npoly;
    if (np == 0 || kbot - ktop + 1 < 3) continue;
    // ---- sweep: chains of equal length, one after another (plan_chain) ----
    const int W = kBigChase, nchain = (np + kBigBulges - 1) / kBigBulges, each = (np + nchain - 1) / nchain;
    for (int p0 = 0; p0 < np; p0 += each) {
      const int nb = min(each, np - p0), adv = W - 4 - 3 * (nb - 1);
      int top = 0;  // row of the topmost bulge, the last one
      bool first = true;
      for (;;) {
        const int w = first ? ktop : top - 1, wk = min(W, kbot - w + 1);
        const bool fin = w + wk - 1 >= kbot;
        const int last = fin ? kbot - w : wk - 1;
        int tmax = 0;
        __syncthreads();
        for (int k = 0; k < nb; ++k) {
          // bulges stay three rows apart: bulge k is 3 (nb-1-k) rows below the last
          const int base = first ? -3 * k : top + 3 * (nb - 1 - k) - w;
          const int thi = fin ? (kbot - w) - base : first ? adv + 3 * nb - 2 : adv;
          tmax = max(tmax, thi);
          if (tid == k)
            sh->bl[k] = Bulge{base, first ? 3 * k : 0, thi, first ? 1 : 0, sh->poly[3 * (p0 + k)],
                              sh->poly[3 * (p0 + k) + 1], sh->poly[3 * (p0 + k) + 2]};
          if (k == nb - 1) top = w + base + thi;
        }
        // U, V: fragments of the updates on distinct banks
        const int ld = big_ld(wk), ldu = ((wk + 7) & ~7) + 4;
        double *Hs = m.win, *Ts = Hs + wk * ld, *Us = Ts + wk * ld, *Vs = Us + wk * ldu;
        big_load(p, w, wk, Hs, Ts, Us, Vs, ld, ldu);
        const bool ok = big_chase(wk, last, ld, ldu, nb, tmax);
        if (!ok) return kbot + 1;
        big_store(p, w, wk, Hs, Ts, ld);
        big_update(p, w, wk, Us, Vs, ldu, big_slab(m, 2 * wk * (ld + ldu)));
        if (fin) break;
        first = false;
      }
    }
  }
  return kbot + 1;
}

#endif

}  // namespace qz
