// Chase of a chain of bulges through a window in shared memory (device):
// the transformations of cta_chase_window (qz_chase.cuh) in its lockstep
// order, with the work split for one SM:
//   * lane b of the coefficient warp forms the reflectors of bulge b's step
//     (the opposite one needs only the bulge's 3x3 block of T, which the lane
//     transforms itself) and posts them in a ring;
//   * the chase warps, a bulge each at a time, apply the left reflectors to
//     the columns of H and T, then the right ones to the rows;
//   * the factor warps apply the reflectors to U and V, which nobody reads
//     before the end, a step or more behind.
// A step has three parts with a barrier after each: the left reflectors are
// formed (the chase warps load their columns meanwhile); they are applied
// while the opposite reflectors are formed; those are applied.
// The reflectors come from reciprocal square roots and reciprocals, and the
// null vector of the opposite reflector from a product form that is stable
// for every block, where a cross product needs a branch to an RQ
// factorisation for nearly parallel rows (one block in ten, which held up
// the whole lockstep step).
#pragma once
#include "qz_roles.cuh"

namespace qz {

constexpr int kChaseWarps = 8;                         // chase warps (bulges at a time)
constexpr int kChaseMain = 32 * (kChaseWarps + 1);     // threads of the chase barrier (and the coefficient warp)
constexpr int kChaseFactor = 128;                      // factor threads (a row of U or V each at a time)
// Warp w runs on scheduler w mod 4: the coefficient warp has the first to
// itself (three warps idle), the chase warps two, the factor warps the
// last, so that each scheduler's instruction cache holds one role's code.
constexpr int kChaseRoleThreads = 512;
constexpr int kChaseSlots = 4;                         // steps in the ring
constexpr int kChaseRecDoubles = 10;                   // L, R, (kind, row), new H(row, row-1)

// per-launch shared state behind the window matrices
struct ChaseShare {
  int posted, err;
  int stop;  // written by the coefficient warp between barriers of the chase threads
  int done[kChaseFactor / 32];
};
constexpr size_t chase_ring_doubles(int nb) { return (size_t)kChaseSlots * nb * kChaseRecDoubles; }

#ifdef __CUDACC__

// The rare forms are out of line: the step's code has to stay in the
// schedulers' instruction caches (fetches were a third of its stalls).
struct ChaseHouse {
  House3 h;
  double beta;
};
static __device__ __noinline__ ChaseHouse chase_house_any(double x0, double x1, double x2) {
  ChaseHouse o;
  house3(x0, x1, x2, o.h, o.beta);
  return o;
}
static __device__ __noinline__ House3 chase_opposite_any(double y0, double y1, double y2, double x0, double x1,
                                                         double x2) {
  const double m[9] = {0.0, y0, x0, 0.0, y1, x1, 0.0, y2, x2};
  double tau, v1, v2;
  opposite_reflector3(m, tau, v1, v2);
  return House3{tau, 1.0, v1, v2};
}
struct ChaseVec {
  double v0, v1, v2;
};
static __device__ __noinline__ ChaseVec chase_intro(const double* h, const double* t, int ld, double c2, double c1,
                                                    double c0) {
  ChaseVec o;
  shift_column(h[0], h[1], h[ld], h[1 + ld], h[2 + ld], t[0], t[ld], t[1 + ld], c2, c1, c0, o.v0, o.v1, o.v2);
  return o;
}

static __device__ __noinline__ ChaseVec chase_rot_any(double f, double g) {
  ChaseVec o;
  lartg(f, g, o.v0, o.v1, o.v2);
  return o;
}
static __device__ __noinline__ void chase_rot_lines(double c, double s, double* p, double* q, int step, int st,
                                                    int count) {
  for (int i = 0; i < count; ++i) {
    rot_vec(c, s, p, st);
    rot_vec(c, s, q, st);
    p += step;
    q += step;
  }
}

// house3 with a reciprocal square root and a reciprocal (in range; the
// scaled form elsewhere).  s = 2 / u^T u is formed from the stored u, so the
// reflector is orthogonal to rounding whatever the accuracy of the norm.
__device__ __forceinline__ void chase_house(double x0, double x1, double x2, House3& h, double& beta) {
  const double q1 = x1 * x1 + x2 * x2, q = x0 * x0 + q1;
  const double nrm = q * role_rsqrt(q);
  const double b = -copysign(nrm, x0);
  const double u0 = x0 - b, uu = u0 * u0 + q1;
  h.s = 2.0 * role_rcp(uu);
  h.u0 = u0; h.u1 = x1; h.u2 = x2;
  beta = b;
  // q1 = 0: the identity, as house3 has it
  if (!role_in_range(q) || !(q1 > kRoleTiny)) {
    const ChaseHouse o = chase_house_any(x0, x1, x2);
    h = o.h;
    beta = o.beta;
  }
}

// The opposite reflector of a block with rows 1 and 2 (y0, y1, y2) and
// (x0, x1, x2): its first column spans their null space.  Rotating row 2 to
// (0, 0, *) and row 1 to (0, *, *) gives the null vector as the first column
// of the rotations' product; with the square roots multiplied out it is
//   w = (D x1 - B x2 x0, -(D x0 + B x2 x1), B (x0^2 + x1^2)),
//   B = x1 y0 - x0 y1,  D = x2 (x0 y0 + x1 y1) - (x0^2 + x1^2) y2,
// the cross product times x0^2 + x1^2, but with residuals on both rows of a
// few rounding errors of the rows for any block: given D and B every
// component is accurate relative to |w|, and their own errors leave row 2
// orthogonal to w and turn w within row 1's plane by a rounding error.
__device__ __forceinline__ void chase_opposite(double y0, double y1, double y2, double x0, double x1, double x2,
                                               House3& h) {
  const double qa = x0 * x0 + x1 * x1, dot = x0 * y0 + x1 * y1, bb = x1 * y0 - x0 * y1;
  const double dd = x2 * dot - qa * y2, t = bb * x2;
  const double w0 = dd * x1 - t * x0, w1 = -(dd * x0 + t * x1), w2 = bb * qa;
  const double ww = w0 * w0 + w1 * w1 + w2 * w2;
  if (role_in_range(ww)) {
    double beta;
    chase_house(w0, w1, w2, h, beta);
  } else {
    h = chase_opposite_any(y0, y1, y2, x0, x1, x2);  // row 2 already (0, 0, *), parallel rows, or out of range
  }
}

// entries of a bulge's reflector in the ring, a: 0 left, 4 right
__device__ __forceinline__ House3 chase_rec(const double* r, int a) {
  const double2 u = *(const double2*)(r + a), v = *(const double2*)(r + a + 2);
  return House3{u.x, u.y, v.x, v.y};
}
__device__ __forceinline__ void chase_bar() { asm volatile("bar.sync 1, %0;" ::"n"(kChaseMain) : "memory"); }

// One lane's view of its bulge's step at window row j: the left reflector and
// the 3x3 block of T (c, s and a 2x2 block in the terminal step).
struct ChaseLane {
  House3 L;
  double b00, b10, b20, b01, b11, b21, b02, b12, b22;
};
// Part one: the left reflector, to the ring entry r.
__device__ __forceinline__ void chase_coef_left(const double* Hp, const double* Tp, int ld, int j, int last,
                                                const Bulge& g, bool intro, double* r, ChaseLane& e) {
  const double* const h = Hp + j + j * ld;  // H(j, j)
  const double* const t = Tp + j + j * ld;
  double2* const r2 = (double2*)r;
  double beta = 0.0;
  if (j + 2 <= last) {
    double a0, a1, a2;
    if (intro) {
      const ChaseVec v = chase_intro(h, t, ld, g.c2, g.c1, g.c0);
      a0 = v.v0; a1 = v.v1; a2 = v.v2;
    } else {
      a0 = h[-ld]; a1 = h[1 - ld]; a2 = h[2 - ld];
    }
    e.b00 = t[0]; e.b10 = t[1]; e.b20 = t[2];
    e.b01 = t[ld]; e.b11 = t[1 + ld]; e.b21 = t[2 + ld];
    e.b02 = t[2 * ld]; e.b12 = t[1 + 2 * ld]; e.b22 = t[2 + 2 * ld];
    chase_house(a0, a1, a2, e.L, beta);
    r2[1] = make_double2(e.L.u1, e.L.u2);
  } else {
    const ChaseVec v = chase_rot_any(h[-ld], h[1 - ld]);
    e.b10 = t[1]; e.b11 = t[1 + ld]; e.b00 = t[0]; e.b01 = t[ld];
    e.L.s = v.v0;
    e.L.u0 = v.v1;
    beta = v.v2;
  }
  r2[0] = make_double2(e.L.s, e.L.u0);
  r[9] = beta;
}
// Part two: the opposite reflector.
__device__ __forceinline__ void chase_coef_right(int j, int last, double* r, ChaseLane& e) {
  double2* const r2 = (double2*)r;
  if (j + 2 <= last) {
    House3 R;
    house3_apply(e.L, e.b00, e.b10, e.b20);
    house3_apply(e.L, e.b01, e.b11, e.b21);
    house3_apply(e.L, e.b02, e.b12, e.b22);
    chase_opposite(e.b10, e.b11, e.b12, e.b20, e.b21, e.b22, R);
    r2[2] = make_double2(R.s, R.u0);
    r2[3] = make_double2(R.u1, R.u2);
    *(int2*)(r + 8) = make_int2(1, j);
  } else {
    rot2(e.L.s, e.L.u0, e.b00, e.b10);
    rot2(e.L.s, e.L.u0, e.b01, e.b11);
    const ChaseVec v = chase_rot_any(e.b11, -e.b10);  // opposite_rot2
    r2[2] = make_double2(v.v0, v.v1);
    *(int2*)(r + 8) = make_int2(2, j);
  }
}

// A chase warp's two lines of H and of T per lane (columns j + lane, + 32
// for the left reflector, rows lane, + 32 for the right one); lanes without a
// line read the first one and store nothing.
struct ChasePair {
  double a0, a1, a2, b0, b1, b2, c0, c1, c2, d0, d1, d2;
  unsigned ah, at, ch, ct;
  bool on0, on1;
};
__device__ __forceinline__ void chase_pair_load(ChasePair& v, const double* Hp, const double* Tp, int o0, int o1,
                                                int st) {
  const double *h0 = Hp + o0, *t0 = Tp + o0, *h1 = Hp + o1, *t1 = Tp + o1;
  v.a0 = h0[0]; v.a1 = h0[st]; v.a2 = h0[2 * st];
  v.b0 = t0[0]; v.b1 = t0[st]; v.b2 = t0[2 * st];
  v.c0 = h1[0]; v.c1 = h1[st]; v.c2 = h1[2 * st];
  v.d0 = t1[0]; v.d1 = t1[st]; v.d2 = t1[2 * st];
  v.ah = role_sm(h0); v.at = role_sm(t0); v.ch = role_sm(h1); v.ct = role_sm(t1);
}
__device__ __forceinline__ void chase_pair_apply(ChasePair& v, const House3& e, int st, bool ot0, bool ot1, bool z0,
                                                 bool z1) {
  house3_apply(e, v.a0, v.a1, v.a2);
  house3_apply(e, v.b0, v.b1, v.b2);
  house3_apply(e, v.c0, v.c1, v.c2);
  house3_apply(e, v.d0, v.d1, v.d2);
  role_put3(v.on0, v.ah, 8 * st, v.a0, v.a1, v.a2);
  role_put3(ot0, v.at, 8 * st, z0 ? 0.0 : v.b0, v.b1, v.b2);
  role_put3(v.on1, v.ch, 8 * st, v.c0, v.c1, v.c2);
  role_put3(ot1, v.ct, 8 * st, z1 ? 0.0 : v.d0, v.d1, v.d2);
}
__device__ __forceinline__ void chase_left_load(ChasePair& v, const double* Hp, const double* Tp, int ld, int wk,
                                                int j, int c) {
  v.on0 = c < wk;
  v.on1 = c + 32 < wk;
  chase_pair_load(v, Hp, Tp, j + (v.on0 ? c : j) * ld, j + (v.on1 ? c + 32 : j) * ld, 1);
}

// Left reflector of one bulge (ring entry r) on columns j.. of H and T, by
// one warp; v: the first two lines of each lane, loaded.
__device__ __forceinline__ void chase_left(double* Hp, double* Tp, int ld, int wk, int j, int last, bool intro,
                                           const double* r, ChasePair& v, int lane) {
  if (j + 2 <= last) {
    const House3 L = chase_rec(r, 0);
    role_put(!intro && lane < 3, role_sm(Hp + j + lane + (j - 1) * ld), lane == 0 ? r[9] : 0.0);
    chase_pair_apply(v, L, 1, v.on0, v.on1, false, false);
    for (int c = j + lane + 64; c - lane < wk; c += 64) {
      chase_left_load(v, Hp, Tp, ld, wk, j, c);
      chase_pair_apply(v, L, 1, v.on0, v.on1, false, false);
    }
  } else {
    const int o = j + (j + lane) * ld;
    chase_rot_lines(r[0], r[1], Hp + o, Tp + o, 32 * ld, 1, (wk - j - lane + 31) >> 5);
    role_put(lane < 2, role_sm(Hp + j + lane + (j - 1) * ld), lane == 0 ? r[9] : 0.0);
  }
}

// Right reflector: rows of H down to j+3 (or the last) and of T down to j+2.
__device__ __forceinline__ void chase_right(double* Hp, double* Tp, int ld, int j, int last, const double* r,
                                            int lane) {
  if (j + 2 <= last) {
    const House3 R = chase_rec(r, 4);
    const int hr = j + 4 < last + 1 ? j + 4 : last + 1;
    for (int t = lane; t - lane < hr; t += 64) {
      ChasePair v;
      v.on0 = t < hr;
      v.on1 = t + 32 < hr;
      const int t0 = v.on0 ? t : 0, t1 = v.on1 ? t + 32 : 0;
      chase_pair_load(v, Hp, Tp, t0 + j * ld, t1 + j * ld, ld);
      // the block's rows j+1, j+2 of T: column j is zero now
      chase_pair_apply(v, R, ld, v.on0 && t0 < j + 3, v.on1 && t1 < j + 3, t0 > j, t1 > j);
    }
  } else {
    const int o = lane + j * ld;
    chase_rot_lines(r[4], r[5], Hp + o, Tp + o, 32, ld, (last + 32 - lane) >> 5);
    role_put(lane == ((j + 1) & 31), role_sm(Tp + j + 1 + j * ld), 0.0);
  }
}

// bulges kChaseWarps, .. of a longer chain
static __device__ __noinline__ void chase_left_rest(double* Hp, double* Tp, int ld, int wk, int last, const Bulge* bl,
                                                    int nb, int tau, const double* recs, int warp, int lane) {
  for (int b = warp + kChaseWarps; b < nb; b += kChaseWarps) {
    const int j = bl[b].base + tau;
    if (tau < bl[b].tlo || tau >= bl[b].thi) continue;
    ChasePair v;
    chase_left_load(v, Hp, Tp, ld, wk, j, j + lane);
    chase_left(Hp, Tp, ld, wk, j, last, bl[b].intro && tau == bl[b].tlo, recs + b * kChaseRecDoubles, v, lane);
  }
}
static __device__ __noinline__ void chase_right_rest(double* Hp, double* Tp, int ld, int last, const Bulge* bl, int nb,
                                                     int tau, const double* recs, int warp, int lane) {
  for (int b = warp + kChaseWarps; b < nb; b += kChaseWarps)
    if (tau >= bl[b].tlo && tau < bl[b].thi)
      chase_right(Hp, Tp, ld, bl[b].base + tau, last, recs + b * kChaseRecDoubles, lane);
}

// The window's chase by kChaseRoleThreads threads; false: a wait gave up.
// ring: chase_ring_doubles(nb) doubles, 16-byte aligned.
__device__ inline bool cta_chase_roles(int wk, int last, MatV H, MatV T, MatV U, MatV V, const Bulge* bl, int nb,
                                       int tmax, double* ring, ChaseShare* sh) {
  const int tid = threadIdx.x, lane = tid & 31, ld = H.ld;
  auto rec = [&](int tau, int b) { return ring + ((tau & (kChaseSlots - 1)) * nb + b) * kChaseRecDoubles; };
  if (tid == 0) { sh->posted = 0; sh->err = 0; sh->stop = 0; }
  if (tid < kChaseFactor / 32) sh->done[tid] = 0;
  __syncthreads();
  const int wid = tid >> 5, col = wid & 3;
  if (col == 0 && wid != 0) {
    // idle
  } else if (col != 3) {
    const int warp = col == 0 ? -1 : 2 * (wid >> 2) + col - 1;
    // the lane's bulge (coefficient warp) or the warp's first one
    const int own = warp < 0 ? lane : warp;
    Bulge mine{};
    mine.tlo = tmax;  // none: never active
    if (own < nb) mine = bl[own];
    double* const Hp = H.p;
    double* const Tp = T.p;
    for (int tau = 0; tau < tmax; ++tau) {
      const int j = mine.base + tau;
      const bool on = tau >= mine.tlo && tau < mine.thi, intro = mine.intro && tau == mine.tlo;
      if (warp < 0) {
        ChaseLane e;
        double* const r = rec(tau, lane < nb ? lane : 0);
        if (on) chase_coef_left(Hp, Tp, ld, j, last, mine, intro, r, e);
        chase_bar();
        if (on) chase_coef_right(j, last, r, e);
        else if (lane < nb) *(int2*)(r + 8) = make_int2(0, 0);
        chase_bar();
        if (lane == 0) role_st(&sh->posted, tau + 1);
        if (tau + 1 >= kChaseSlots) {
          // the next step's ring entries have been applied to U and V
          const int need = tau + 2 - kChaseSlots;
          bool ok = false;
          for (int it = 0; it < kRoleSpin && !ok; ++it)
            ok = __all_sync(0xffffffffu, lane >= kChaseFactor / 32 ||
                                             role_ld(&sh->done[lane < kChaseFactor / 32 ? lane : 0]) >= need);
          __syncwarp();
          if (lane == 0 && (!ok || role_ld(&sh->err) != 0)) { role_st(&sh->err, 1); sh->stop = 1; }
        }
        chase_bar();
      } else {
        ChasePair v;
        if (on) chase_left_load(v, Hp, Tp, ld, wk, j, j + lane);
        chase_bar();
        if (on) chase_left(Hp, Tp, ld, wk, j, last, intro, rec(tau, warp), v, lane);
        if (nb > kChaseWarps) chase_left_rest(Hp, Tp, ld, wk, last, bl, nb, tau, rec(tau, 0), warp, lane);
        chase_bar();
        if (on) chase_right(Hp, Tp, ld, j, last, rec(tau, warp), lane);
        if (nb > kChaseWarps) chase_right_rest(Hp, Tp, ld, last, bl, nb, tau, rec(tau, 0), warp, lane);
        chase_bar();
      }
      if (sh->stop != 0) break;
    }
  } else {
    const int warp = wid >> 2, f = 32 * warp + lane, ldf = U.ld;
    for (int tau = 0; tau < tmax; ++tau) {
      bool ok = false;
      for (int it = 0; it < kRoleSpin; ++it) {
        if (role_ld(&sh->posted) > tau) { ok = true; break; }
        if (role_ld(&sh->err) != 0) break;
      }
      if (!__all_sync(0xffffffffu, ok)) {
        if (lane == 0) role_st(&sh->err, 1);
        break;
      }
      __syncwarp();
      for (int it = f; it < 2 * wk; it += kChaseFactor) {
        const bool u = it < wk;
        double* const row = u ? U.p + it : V.p + it - wk;
        const int off = u ? 0 : 4;
        // the bulges of one step touch disjoint columns: four at a time
        for (int b0 = 0; b0 < nb; b0 += 4) {
          double x0[4], x1[4], x2[4];
          House3 h[4];
          int2 kj[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const double* r = rec(tau, b0 + i < nb ? b0 + i : b0);
            kj[i] = *(const int2*)(r + 8);
            if (b0 + i >= nb) kj[i].x = 0;
            h[i] = chase_rec(r, off);
            const double* q = row + (kj[i].x == 1 ? kj[i].y : 0) * ldf;
            x0[i] = q[0]; x1[i] = q[ldf]; x2[i] = q[2 * ldf];
          }
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            house3_apply(h[i], x0[i], x1[i], x2[i]);
            role_put3(kj[i].x == 1, role_sm(row + kj[i].y * ldf), 8 * ldf, x0[i], x1[i], x2[i]);
            if (kj[i].x == 2) rot_vec(h[i].s, h[i].u0, row + kj[i].y * ldf, ldf);
          }
        }
      }
      __syncwarp();
      if (lane == 0) role_st(&sh->done[warp], tau + 1);
    }
  }
  __syncthreads();
  return sh->err == 0;
}

#endif  // __CUDACC__

}  // namespace qz
