// Window QZ with a role per warp (device only, windows in shared memory).
//
// The double-shift sweeps of a window are a chain of dependent 3x3 steps;
// everything a step does outside its own block can lag behind.  Warp 0 (the
// core) runs the chain, the other warps follow it through a ring of posted
// transformations in shared memory:
//   core   per step s: the left rotations from the bulge column, applied to
//          rows s..s+2 of H and T (a lane per column), the right rotations
//          from rows s+1, s+2 of T, applied to rows s..s+3 of H and s..s+2 of
//          T (a lane per row).  What the next step's rotations depend on (the
//          bulge column, the 3x3 block of T) is carried in registers by every
//          lane, so no exchange between lanes lies on the dependent chain;
//   right  warps 1, 2: the right transformation on rows above s of H and T
//          (a thread per row);
//   Q, Z   warps 3, 5 and 6, 7: a thread per row of Q and Z.
// Warp 4 shares the core's scheduler and idles.  No barrier separates steps
// or sweeps: the followers poll the core's step count, and the core waits
// for the right warps once per sweep (before it reads rows they may still be
// writing) and for everybody only when the ring is full.  The deflation test
// reads the diagonals and the subdiagonal, which only the core writes, and so
// do the shifts of a block that ends where the last sweep ended (its final
// step leaves rows l-1 and l to the core), so both overlap with the tail of
// that sweep.  After a deflation at the bottom the block's last 2x2 lies
// higher, and its entries H(l-1, l) and T(l-1, l) are the right warps': the
// core waits for them before it forms the shift.
//
// Transformations are pairs of plane rotations formed with reciprocal
// square roots.  Left: (a1, a2) -> (rho, 0), then (a0, rho) -> (beta, 0); both
// roots are of sums of squares of the a's and run side by side.  Right: T is
// upper triangular before a step, so after the left rotations row s+2 of its
// block is (0, x1, x2) and row s+1 is (y0, y1, y2); the rotation of columns
// s+2, s+1 that clears x1, then of columns s+1, s that clears y0.  The second
// one's argument (x2 y1 - x1 y2, y0 |x|) is a polynomial in x and y up to the
// common factor |x|, so again both roots run side by side.  This is the RQ
// form, stable for every block; sums of squares outside a safe range take an
// out-of-line path with scaling, decided after the fast values are formed so
// that the test is off the chain.
//
// Bound: the dependent chain of a step, about 290 cycles by latency (FP64
// operation 10 cycles, reciprocal square root 50), and the core warp's issue
// slots (about 115 FP64 instructions of two cycles a step).  2x2 blocks are
// left general until the caller standardises the window in one pass
// (cta_std_all).
#pragma once
#include "qz_window.cuh"

namespace qz {

constexpr int kRoleThreads = 256;
constexpr int kRoleMax = 80;   // largest window
constexpr int kRoleRing = 64;  // posted steps kept (a power of two)
struct RoleBuf {
  // step: left c1, s1, c2, s2, right cb, sb, cc, sc, then as ints row s and
  // kind (3: rows and columns s..s+2, 2: s, s+1 with one rotation c1, s1 and
  // one cb, sb)
  double ring[kRoleRing][10];
  int ready, stop, err, code;
  int done[8];
  int arg[4];
};
constexpr int kRoleDoubles = (int)((sizeof(RoleBuf) + 15) / 16) * 2;
constexpr int kRoleSpin = 1 << 22;  // polls before a wait gives up

#ifdef __CUDACC__

__device__ __forceinline__ int role_ld(const int* p) {
  int v;
  asm volatile("ld.acquire.cta.shared.b32 %0, [%1];" : "=r"(v) : "r"((unsigned)__cvta_generic_to_shared(p)) : "memory");
  return v;
}
__device__ __forceinline__ void role_st(int* p, int v) {
  asm volatile("st.release.cta.shared.b32 [%0], %1;" ::"r"((unsigned)__cvta_generic_to_shared(p)), "r"(v) : "memory");
}

// Predicated shared-memory stores: the step's stores are by a few lanes each,
// and a branch around them (a divergence and a reconvergence) costs more
// than the stores.
__device__ __forceinline__ unsigned role_sm(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void role_put(bool on, unsigned a, double v) {
  asm volatile("{\n .reg .pred p;\n setp.ne.b32 p, %0, 0;\n @p st.shared.f64 [%1], %2;\n}" ::"r"((int)on), "r"(a), "d"(v)
               : "memory");
}
__device__ __forceinline__ void role_put3(bool on, unsigned a, unsigned st, double v0, double v1, double v2) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %0, 0;\n @p st.shared.f64 [%1], %4;\n @p st.shared.f64 [%2], %5;\n"
      " @p st.shared.f64 [%3], %6;\n}" ::"r"((int)on),
      "r"(a), "r"(a + st), "r"(a + 2 * st), "d"(v0), "d"(v1), "d"(v2)
      : "memory");
}
__device__ __forceinline__ void role_put8(bool on, unsigned a, double v0, double v1, double v2, double v3, double v4,
                                          double v5, double v6, double v7) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %0, 0;\n @p st.shared.v2.f64 [%1], {%2, %3};\n"
      " @p st.shared.v2.f64 [%1+16], {%4, %5};\n @p st.shared.v2.f64 [%1+32], {%6, %7};\n"
      " @p st.shared.v2.f64 [%1+48], {%8, %9};\n}" ::"r"((int)on),
      "r"(a), "d"(v0), "d"(v1), "d"(v2), "d"(v3), "d"(v4), "d"(v5), "d"(v6), "d"(v7)
      : "memory");
}
__device__ __forceinline__ void role_put_int2(bool on, unsigned a, int v0, int v1) {
  asm volatile("{\n .reg .pred p;\n setp.ne.b32 p, %0, 0;\n @p st.shared.v2.b32 [%1], {%2, %3};\n}" ::"r"((int)on), "r"(a),
               "r"(v0), "r"(v1)
               : "memory");
}
__device__ __forceinline__ void role_post(bool on, int* p, int v) {
  asm volatile("{\n .reg .pred p;\n setp.ne.b32 p, %0, 0;\n @p st.release.cta.shared.b32 [%1], %2;\n}" ::"r"((int)on),
               "r"(role_sm(p)), "r"(v)
               : "memory");
}

// 1/sqrt(x) for x in the normal range: the hardware's approximation and one
// third-order (Halley) correction y (1 + e/2 + 3 e^2/8), e = 1 - x y^2.
// Largest error measured over 1e-240..1e240: 1.25 units of rounding (2^-53),
// root mean square 0.47; rsqrt() has 1.01 and 0.42, sqrt and a division 1.50
// and 0.60.  49 cycles of latency against 83 of rsqrt().
__device__ __forceinline__ double role_rsqrt(double x) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  const double e = fma(-(x * y), y, 1.0);
  const double p = fma(e, 0.375, 0.5);
  return fma(p, e * y, y);
}

// 1/x, the approximation and two Newton steps (1.00 units of rounding); for
// scale factors of shifts and of reflectors
__device__ __forceinline__ double role_rcp(double x) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  double e = fma(-x, y, 1.0);
  y = fma(y, e, y);
  e = fma(-x, y, 1.0);
  return fma(y, e, y);
}

// Sums of squares outside about (1e-240, 1e240) take the scaled path; the
// test is on the exponent bits, so NaN and infinity fail it too.
__device__ __forceinline__ bool role_in_range(double q) {
  constexpr int lo = (1023 - 797) << 20, hi = (1023 + 797) << 20;
  return (unsigned)(__double2hiint(q) - lo) < (unsigned)(hi - lo);
}
constexpr double kRoleTiny = 1e-290;

// rotation taking (f, g) to (r, 0), r >= 0, any range
__device__ __forceinline__ void role_rot(double f, double g, double& c, double& s, double& r) {
  double q = f * f + g * g, sc = 1.0;
  if (!role_in_range(q)) {
    const double m = dmax(fabs(f), fabs(g));
    if (!(m > 0.0) || !isfinite(m)) { c = 1.0; s = 0.0; r = f; return; }
    f /= m; g /= m;
    sc = m;
    q = f * f + g * g;
  }
  const double inv = role_rsqrt(q);
  c = f * inv;
  s = g * inv;
  r = (q * inv) * sc;
}

struct RoleRot {
  double c1, s1, c2, s2, r;
};
// The left rotations of (a0, a1, a2) with scaling; r = beta.
__device__ __forceinline__ RoleRot role_left_scaled(double a0, double a1, double a2) {
  RoleRot o{1.0, 0.0, 1.0, 0.0, a0};
  const double m = dmax(fabs(a0), dmax(fabs(a1), fabs(a2)));
  if (!(m > 0.0) || !isfinite(m)) return o;
  a0 /= m; a1 /= m; a2 /= m;
  const double q23 = a1 * a1 + a2 * a2, q = a0 * a0 + q23;
  const bool z = !(q23 > kRoleTiny);  // |a1|, |a2| below 1e-145 of the largest
  const double r1 = role_rsqrt(z ? 1.0 : q23), r2 = role_rsqrt(q);
  o.c1 = z ? 1.0 : a1 * r1;
  o.s1 = z ? 0.0 : a2 * r1;
  o.c2 = a0 * r2;
  o.s2 = z ? 0.0 : (q23 * r1) * r2;
  o.r = (q * r2) * m;
  return o;
}
// The right rotations of rows (0, x1, x2), (y0, y1, y2) with scaling.
__device__ __forceinline__ RoleRot role_right_scaled(double x1, double x2, double y0, double y1, double y2) {
  RoleRot o;
  role_rot(x2, x1, o.c1, o.s1, o.r);
  double r;
  role_rot(o.c1 * y1 - o.s1 * y2, y0, o.c2, o.s2, r);
  return o;
}

__device__ __forceinline__ void role_apply_left(double c1, double s1, double c2, double s2, double& x0, double& x1,
                                                double& x2) {
  const double y1 = c1 * x1 + s1 * x2;
  x2 = c1 * x2 - s1 * x1;
  x1 = c2 * y1 - s2 * x0;
  x0 = c2 * x0 + s2 * y1;
}
// columns (s+2, s+1) by (cb, sb), then (s+1, s) by (cc, sc)
__device__ __forceinline__ void role_apply_right(double cb, double sb, double cc, double sc, double& x0, double& x1,
                                                 double& x2) {
  const double d = cb * x1 - sb * x2;
  x2 = cb * x2 + sb * x1;
  x1 = cc * d + sc * x0;
  x0 = cc * x0 - sc * d;
}

// wait until every flag of the mask (bit w: done[w]) is at least v (a vote
// orders no memory: the lanes that polled nothing get the pollers' acquire
// from the warp barrier)
__device__ __forceinline__ bool role_wait_done(RoleBuf* rb, unsigned mask, int v, int lane) {
  const bool mine = lane < 8 && ((mask >> lane) & 1);
  for (int it = 0; it < kRoleSpin; ++it) {
    const bool ok = !mine || role_ld(&rb->done[lane & 7]) >= v;
    if (__all_sync(0xffffffffu, ok)) {
      __syncwarp();
      return true;
    }
  }
  if (lane == 0) role_st(&rb->err, 1);
  __syncwarp();
  return false;
}
constexpr unsigned kRoleRight = 0x06, kRoleQ = 0x28, kRoleZ = 0xC0, kRoleAll = kRoleRight | kRoleQ | kRoleZ;

// The core's view of one window.
struct RoleCore {
  // A shift polynomial c2 M^2 - c1 M + c0, M = H T^{-1}, in units of H / ha =
  // H', T tb = T' (M' = M / (ha tb)), so that its coefficients do not leave
  // the range when H and T are far apart in magnitude.
  struct Shift {
    double c2, c1, c0, ha, tb;
  };
  WinState* w;
  RoleBuf* rb;
  int lane;
  int g = 0;      // steps posted since the start
  int seen = 0;   // steps everybody was last seen to have finished

  __device__ bool slot_free() {
    if (g - seen < kRoleRing) return true;
    if (!role_wait_done(rb, kRoleAll, g - kRoleRing / 2, lane)) return false;
    seen = g - kRoleRing / 2;
    return true;
  }

  // one sweep over the active block [f, l], l - f >= 2
  __device__ bool sweep(int f, int l, const Shift& p) {
    const int n = w->n, ld = w->H.ld;
    double* const Hb = w->H.p;
    double* const Tb = w->T.p;
    // the previous sweep's right transformations on rows of this one
    if (!role_wait_done(rb, kRoleRight, g, lane)) return false;
    double a0, a1, a2, t00, t01, t11;
    {
      const double* h = Hb + f + f * ld;
      const double* t = Tb + f + f * ld;
      t00 = t[0]; t01 = t[ld]; t11 = t[1 + ld];
      shift_vector(h[0], h[1], h[ld], h[1 + ld], h[2 + ld], t00, t01, t11, p, a0, a1, a2);
    }
    // the entries of step s, all moving one row and column a step: column
    // s + lane and s + 32 + lane, and the rows of the block (H rows s..s+3 on
    // lanes 0..3, T rows s..s+2 on lanes 4..6)
    const int diag = ld + 1, far = 32 * ld;
    const bool isT = lane >= 4;
    const int rr = isT ? lane - 4 : lane;
    double* rp = (isT ? Tb : Hb) + f + (lane < 7 ? rr : 0) + f * ld;
    double* dh = Hb + f + f * ld;  // H(s, s)
    double* dt = Tb + f + f * ld;  // T(s, s)
    // The left rotations of the first step; each step forms the next one's as
    // soon as it has the bulge column, ahead of its own stores.  (The added
    // constant stands in for a1 = a2 = 0 and is below 1e-24 of the largest
    // entry in range.)
    double c1, s1, c2, s2, beta, q23, q;
    auto left = [&]() {
      const double a1t = a1 + 1e-145;
      q23 = a1t * a1t + a2 * a2;
      q = a0 * a0 + q23;
      const double v1 = role_rsqrt(q23), v2 = role_rsqrt(q);
      c1 = a1t * v1; s1 = a2 * v1; c2 = a0 * v2; s2 = (q23 * v1) * v2; beta = q * v2;
    };
    left();
    for (int s = f; s < l - 1; ++s, rp += diag, dh += diag, dt += diag) {
      const int c = s + lane;
      const bool has = c < n, two = s + 32 < n, has2 = c + 32 < n;
      // a lane per column: rows s..s+2 of H and T (lanes without a column
      // read the block's first one); column s+2 of T for all
      const int o1 = has ? lane * ld : 0, o2 = has2 ? o1 + far : 0;
      double h0 = dh[o1], h1 = dh[o1 + 1], h2 = dh[o1 + 2], u0 = dt[o1], u1 = dt[o1 + 1], u2 = dt[o1 + 2];
      const double t02 = dt[2 * ld], t12 = dt[2 * ld + 1], t22 = dt[2 * ld + 2];
      double p0 = 0.0, p1 = 0.0, p2 = 0.0, w0 = 0.0, w1 = 0.0, w2 = 0.0;
      if (two) {
        p0 = dh[o2]; p1 = dh[o2 + 1]; p2 = dh[o2 + 2];
        w0 = dt[o2]; w1 = dt[o2 + 1]; w2 = dt[o2 + 2];
      }
      if (!(role_in_range(q) && q23 > 0.5 * kRoleTiny)) {
        const RoleRot o = role_left_scaled(a0, a1, a2);
        c1 = o.c1; s1 = o.s1; c2 = o.c2; s2 = o.s2; beta = o.r;
      }
      if (!slot_free()) return false;
      role_apply_left(c1, s1, c2, s2, h0, h1, h2);
      role_apply_left(c1, s1, c2, s2, u0, u1, u2);
      const unsigned ar = role_sm(rb->ring[g & (kRoleRing - 1)]);
      __syncwarp();
      role_put3(has, role_sm(dh + o1), 8, h0, h1, h2);
      role_put3(has, role_sm(dt + o1), 8, u0, u1, u2);
      role_put(s > f && lane < 3, role_sm(dh + (lane - ld)), lane == 0 ? beta : 0.0);
      __syncwarp();
      // rows s+1..s+3 of H for all (row l + 1 is outside the block), and the
      // lane's row
      const double* const hr = dh + 1;
      const bool in3 = s + 3 <= l, rowok = isT ? lane < 7 : s + lane <= l;
      const double g10 = hr[0], g11 = hr[ld], g12 = hr[2 * ld], g20 = hr[1], g21 = hr[1 + ld], g22 = hr[1 + 2 * ld];
      const double q30 = hr[2], q31 = hr[2 + ld], q32 = hr[2 + 2 * ld];  // past the window's last row: not used
      double r0 = rp[0], r1 = rp[ld], r2 = rp[2 * ld];
      // rows s+1, s+2 of T's block after the left rotations, and the right ones
      const double y0 = -s2 * t00, x1 = -s1 * t11, y1 = c2 * (c1 * t11) - s2 * t01;
      const double x2 = c1 * t22 - s1 * t12, y2 = c2 * (c1 * t12 + s1 * t22) - s2 * t02;
      const double qb = x1 * x1 + x2 * x2, dd = x2 * y1 - x1 * y2, qc = dd * dd + (y0 * y0) * qb;
      const double vb = role_rsqrt(qb), vc = role_rsqrt(qc);
      double cb = x2 * vb, sb = x1 * vb, cc = dd * vc, sc = (y0 * (qb * vb)) * vc;
      if (!(role_in_range(qb) && role_in_range(qc))) {
        const RoleRot z = role_right_scaled(x1, x2, y0, y1, y2);
        cb = z.c1; sb = z.s1; cc = z.c2; sc = z.s2;
      }
      role_put8(lane == 0, ar, c1, s1, c2, s2, cb, sb, cc, sc);
      role_put_int2(lane == 0, ar + 64, s, 3);
      if (two) {
        role_apply_left(c1, s1, c2, s2, p0, p1, p2);
        role_apply_left(c1, s1, c2, s2, w0, w1, w2);
        role_put3(has2, role_sm(dh + o2), 8, p0, p1, p2);
        role_put3(has2, role_sm(dt + o2), 8, w0, w1, w2);
        // columns from s + 64 on
        for (int k = c + 64; k < n; k += 32) {
          double* const hq = Hb + s + k * ld;
          double* const tq = Tb + s + k * ld;
          double b0 = hq[0], b1 = hq[1], b2 = hq[2], f0 = tq[0], f1 = tq[1], f2 = tq[2];
          role_apply_left(c1, s1, c2, s2, b0, b1, b2);
          role_apply_left(c1, s1, c2, s2, f0, f1, f2);
          hq[0] = b0; hq[1] = b1; hq[2] = b2;
          tq[0] = f0; tq[1] = f1; tq[2] = f2;
        }
      }
      // the next step's bulge column, block of T and left rotations
      a0 = cc * g10 - sc * (cb * g11 - sb * g12);
      a1 = cc * g20 - sc * (cb * g21 - sb * g22);
      a2 = cc * q30 - sc * (cb * q31 - sb * q32);
      a2 = in3 ? a2 : 0.0;
      left();
      t00 = cc * (cb * y1 - sb * y2) + sc * y0;
      t01 = cb * y2 + sb * y1;
      t11 = cb * x2 + sb * x1;
      role_apply_right(cb, sb, cc, sc, r0, r1, r2);
      r0 = isT && rr >= 1 ? 0.0 : r0;
      r1 = isT && rr >= 2 ? 0.0 : r1;
      __syncwarp();
      role_put3(rowok, role_sm(rp), 8 * ld, r0, r1, r2);
      ++g;
      __syncwarp();
      role_post(lane == 0, &rb->ready, g);
    }
    // final 2x2 step at rows and columns l-1, l
    const int s = l - 1;
    double c, sn, r;
    role_rot(a0, a1, c, sn, r);
    __syncwarp();
    if (lane < 2) Hb[s + lane + (s - 1) * ld] = lane == 0 ? r : 0.0;
    for (int cc = s + lane; cc < n; cc += 32) {
      double* hq = Hb + s + cc * ld;
      double* tq = Tb + s + cc * ld;
      const double u0 = hq[0], u1 = hq[1], v0 = tq[0], v1 = tq[1];
      hq[0] = c * u0 + sn * u1; hq[1] = c * u1 - sn * u0;
      tq[0] = c * v0 + sn * v1; tq[1] = c * v1 - sn * v0;
    }
    __syncwarp();
    double cz, sz, rz;
    role_rot(Tb[s + 1 + (s + 1) * ld], Tb[s + 1 + s * ld], cz, sz, rz);  // (col l, col l-1)
    // H rows l-1, l on lanes 0, 1, T's on lanes 2, 3
    double* const ep = (lane >= 2 ? Tb : Hb) + s + (lane & 1) + s * ld;
    const double p0 = ep[0], p1 = ep[ld];
    __syncwarp();
    if (lane < 4) {
      ep[ld] = cz * p1 + sz * p0;
      ep[0] = lane == 3 ? 0.0 : cz * p0 - sz * p1;
    }
    if (!slot_free()) return false;
    double* sl = rb->ring[g & (kRoleRing - 1)];
    if (lane == 0) {
      sl[0] = c; sl[1] = sn; sl[4] = cz; sl[5] = sz;
      ((int*)(sl + 8))[0] = s;
      ((int*)(sl + 8))[1] = 2;
    }
    __syncwarp();
    ++g;
    if (lane == 0) role_st(&rb->ready, g);
    return true;
  }

  // First column of the polynomial times t11^2 t22 (as shift_column, with H
  // and T scaled to about one by reciprocals and the result left unscaled:
  // only its direction is used).
  __device__ static void shift_vector(double h11, double h21, double h12, double h22, double h32, double t11,
                                      double t12, double t22, const Shift& p, double& v0, double& v1, double& v2) {
    const double hm = dmax(dmax(fabs(h11), fabs(h21)), dmax(dmax(fabs(h12), fabs(h22)), fabs(h32)));
    const double tm = dmax(fabs(t11), dmax(fabs(t12), fabs(t22)));
    if (!role_in_range(hm) || !role_in_range(tm)) {
      const double k = p.ha * p.tb;
      shift_column(h11, h21, h12, h22, h32, t11, t12, t22, p.c2, p.c1 * k, p.c0 * k * k, v0, v1, v2);
      return;
    }
    const double rh = role_rcp(hm), rt = role_rcp(tm), k = (p.ha * rh) * (p.tb * tm);
    h11 *= rh; h21 *= rh; h12 *= rh; h22 *= rh; h32 *= rh;
    t11 *= rt; t12 *= rt; t22 *= rt;
    const double c2 = p.c2, c1 = p.c1 * k, c0 = p.c0 * k * k;
    const double gg = h11 * t22 - t12 * h21, tt = t11 * t22;
    v0 = c2 * (h11 * gg + h12 * h21 * t11) - c1 * h11 * tt + c0 * t11 * tt;
    v1 = c2 * (h21 * gg + h22 * h21 * t11) - c1 * h21 * tt;
    v2 = c2 * h32 * h21 * t11;
  }
  // the characteristic polynomial of a 2x2 pencil (as pencil2_poly)
  __device__ static Shift shift_poly(double a00, double a10, double a01, double a11, double b00, double b01,
                                     double b11) {
    const double sa = dmax(dmax(fabs(a00), fabs(a10)), dmax(fabs(a01), fabs(a11)));
    const double sb = dmax(dmax(fabs(b00), fabs(b01)), fabs(b11));
    Shift p;
    if (!role_in_range(sa) || !role_in_range(sb)) {
      p.ha = p.tb = 1.0;
      pencil2_poly(a00, a10, a01, a11, b00, b01, b11, p.c2, p.c1, p.c0);
      return p;
    }
    const double ra = role_rcp(sa), rbb = role_rcp(sb);
    a00 *= ra; a10 *= ra; a01 *= ra; a11 *= ra;
    b00 *= rbb; b01 *= rbb; b11 *= rbb;
    p.ha = sa;
    p.tb = rbb;
    p.c2 = b00 * b11;
    p.c1 = a00 * b11 + a11 * b00 - a10 * b01;
    p.c0 = a00 * a11 - a01 * a10;
    return p;
  }

  // lowest row j in [lo, hi] whose test holds, or -1
  template <class F>
  __device__ int last_row(int hi, int lo, F test) {
    for (int base = hi; base >= lo; base -= 32) {
      const int j = base - lane;
      const unsigned m = __ballot_sync(0xffffffffu, j >= lo && test(j));
      if (m) return base - (__ffs(m) - 1);
    }
    return -1;
  }
};

// One line of a follower (a row of H, T, Q or Z): the entries of columns s
// and s+1 stay in registers from step to step of a sweep, so a step loads
// one entry and stores one; the sweep's last step stores both.
struct RoleLine {
  double x0, x1;
  bool on;  // x0, x1 hold columns s, s+1
};
template <bool kLeft>
__device__ __forceinline__ void role_line3(RoleLine& r, double* q, int ld, double a, double b, double c, double d) {
  double x0, x1, x2 = q[2 * ld];
  if (r.on) { x0 = r.x0; x1 = r.x1; }
  else { x0 = q[0]; x1 = q[ld]; }
  if (kLeft) role_apply_left(a, b, c, d, x0, x1, x2);
  else role_apply_right(a, b, c, d, x0, x1, x2);
  q[0] = x0;
  r.x0 = x1;
  r.x1 = x2;
  r.on = true;
}
template <bool kLeft>
__device__ __forceinline__ void role_line2(RoleLine& r, double* q, int ld, double c, double s) {
  const double x0 = r.on ? r.x0 : q[0], x1 = r.on ? r.x1 : q[ld];
  if (kLeft) { q[0] = c * x0 + s * x1; q[ld] = c * x1 - s * x0; }
  else { q[ld] = c * x1 + s * x0; q[0] = c * x0 - s * x1; }
  r.on = false;
}

// The followers of a sweep: apply posted steps until the core stops them.
__device__ inline void role_follow(WinState& w, RoleBuf* rb, int warp, int lane) {
  const unsigned bit = 1u << warp;
  const bool right = bit & kRoleRight, isq = bit & kRoleQ;
  const int half = (warp == 2 || warp == 5 || warp == 7) ? 32 : 0;
  const int id = half + lane, n = w.n, ld = w.H.ld;
  double* const P = right ? w.H.p : isq ? w.Q.p : w.Z.p;
  double* const P2 = w.T.p;
  constexpr int kLines = (kRoleMax + 63) / 64;
  RoleLine ln[kLines], lt[kLines];
#pragma unroll
  for (int k = 0; k < kLines; ++k) ln[k].on = lt[k].on = false;
  for (int g = 0;; ++g) {
    bool go = false;
    for (int it = 0; it < kRoleSpin; ++it) {
      if (role_ld(&rb->ready) > g) { go = true; break; }
      if (role_ld(&rb->stop) != 0) {
        go = role_ld(&rb->ready) > g;  // the steps posted before the stop
        break;
      }
    }
    // the end, or the wait gave up: cta_role_qz compares the counts
    if (!__any_sync(0xffffffffu, go)) return;
    __syncwarp();
    const double* sl = rb->ring[g & (kRoleRing - 1)];
    const int s = ((const int*)(sl + 8))[0];
    const bool three = ((const int*)(sl + 8))[1] == 3;
    const double* const k4 = isq ? sl : sl + 4;
    const double a = k4[0], b = k4[1], c = k4[2], d = k4[3];
    const int end = right ? s : n;
#pragma unroll
    for (int k = 0; k < kLines; ++k) {
      const int t = id + 64 * k;
      if (t < end) {
        double* const q = P + t + s * ld;
        if (isq) {
          if (three) role_line3<true>(ln[k], q, ld, a, b, c, d);
          else role_line2<true>(ln[k], q, ld, a, b);
        } else {
          if (three) role_line3<false>(ln[k], q, ld, a, b, c, d);
          else role_line2<false>(ln[k], q, ld, a, b);
          if (right) {
            double* const p = P2 + t + s * ld;
            if (three) role_line3<false>(lt[k], p, ld, a, b, c, d);
            else role_line2<false>(lt[k], p, ld, a, b);
          }
        }
      }
    }
    __syncwarp();
    if (lane == 0) role_st(&rb->done[warp], g + 1);
  }
}

// Window QZ of a window in shared memory by kRoleThreads threads: 0, or
// ilast+1 (at least 1) if it did not converge or a wait gave up.  The 2x2
// blocks stay general.
template <class X>
__device__ int cta_role_qz(X& x, WinState& w, int maxit, RoleBuf* rb) {
  const int n = w.n, ld = w.H.ld, lane = x.tid & 31, warp = x.tid >> 5;
  double* const Hb = w.H.p;
  double* const Tb = w.T.p;
  int ilast = n - 1, iiter = 0, jiter = 0;  // the core's
  for (;;) {
    if (x.tid == 0) { rb->ready = 0; rb->stop = 0; rb->err = 0; rb->code = 0; }
    if (x.tid < 8) rb->done[x.tid] = 0;
    x.sync();
    if (warp == 0) {
      RoleCore core{&w, rb, lane};
      int code = 0, a_if = 0, a_jz = -1;
      int lswept = -1;  // last row of the latest sweep
      while (ilast >= 0) {
        // deflation: negligible subdiagonal, then zeros on T's diagonal
        bool dead = false;
        const Tol tol = w.tol;
        int ifirst = core.last_row(ilast, 1, [&](int j) {
          const double tst = fabs(Hb[j - 1 + (j - 1) * ld]) + fabs(Hb[j + j * ld]);
          if (tst == 0.0) dead = true;
          return fabs(Hb[j + (j - 1) * ld]) <= dmax(tol.smlnum, tol.ulp * tst);
        });
        if (__any_sync(0xffffffffu, dead)) {
          // two zero diagonal entries: the test also reads H(j-1, j), which
          // the right warps write
          if (!role_wait_done(rb, kRoleRight, core.g, lane)) { code = 2; break; }
          ifirst = core.last_row(ilast, 1, [&](int j) {
            double tst = fabs(Hb[j - 1 + (j - 1) * ld]) + fabs(Hb[j + j * ld]);
            if (tst == 0.0) tst = fabs(Hb[j - 1 + j * ld]) + fabs(Hb[j + (j - 1) * ld]);
            return fabs(Hb[j + (j - 1) * ld]) <= dmax(tol.smlnum, tol.ulp * tst);
          });
        }
        if (ifirst < 0) ifirst = 0;
        else if (lane == 0) Hb[ifirst + (ifirst - 1) * ld] = 0.0;
        __syncwarp();
        const int jz = core.last_row(ilast, ifirst, [&](int j) { return fabs(Tb[j + j * ld]) <= tol.ttol; });
        if (ifirst == ilast) {
          if (jz >= 0 && lane == 0) Tb[jz + jz * ld] = 0.0;
          __syncwarp();
          ilast -= 1;
          iiter = 0;
          continue;
        }
        if (jz >= 0) {
          if (lane == 0) Tb[jz + jz * ld] = 0.0;
          __syncwarp();
          code = 1;
          a_if = ifirst;
          a_jz = jz;
          break;
        }
        if (ifirst + 1 == ilast) { ilast -= 2; iiter = 0; continue; }
        ++iiter;
        ++jiter;
        if (jiter > maxit) { code = 2; break; }
        const int l = ilast;
        if (l != lswept && !role_wait_done(rb, kRoleRight, core.g, lane)) { code = 2; break; }
        lswept = l;
        const double* h = Hb + (l - 1) + (l - 1) * ld;
        const double* t = Tb + (l - 1) + (l - 1) * ld;
        RoleCore::Shift p;
        if (iiter % 10 == 0) {
          // exceptional shift from the bottom subdiagonals
          const double sc = fabs(h[1] / t[0]) + fabs(h[-ld] / t[-1 - ld]);
          const double h11 = 0.75 * sc + h[1 + ld] / t[1 + ld];
          p = RoleCore::Shift{1.0, 2.0 * h11, h11 * h11 + 0.4375 * sc * sc, 1.0, 1.0};
        } else {
          p = RoleCore::shift_poly(h[0], h[1], h[ld], h[1 + ld], t[0], t[ld], t[1 + ld]);
        }
        if (lane == 0) x.count(0);
        if (!core.sweep(ifirst, l, p)) { code = 2; break; }
      }
      __syncwarp();
      if (lane == 0) {
        rb->code = code;
        rb->arg[0] = a_if; rb->arg[1] = a_jz; rb->arg[2] = ilast;
        role_st(&rb->stop, 1);
      }
    } else if (warp != 4) {
      role_follow(w, rb, warp, lane);
    }
    x.sync();
    const int code = rb->code, f = rb->arg[0], jz = rb->arg[1], il = rb->arg[2], err = rb->err;
    // a follower that gave up has not done every step; the core waits for the
    // Q and Z warps only when the ring is full, so it may not have noticed
    bool lost = false;
    for (int i = 0; i < 8; ++i)
      if ((kRoleAll >> i) & 1) lost = lost || rb->done[i] != rb->ready;
    x.sync();
    if (err != 0 || code == 2 || lost) return il >= 0 ? il + 1 : 1;
    if (code == 0) return 0;
    // a zero on T's diagonal: infinite eigenvalue, all threads
    if (jz == f) {
      cta_inf_top(x, w, f);
    } else {
      if (jz < il) cta_inf_chase_down(x, w, f, jz, il);
      cta_inf_bottom(x, w, il);
      ilast = il - 1;
    }
    iiter = 0;
  }
}

// ---------------------------------------------------------------------------
// Several block swaps at once (disjoint blocks): a thread forms each, the
// block applies their factors.
// ---------------------------------------------------------------------------
constexpr int kRoleSwap = 64;  // a swap's record: Q, Z, S2, T2 (16 each)
// one swap of blocks of sizes N1, N2 at window row j, by one thread, to rec
template <int N1, int N2>
__device__ __forceinline__ bool role_swap(double* S, double* T, int ld, int j, const Tol& tol, double* rec) {
  constexpr int M = N1 + N2;
  const MatV hb{S + j + j * ld, ld}, tb{T + j + j * ld, ld};
  double S2[M * M], T2[M * M], Qs[M * M], Zs[M * M];
  int res;
  if constexpr (N1 == 1 && N2 == 1)
    // two rotations; the Sylvester path where they fail the stability test
    res = swap_compute11(hb, tb, S2, T2, Qs, Zs, tol.ulp, tol.smlnum)
              ? 1
              : swap_compute_try<1, 1>(hb, tb, S2, T2, Qs, Zs, tol.ulp, tol.smlnum);
  else
    res = swap_compute_try<N1, N2>(hb, tb, S2, T2, Qs, Zs, tol.ulp, tol.smlnum);
  if (res > 0) {
#pragma unroll
    for (int i = 0; i < M * M; ++i) { rec[i] = Qs[i]; rec[16 + i] = Zs[i]; rec[32 + i] = S2[i]; rec[48 + i] = T2[i]; }
    return true;
  }
  return res < 0 && swap_retry<N1, N2>(hb, tb, rec + 32, rec + 48, rec, rec + 16, tol.ulp, tol.smlnum);
}

// y = F^T x (rows) or x F (columns) for the M entries at p, p + st, ..: the
// same sums, F = Q or Z
template <int M>
__device__ __forceinline__ void role_line(const double* f, double* p, int st) {
  double x[M];
#pragma unroll
  for (int i = 0; i < M; ++i) x[i] = p[i * st];
#pragma unroll
  for (int c = 0; c < M; ++c) {
    double a = 0.0;
#pragma unroll
    for (int k = 0; k < M; ++k) a += x[k] * f[k + M * c];
    p[c * st] = a;
  }
}
__device__ __forceinline__ void role_line_any(int m, const double* f, double* p, int st) {
  if (m == 2) role_line<2>(f, p, st);
  else if (m == 3) role_line<3>(f, p, st);
  else role_line<4>(f, p, st);
}


// The swaps sw[0..np) (row | size of the first block << 8 | of the second
// << 12) of one window, by all threads of a block: recs holds np records,
// good[k] tells whether swap k was applied.  Ends with a barrier.
template <class X>
__device__ void cta_role_swaps(X& x, const WinState& w, const int* sw, int np, double* recs, int* good) {
  const int tid = x.tid, warp = tid >> 5, lane = tid & 31, nw = x.nt >> 5, ld = w.H.ld, n = w.n;
  double *const Hs = w.H.p, *const Ts = w.T.p, *const Us = w.Q.p, *const Vs = w.Z.p;
  // a thread per swap, the four kinds on four warps
  if (warp < 4)
    for (int k = lane; k < np; k += 32) {
      const int e = sw[k], j = e & 255, n1 = (e >> 8) & 15, n2 = e >> 12;
      if (2 * (n1 - 1) + n2 - 1 != warp) continue;
      double* const rec = recs + k * kRoleSwap;
      if (warp == 0) good[k] = role_swap<1, 1>(Hs, Ts, ld, j, w.tol, rec);
      else if (warp == 1) good[k] = role_swap<1, 2>(Hs, Ts, ld, j, w.tol, rec);
      else if (warp == 2) good[k] = role_swap<2, 1>(Hs, Ts, ld, j, w.tol, rec);
      else good[k] = role_swap<2, 2>(Hs, Ts, ld, j, w.tol, rec);
    }
  x.sync();
  // left factors: rows of H, T right of the block; columns of Q
  for (int k = warp; k < np; k += nw) {
    if (!good[k]) continue;
    const int e = sw[k], j = e & 255, m = ((e >> 8) & 15) + (e >> 12);
    const double* const rec = recs + k * kRoleSwap;
    for (int c = j + m + lane; c < n; c += 32) {
      role_line_any(m, rec, Hs + j + c * ld, 1);
      role_line_any(m, rec, Ts + j + c * ld, 1);
    }
    for (int i = lane; i < n; i += 32) role_line_any(m, rec, Us + i + j * ld, ld);
  }
  x.sync();
  // right factors: columns of H, T above the block; columns of Z; the block
  for (int k = warp; k < np; k += nw) {
    if (!good[k]) continue;
    const int e = sw[k], j = e & 255, m = ((e >> 8) & 15) + (e >> 12);
    const double* const rec = recs + k * kRoleSwap;
    for (int i = lane; i < j; i += 32) {
      role_line_any(m, rec + 16, Hs + i + j * ld, ld);
      role_line_any(m, rec + 16, Ts + i + j * ld, ld);
    }
    for (int i = lane; i < n; i += 32) role_line_any(m, rec + 16, Vs + i + j * ld, ld);
    if (lane < m * m) {
      Hs[j + lane % m + (j + lane / m) * ld] = rec[32 + lane];
      Ts[j + lane % m + (j + lane / m) * ld] = rec[48 + lane];
    }
  }
  x.sync();
}

// ---------------------------------------------------------------------------
// Spike test with reordering (the loop of cta_aed_deflate) with the moves of
// undeflatable blocks overlapped.  A move's first swap settles the block that
// is tested next, so the next test and the next move start a round later and
// follow the earlier move up the window, two blocks behind; a round forms the
// swaps of all moves under way at once.  The same tests on the same blocks in
// the same order as one move after another; returns the last undeflated row.
// A rejected swap ends the test with the moves where they are.
// Bound: a swap's serial computation per round; a window of 48 takes about 26
// rounds instead of 88 swaps in sequence when the test stops after four
// undeflatable blocks.
// ---------------------------------------------------------------------------
constexpr int kRoleMoves = kRoleDoubles / kRoleSwap;  // records in the role buffer
template <class X>
__device__ int cta_role_spike(X& x, WinState& w, double s, int nskip, bool swapfail, RoleBuf* rb) {
  const int n = w.n;
  double* const recs = (double*)rb;
  int* const sw = x.si + 16;              // swaps of the round
  int* const good = sw + kRoleMoves;
  int* const ctl = good + kRoleMoves;     // swaps, last row
  // thread 0's: moves under way, in order
  int pos[kRoleMoves], size[kRoleMoves], goal[kRoleMoves], act = 0;
  int who[kRoleMoves];
  int kb = n - 1, ilst = 0, fails = 0;
  bool stop = false;
  for (;;) {
    int np = 0;
    if (x.tid == 0) {
      // settled blocks at the bottom
      while (!stop && act < kRoleMoves) {
        if (kb < ilst || (nskip > 0 && fails >= nskip)) { stop = true; break; }
        const int free0 = act ? pos[act - 1] + size[act - 1] : 0;
        if (kb < free0) break;
        const bool bulge = (kb > ilst) && (w.H(kb, kb - 1) != 0.0);
        const int nb = bulge ? 2 : 1, at = kb - nb + 1;
        if (at < free0) break;
        bool dfl;
        if (!bulge) {
          const double temp = fabs(s) + fabs(w.H(kb, kb));
          dfl = fabs(s * w.Q(0, kb)) <= dmax(w.tol.ulp * temp, w.tol.smlnum);
        } else {
          const double h11 = w.H(kb - 1, kb - 1), h21 = w.H(kb, kb - 1), h12 = w.H(kb - 1, kb), h22 = w.H(kb, kb);
          double rtdet;
          if (h11 == 0.0 && h21 == 0.0) rtdet = 0.0;
          else if (fabs(h11) >= fabs(h21)) rtdet = sqrt(fabs(h11)) * sqrt(fabs(h22 - (h21 / h11) * h12));
          else rtdet = sqrt(fabs(h21)) * sqrt(fabs(h12 - (h11 / h21) * h22));
          const double temp = fabs(s) + rtdet;
          dfl = dmax(fabs(s * w.Q(0, kb)), fabs(s * w.Q(0, kb - 1))) <= dmax(w.tol.ulp * temp, w.tol.smlnum);
        }
        if (dfl) { kb -= nb; fails = 0; continue; }
        if (swapfail) { stop = true; act = 0; break; }
        if (at > ilst) {
          pos[act] = at;
          size[act] = nb;
          goal[act] = ilst;
          ++act;
        }
        ilst += nb;
        ++fails;
      }
      for (int i = 0; i < act; ++i) {
        const int nbn = (pos[i] - 2 >= goal[i] && w.H(pos[i] - 1, pos[i] - 2) != 0.0) ? 2 : 1, lo = pos[i] - nbn;
        if (i > 0 && lo < pos[i - 1] + size[i - 1]) continue;
        sw[np] = lo | nbn << 8 | size[i] << 12;
        who[np++] = i;
      }
      ctl[0] = np;
      ctl[1] = kb;
    }
    x.sync();
    np = ctl[0];
    if (np == 0) break;
    cta_role_swaps(x, w, sw, np, recs, good);
    if (x.tid == 0) {
      for (int k = 0; k < np; ++k) {
        x.count(1);
        const int i = who[k];
        if (!good[k]) { stop = true; act = 0; break; }
        pos[i] = sw[k] & 255;
        // the moved block must keep its size (a complex pair stays 2x2)
        if (size[i] == 2 && w.H(pos[i] + 1, pos[i]) == 0.0) { stop = true; act = 0; break; }
      }
      int keep = 0;
      for (int i = 0; i < act; ++i)
        if (pos[i] > goal[i]) { pos[keep] = pos[i]; size[keep] = size[i]; goal[keep] = goal[i]; ++keep; }
      act = keep;
    }
  }
  kb = ctl[1];
  x.sync();
  return kb;
}

// ---------------------------------------------------------------------------
// Hessenberg-triangular re-reduction of the leading m x m block (the job of
// cta_hessred, the same rotations up to signs) by kRoleThreads threads.
//
// Per column jc, all row rotations at once, then the column rotations:
//   1. the rotations that clear column jc from the bottom are quotients of
//      suffix norms, so one warp scan of squares gives all of them;
//   2. they are applied to the columns of H and T and the rows of Q as walks,
//      a thread per walk, which leaves T upper Hessenberg;
//   3. warp 0 clears T's subdiagonal from the bottom (a lane per row; the
//      row of the pair hands its two entries to all lanes, which form the
//      rotation), posting each rotation; the other warps follow it along the
//      rows of H and Z.
// Three barriers a column instead of one per pair.  Bound: the chain of part
// 3, about 125 cycles a pair (shuffle, sum of squares, reciprocal square
// root, update).  Returns false if a wait gave up.
// ---------------------------------------------------------------------------
template <class X>
__device__ bool cta_role_hessred(X& x, WinState& w, int m, RoleBuf* rb) {
  const int n = w.n, ld = w.H.ld, lane = x.tid & 31, warp = x.tid >> 5;
  double* const Hb = w.H.p;
  double* const Tb = w.T.p;
  double2* const gr = (double2*)rb->ring;  // row rotation of pair jr
  double2* const zr = gr + kRoleMax;       // column rotation
  constexpr int kB = (kRoleMax + 31) / 32;
  constexpr unsigned kF = 0xffffffffu;
  if (x.tid == 0) { rb->ready = 0; rb->err = 0; }
  for (int jc = 0; jc < m - 2; ++jc) {
    if (warp == 0) {
      // element k (from the bottom) is row m-1-k of the column
      const int L = m - 1 - jc;
      double a[kB], q[kB], sc = 1.0;
#pragma unroll
      for (int b = 0; b < kB; ++b) {
        const int k = lane + 32 * b;
        a[b] = k < L ? Hb[m - 1 - k + jc * ld] : 0.0;
      }
      for (int pass = 0;; ++pass) {
        double carry = 0.0;
#pragma unroll
        for (int b = 0; b < kB; ++b) {
          double t = a[b] * a[b];
#pragma unroll
          for (int o = 1; o < 32; o <<= 1) {
            const double u = __shfl_up_sync(kF, t, o);
            if (lane >= o) t += u;
          }
          q[b] = t + carry;
          carry = __shfl_sync(kF, q[b], 31);
        }
        if (pass || role_in_range(carry)) break;
        double mx = 0.0;
#pragma unroll
        for (int b = 0; b < kB; ++b) mx = dmax(mx, fabs(a[b]));
        for (int o = 16; o; o >>= 1) mx = dmax(mx, __shfl_xor_sync(kF, mx, o));
        if (!(mx > 0.0) || !isfinite(mx)) break;  // a zero column: identity rotations
        sc = mx;
#pragma unroll
        for (int b = 0; b < kB; ++b) a[b] /= mx;
      }
      double below = 0.0;  // norm of the elements below this lane's first
#pragma unroll
      for (int b = 0; b < kB; ++b) {
        const int k = lane + 32 * b;
        const bool z = !(q[b] > kRoleTiny);
        const double inv = role_rsqrt(z ? 1.0 : q[b]);
        double rho = z ? 0.0 : q[b] * inv;
        if (k == 0) rho = a[0];  // the bottom entry keeps its sign
        double prev = __shfl_up_sync(kF, rho, 1);
        if (lane == 0) prev = below;
        below = __shfl_sync(kF, rho, 31);
        if (k >= 1 && k < L) gr[m - k] = z ? make_double2(1.0, 0.0) : make_double2(a[b] * inv, prev * inv);
        if (k < L) Hb[m - 1 - k + jc * ld] = k == L - 1 ? rho * sc : 0.0;
      }
    }
    x.sync();
    // 2. rows jr-1, jr of H, T and columns jr-1, jr of Q
    const int nc = n - 1 - jc;
    for (int it = x.tid; it < 2 * nc + n; it += x.nt) {
      double* p;
      int st = 1, jhi = m - 1;
      if (it < nc) {
        p = Hb + (jc + 1 + it) * ld;
      } else if (it < 2 * nc) {
        const int c = jc + 1 + it - nc;
        p = Tb + c * ld;
        jhi = c + 1 < m - 1 ? c + 1 : m - 1;  // below its diagonal the column is zero
      } else {
        p = w.Q.p + (it - 2 * nc);
        st = ld;
      }
      double y = p[jhi * st];
      for (int j = jhi; j >= jc + 2; --j) {
        const double2 g = gr[j];
        const double v = p[(j - 1) * st];
        p[j * st] = g.x * y - g.y * v;
        y = g.x * v + g.y * y;
      }
      p[(jc + 1) * st] = y;
    }
    x.sync();
    // 3. columns jr, jr-1: T on warp 0, H and Z behind it
    const int base = rb->ready;  // pairs posted by the columns before (nobody posts here)
    x.sync();
    if (warp == 0) {
      double v[kB], y[kB];
#pragma unroll
      for (int b = 0; b < kB; ++b) {
        const int i = lane + 32 * b;
        v[b] = i < m ? Tb[i + (m - 1) * ld] : 0.0;
        y[b] = i < m ? Tb[i + (m - 2) * ld] : 0.0;
      }
      for (int jr = m - 1; jr >= jc + 2; --jr) {
        // the pair's own row: its diagonal and subdiagonal entries
        const int ob = jr >> 5, ol = jr & 31;
        double f = v[0], g = y[0];
#pragma unroll
        for (int b = 1; b < kB; ++b)
          if (ob == b) { f = v[b]; g = y[b]; }
        f = __shfl_sync(kF, f, ol);
        g = __shfl_sync(kF, g, ol);
        double yn[kB];
#pragma unroll
        for (int b = 0; b < kB; ++b) {
          const int i = lane + 32 * b;
          yn[b] = (jr >= 2 && i < m) ? Tb[i + (jr - 2) * ld] : 0.0;
        }
        double c, s, r;
        role_rot(f, g, c, s, r);
        if (lane == 0) zr[jr] = make_double2(c, s);
#pragma unroll
        for (int b = 0; b < kB; ++b) {
          const int i = lane + 32 * b;
          if (i <= jr) Tb[i + jr * ld] = i == jr ? r : c * v[b] + s * y[b];
          if (i == jr) Tb[i + (jr - 1) * ld] = 0.0;
          v[b] = c * y[b] - s * v[b];
          y[b] = yn[b];
        }
        __syncwarp();
        if (lane == 0) {
          x.count(2);
          role_st(&rb->ready, base + m - jr);
        }
      }
#pragma unroll
      for (int b = 0; b < kB; ++b) {
        const int i = lane + 32 * b;
        if (i <= jc + 1) Tb[i + (jc + 1) * ld] = v[b];
      }
    } else {
      const int it = x.tid - 32;
      const bool on = it < m + n;
      double* const p = it < m ? Hb + it : w.Z.p + (on ? it - m : 0);
      double v = on ? p[(m - 1) * ld] : 0.0;
      int avail = base;
      bool ok = true;
      for (int jr = m - 1; jr >= jc + 2 && ok; --jr) {
        const double y = on ? p[(jr - 1) * ld] : 0.0;
        if (avail < base + m - jr) {
          ok = false;
          for (int k = 0; k < kRoleSpin; ++k) {
            avail = role_ld(&rb->ready);
            if (avail >= base + m - jr) { ok = true; break; }
          }
          ok = __all_sync(kF, ok);
          avail = __shfl_sync(kF, avail, 0);
          __syncwarp();
        }
        const double2 z = zr[jr];
        if (on) p[jr * ld] = z.x * v + z.y * y;
        v = z.x * y - z.y * v;
      }
      if (on) p[(jc + 1) * ld] = v;
      if (!ok && lane == 0) role_st(&rb->err, 1);
    }
    x.sync();
  }
  x.sync();
  return rb->err == 0;
}

#endif  // __CUDACC__

}  // namespace qz
