// The flag loads, flag stores and predicated stores of qz_roles.cuh for the
// host block emulation (PTX there).
#pragma once
#include "warp_emu.h"

#include "qz_window.cuh"

namespace qz {
inline int role_ld(const int* p) { return emu::polled(p); }
inline void role_st(int* p, int v) {
  *(volatile int*)p = v;
  emu::posted();
}
inline unsigned role_sm(const void* p) { return (unsigned)((const char*)p - emu::block()->arena); }
inline double* emu_at(unsigned a) { return (double*)(emu::block()->arena + a); }
inline void role_put(bool on, unsigned a, double v) {
  if (on) *emu_at(a) = v;
}
inline void role_put3(bool on, unsigned a, unsigned st, double v0, double v1, double v2) {
  if (!on) return;
  *emu_at(a) = v0;
  *emu_at(a + st) = v1;
  *emu_at(a + 2 * st) = v2;
}
inline void role_put8(bool on, unsigned a, double v0, double v1, double v2, double v3, double v4, double v5, double v6,
                      double v7) {
  const double v[8] = {v0, v1, v2, v3, v4, v5, v6, v7};
  if (on) memcpy(emu_at(a), v, sizeof v);
}
inline void role_put_int2(bool on, unsigned a, int v0, int v1) {
  const int v[2] = {v0, v1};
  if (on) memcpy(emu_at(a), v, sizeof v);
}
inline void role_post(bool on, int* p, int v) {
  if (on) role_st(p, v);
}
inline double role_rsqrt(double x) { return 1.0 / sqrt(x); }
inline double role_rcp(double x) { return 1.0 / x; }
}  // namespace qz
