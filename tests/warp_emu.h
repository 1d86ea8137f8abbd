// Device code of a thread block on one host thread: a fiber per CUDA thread.
//
// Warp collectives and block barriers are rendezvous of the fibers; flags in
// "shared memory" are plain loads and stores, at which a fiber may be
// switched out.  The order in which warps run is chosen by the test: every
// warp in turn, or chosen warps only when no other can get on.  Code that
// waits for what it reads gives the same bits under any order.
#pragma once
#include <setjmp.h>
#include <ucontext.h>

#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <map>
#include <vector>

namespace emu {

constexpr int kLanes = 32;
struct Fiber {
  ucontext_t ctx;        // where it begins
  jmp_buf at;            // where it goes on
  bool begun = false;
  bool done = false;
  bool waiting = false;  // at a rendezvous
  int bar = 0;           // the named barrier, if it is one
  uint64_t slot = 0;     // its contribution to a collective
};
struct Warp {
  std::vector<uint64_t> vals = std::vector<uint64_t>(kLanes);
  int arrived = 0;
  long spins = 0;  // polls since the warp last saw a flag change or set one
  const void* flag = nullptr;  // its latest poll
  int value = 0;
};

struct Block {
  std::vector<Fiber> f;
  std::vector<Warp> w;
  jmp_buf home;
  int cur = 0, barrier = 0, named[16] = {};
  unsigned slow = 0;  // warps that run only when the others are stuck
  std::function<void(int)> body;
  char* arena = nullptr;  // "shared memory" (base of 32-bit addresses)
  // With ordered set: the largest value of every flag that each thread's later
  // reads are ordered behind, by a poll of its own or by a warp barrier after
  // another lane's (a vote hands nothing over).
  bool ordered = false;
  std::vector<std::map<const void*, int>> seen;
};
inline Block*& block() {
  static Block* b = nullptr;
  return b;
}
// (jumps between stacks; contexts are for the first entry alone, as they save
// the signal mask by a system call)
__attribute__((noinline)) inline void yield() {
  Block& b = *block();
  if (_setjmp(b.f[b.cur].at) == 0) _longjmp(b.home, 1);
}
__attribute__((noinline)) inline void enter(Block& b, Fiber& x) {
  if (_setjmp(b.home) != 0) return;
  if (x.begun) _longjmp(x.at, 1);
  x.begun = true;
  setcontext(&x.ctx);
}
inline int lane_id() { return block()->cur % kLanes; }

// all lanes of the warp meet; returns the values they brought
inline const std::vector<uint64_t>& meet(uint64_t v) {
  Block& b = *block();
  const int me = b.cur;
  Warp& w = b.w[me / kLanes];
  b.f[me].slot = v;
  b.f[me].waiting = true;
  if (++w.arrived == kLanes) {
    w.arrived = 0;
    const int base = me / kLanes * kLanes;
    for (int i = 0; i < kLanes; ++i) {
      w.vals[i] = b.f[base + i].slot;
      b.f[base + i].waiting = false;
    }
    return w.vals;  // (nobody overwrites them before every lane has gone on to the next meeting)
  }
  while (b.f[me].waiting) yield();
  return w.vals;
}
inline void block_barrier() {
  Block& b = *block();
  const int me = b.cur, total = (int)b.f.size();
  b.f[me].waiting = true;
  b.w[me / kLanes].spins = 0;
  if (++b.barrier == total) {
    b.barrier = 0;
    for (Fiber& x : b.f) x.waiting = false;
    return;
  }
  while (b.f[me].waiting) yield();
}
// a barrier of `count` of the threads (bar.sync id, count)
inline void named_barrier(int id, int count) {
  Block& b = *block();
  const int me = b.cur;
  b.f[me].waiting = true;
  b.f[me].bar = id;
  b.w[me / kLanes].spins = 0;
  if (++b.named[id] == count) {
    b.named[id] = 0;
    for (Fiber& x : b.f)
      if (x.waiting && x.bar == id) {
        x.waiting = false;
        x.bar = 0;
      }
    return;
  }
  while (b.f[me].waiting) yield();
}
// a poll of a flag: the warp may be switched out
inline int polled(const int* p) {
  yield();
  Warp& w = block()->w[block()->cur / kLanes];
  const int v = *(const volatile int*)p;
  if (w.flag == p && w.value != v) w.spins = 0;
  w.flag = p;
  w.value = v;
  ++w.spins;
  if (block()->ordered) {
    int& s = block()->seen[block()->cur][p];
    s = s > v ? s : v;
  }
  return v;
}
inline void posted() {
  Block& b = *block();
  b.w[b.cur / kLanes].spins = 0;
}

inline void entry(unsigned lo, unsigned hi) {
  Block* b = (Block*)(((uintptr_t)hi << 32) | lo);
  const int me = b->cur;
  b->body(me);
  b->f[me].done = true;
  for (;;) yield();
}

// the fibers' stacks, kept from block to block
constexpr size_t kStack = 256 << 10;
inline char* stack(int i) {
  static std::vector<char*> pool;
  while ((int)pool.size() <= i) pool.push_back((char*)malloc(kStack));
  return pool[i];
}

// one turn of a warp: every lane that can run, until all have met or polled;
// true if some lane was not just waiting
inline bool turn(Block& b, int warp) {
  bool ran = false;
  for (int l = 0; l < kLanes; ++l) {
    Fiber& x = b.f[warp * kLanes + l];
    if (x.done || x.waiting) continue;
    ran = true;
    b.cur = warp * kLanes + l;
    enter(b, x);
  }
  return ran;
}

inline void run(int threads, unsigned slow, char* arena, const std::function<void(int)>& body, bool ordered = false) {
  Block b;
  b.ordered = ordered;
  b.seen.resize(threads);
  b.f = std::vector<Fiber>(threads);
  b.w = std::vector<Warp>(threads / kLanes);
  b.slow = slow;
  b.body = body;
  b.arena = arena;
  block() = &b;
  for (int i = 0; i < threads; ++i) {
    ucontext_t& c = b.f[i].ctx;
    getcontext(&c);
    c.uc_stack.ss_sp = stack(i);
    c.uc_stack.ss_size = kStack;
    c.uc_link = nullptr;
    makecontext(&c, (void (*)())entry, 2, (unsigned)(uintptr_t)&b, (unsigned)((uintptr_t)&b >> 32));
  }
  const int warps = (int)b.w.size();
  constexpr long kStuck = 8 * kLanes;  // polls in a row after which a warp counts as stuck
  for (;;) {
    bool left = false, on = false;
    for (Fiber& x : b.f) left = left || !x.done;
    if (!left) break;
    for (int w = 0; w < warps; ++w)
      if (!(slow >> w & 1)) on = (turn(b, w) && b.w[w].spins < kStuck) || on;
    if (on) continue;
    // nobody else gets on: the slow warps take a turn
    for (int w = 0; w < warps; ++w)
      if (slow >> w & 1) turn(b, w);
  }
  block() = nullptr;
}

}  // namespace emu

// ---- the CUDA names the code uses ----
#define __device__
#define __host__
#define __forceinline__ inline
#define __noinline__
struct double2 {
  double x, y;
};
struct int2 {
  int x, y;
};
inline double2 make_double2(double x, double y) { return double2{x, y}; }
inline int2 make_int2(int x, int y) { return int2{x, y}; }
inline uint64_t emu_bits(double v) {
  uint64_t u;
  memcpy(&u, &v, 8);
  return u;
}
inline double emu_double(uint64_t u) {
  double v;
  memcpy(&v, &u, 8);
  return v;
}
struct EmuThreadIndex {
  struct X {
    operator int() const { return emu::block()->cur; }
  } x;
};
static const EmuThreadIndex threadIdx{};
struct EmuIndex {
  int x = 0;
};
inline EmuIndex& emu_block_index() {
  static EmuIndex i;
  return i;
}
inline EmuIndex& emu_grid_size() {
  static EmuIndex i;
  return i;
}
inline EmuIndex& emu_block_size() {
  static EmuIndex i;
  return i;
}
inline void __syncthreads() { emu::block_barrier(); }
inline void __syncwarp() {
  emu::meet(0);
  emu::Block& b = *emu::block();
  if (!b.ordered) return;
  const int base = b.cur / emu::kLanes * emu::kLanes;
  for (int i = base; i < base + emu::kLanes; ++i)
    for (const auto& s : b.seen[i]) {
      int& mine = b.seen[b.cur][s.first];
      mine = mine > s.second ? mine : s.second;
    }
}
inline unsigned __ballot_sync(unsigned, bool p) {
  const auto& v = emu::meet(p);
  unsigned m = 0;
  for (int i = 0; i < emu::kLanes; ++i) m |= (unsigned)(v[i] & 1) << i;
  return m;
}
inline bool __all_sync(unsigned m, bool p) { return __ballot_sync(m, p) == 0xffffffffu; }
inline bool __any_sync(unsigned m, bool p) { return __ballot_sync(m, p) != 0; }
inline double __shfl_sync(unsigned, double v, int src) { return emu_double(emu::meet(emu_bits(v))[src & 31]); }
inline int __shfl_sync(unsigned, int v, int src) { return (int)(uint32_t)emu::meet((uint32_t)v)[src & 31]; }
inline double __shfl_up_sync(unsigned, double v, int d) {
  const int l = emu::lane_id();
  return emu_double(emu::meet(emu_bits(v))[l >= d ? l - d : l]);
}
inline double __shfl_xor_sync(unsigned, double v, int d) { return emu_double(emu::meet(emu_bits(v))[emu::lane_id() ^ d]); }
inline int __ffs(unsigned v) { return __builtin_ffs((int)v); }
inline int __double2hiint(double v) { return (int)(emu_bits(v) >> 32); }
inline int __double2loint(double v) { return (int)emu_bits(v); }
inline double __hiloint2double(int hi, int lo) { return emu_double((uint64_t)(uint32_t)hi << 32 | (uint32_t)lo); }
inline int atomicExch(int* p, int v) {
  const int old = *p;
  *p = v;
  return old;
}
