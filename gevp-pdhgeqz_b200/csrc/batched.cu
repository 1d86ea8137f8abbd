// Batched QZ of many independent small pencils of uneven sizes.
//
// Role in the reference: none directly (PDHGEQZ solves one pencil); this is
// the batched workload of the measurement plan, built from the same
// CTA-level kernels as the endgame (PDHGEQZ4 -> KKQZ): every pencil is
// reduced to generalized Schur form with Q and Z by one CTA.
//
// CTAs pull pencils from an atomic queue ordered by decreasing size
// (longest-first scheduling).  Two persistent launches: pencils of order up to
// kBatchSmemMax are solved in shared memory (H, T, Q, Z with an odd leading
// dimension) by the window QZ with a role per warp (qz_roles.cuh: 600 pencils
// of order 16..80 in 7.0 ms, 33.5 with the two-barrier sweeps); larger ones,
// which come first, by a CTA each that runs the whole windowed iteration
// (batch_big.cuh), as a sweep that touches global memory at every step costs
// several times the windows and their updates.  With 128 threads (an
// autotuned or chosen configuration) one launch solves all by small-bulge
// multishift sweeps (cta_small_qz_ms), in place in global memory above
// smem_max.  beta >= 0, eigenvalues and per-pencil status words at the end;
// no host round trip.
#include <cuda_runtime.h>
#include <float.h>
#include <stdint.h>

#include <algorithm>
#include <mutex>

#include "../../include/b200qz.h"
#include "batch_big.cuh"
#include "kernels.h"
#include "qz_roles.cuh"

namespace qz {

namespace {

struct BExec {
  int tid, nt;
  int* si;
  double* sd;
  __device__ void sync() { __syncthreads(); }
  __device__ void stamp(int) {}
  __device__ void count(int) {}
};

__device__ __forceinline__ double block_sum(double v, double* red) {
  for (int off = 16; off > 0; off >>= 1) v += __shfl_down_sync(0xffffffffu, v, off);
  int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  __syncthreads();
  if (lane == 0) red[wid] = v;
  __syncthreads();
  double t = 0.0;
  if (threadIdx.x == 0)
    for (int i = 0; i < (int)(blockDim.x >> 5); ++i) t += red[i];
  __syncthreads();
  if (threadIdx.x == 0) red[0] = t;
  __syncthreads();
  return red[0];
}

}  // namespace

__global__ void __launch_bounds__(kBatchThreads, 1) k_batch_qz(int count, const int* __restrict__ order,
                                                            const int* __restrict__ nsz,
                                                            const int64_t* __restrict__ moff,
                                                            const int64_t* __restrict__ eoff, double* H, double* T,
                                                            double* Q, double* Z, double* AR, double* AI, double* BE,
                                                            int* status, int* counter, int smem_max) {
  extern __shared__ double smem[];
  __shared__ int s_next;
  __shared__ double red[32];
  __shared__ int si[64];
  __shared__ double sd_small[64];
  __shared__ double ms_scr[kMsScratch];  // multishift window QZ scratch
  for (;;) {
    if (threadIdx.x == 0) s_next = atomicAdd(counter, 1);
    __syncthreads();
    const int idx = s_next;
    __syncthreads();
    if (idx >= count) break;
    const int p = order[idx];
    const int n = nsz[p];
    double* Hg = H + moff[p];
    double* Tg = T + moff[p];
    double* Qg = Q + moff[p];
    double* Zg = Z + moff[p];
    // tolerances of this pencil (PDHGEQZ.f:449-458)
    double hs = 0.0, ts = 0.0;
    for (int k = threadIdx.x; k < n * n; k += blockDim.x) {
      hs += Hg[k] * Hg[k];
      ts += Tg[k] * Tg[k];
    }
    hs = block_sum(hs, red);
    ts = block_sum(ts, red);
    Tol tol;
    tol.safmin = DBL_MIN;
    tol.ulp = DBL_EPSILON;
    tol.smlnum = DBL_MIN * ((double)n / DBL_EPSILON);
    tol.htol = fmax(DBL_MIN, DBL_EPSILON * sqrt(hs));
    tol.ttol = fmax(DBL_MIN, DBL_EPSILON * sqrt(ts));
    const bool in_smem = n <= smem_max;
    const int lw = in_smem ? smem_ld(n) : n;
    double *Hs, *Ts, *Qs, *Zs;
    if (in_smem) {
      Hs = smem;
      Ts = Hs + n * lw;
      Qs = Ts + n * lw;
      Zs = Qs + n * lw;
      for (int k = threadIdx.x; k < n * n; k += blockDim.x) {
        int i = k % n, j = k / n;
        Hs[i + j * lw] = Hg[k];
        Ts[i + j * lw] = Tg[k];
        Qs[i + j * lw] = (i == j) ? 1.0 : 0.0;
        Zs[i + j * lw] = (i == j) ? 1.0 : 0.0;
      }
    } else {
      Hs = Hg;
      Ts = Tg;
      Qs = Qg;
      Zs = Zg;
      for (int k = threadIdx.x; k < n * n; k += blockDim.x) {
        int i = k % n, j = k / n;
        Qs[k] = (i == j) ? 1.0 : 0.0;
        Zs[k] = (i == j) ? 1.0 : 0.0;
      }
    }
    __syncthreads();
    // role-per-warp QZ: its buffer and scratch behind the matrices
    const bool roles = in_smem && blockDim.x == kRoleThreads;
    RoleBuf* const rb = (RoleBuf*)(smem + 4 * smem_max * smem_ld(smem_max));
    BExec x{(int)threadIdx.x, (int)blockDim.x, si, roles ? (double*)(rb + 1) : sd_small};
    WinState w;
    w.n = n;
    w.H = MatV{Hs, lw};
    w.T = MatV{Ts, lw};
    w.Q = MatV{Qs, lw};
    w.Z = MatV{Zs, lw};
    w.wantq = true;
    w.wantz = true;
    w.tol = tol;
    int info;
    if (roles) {
      w.H.p = smem;  // (shared-memory accesses throughout)
      w.T.p = smem + n * lw;
      w.Q.p = smem + 2 * n * lw;
      w.Z.p = smem + 3 * n * lw;
      info = cta_role_qz(x, w, 30 * n, rb);
      if (info == 0) cta_std_all(x, w, x.sd);
    } else {
      info = cta_small_qz_ms(x, w, 30 * n, ms_scr);
    }
    __syncthreads();
    if (info == 0) cta_finalize(x, w, AR + eoff[p], AI + eoff[p], BE + eoff[p]);
    if (in_smem) {
      for (int k = threadIdx.x; k < n * n; k += blockDim.x) {
        int i = k % n, j = k / n;
        Hg[k] = Hs[i + j * lw];
        Tg[k] = Ts[i + j * lw];
        Qg[k] = Qs[i + j * lw];
        Zg[k] = Zs[i + j * lw];
      }
    }
    if (threadIdx.x == 0) status[p] = info;
    __syncthreads();
  }
}

// Pencils above kBatchSmemMax, one CTA each from the same kind of queue.
__global__ void __launch_bounds__(kBigThreads, 1) k_batch_big(int count, const int* __restrict__ order,
                                                              const int* __restrict__ nsz,
                                                              const int64_t* __restrict__ moff,
                                                              const int64_t* __restrict__ eoff, double* H, double* T,
                                                              double* Q, double* Z, double* AR, double* AI,
                                                              double* BE, int* status, int* counter) {
  extern __shared__ double smem[];
  __shared__ int s_next;
  __shared__ double red[32];
  __shared__ int si[64];
  for (;;) {
    if (threadIdx.x == 0) s_next = atomicAdd(counter, 1);
    __syncthreads();
    const int idx = s_next;
    __syncthreads();
    if (idx >= count) break;
    const int q = order[idx];
    BigPencil p{H + moff[q], T + moff[q], Q + moff[q], Z + moff[q], nsz[q], {}};
    const int n = p.n;
    double hs = 0.0, ts = 0.0;
    for (int j = threadIdx.x >> 5; j < n; j += kBigThreads / 32)
      for (int i = threadIdx.x & 31; i < n; i += 32) {
        const size_t k = i + (size_t)j * n;
        hs += p.H[k] * p.H[k];
        ts += p.T[k] * p.T[k];
        p.Q[k] = p.Z[k] = i == j ? 1.0 : 0.0;
      }
    hs = block_sum(hs, red);
    ts = block_sum(ts, red);
    p.tol.safmin = DBL_MIN;
    p.tol.ulp = DBL_EPSILON;
    p.tol.smlnum = DBL_MIN * ((double)n / DBL_EPSILON);
    p.tol.htol = fmax(DBL_MIN, DBL_EPSILON * sqrt(hs));
    p.tol.ttol = fmax(DBL_MIN, DBL_EPSILON * sqrt(ts));
    const int info = big_solve(p, smem, 30 * n);
    __syncthreads();
    if (info == 0) {
      BigExecAll x{(int)threadIdx.x, kBigThreads, si, smem};
      WinState w;
      w.n = n;
      w.H = MatV{p.H, n}; w.T = MatV{p.T, n}; w.Q = MatV{p.Q, n}; w.Z = MatV{p.Z, n};
      w.wantq = w.wantz = true;
      w.tol = p.tol;
      cta_finalize(x, w, AR + eoff[q], AI + eoff[q], BE + eoff[q]);
    }
    if (threadIdx.x == 0) status[q] = info;
    __syncthreads();
  }
}

// H, T, Q, Z, then the role buffer and the standardisation's 3n doubles
size_t batch_smem_bytes(int smem_max) {
  return ((size_t)4 * smem_max * smem_ld(smem_max) + kRoleDoubles + 3 * (size_t)smem_max) * sizeof(double);
}

cudaError_t batch_init() {
  const cudaError_t e = cudaFuncSetAttribute(k_batch_big, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kBigSmem);
  if (e != cudaSuccess) return e;
  return cudaFuncSetAttribute(k_batch_qz, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              (int)batch_smem_bytes(kBatchSmemMax));
}

// Two launches: the pencils above kBatchSmemMax (the first nbig of the order;
// none with 128 threads, which keep the one-kernel form), then the others.
// Returns the status of this call's own memset and launches (cudaLaunchKernel
// reports the launch error directly, so an error left pending by unrelated
// earlier work is neither reported as ours nor cleared).
cudaError_t launch_batch(cudaStream_t st, int grid, int threads, int smem_max, int count, int nbig, int sm_count,
                         const int* order, const int* nsz, const int64_t* moff, const int64_t* eoff, double* H,
                         double* T, double* Q, double* Z, double* AR, double* AI, double* BE, int* status,
                         int* counter) {
  cudaError_t e = cudaMemsetAsync(counter, 0, 2 * sizeof(int), st);
  if (e != cudaSuccess) return e;
  if (threads != kRoleThreads) nbig = 0;
  if (nbig > 0) {
    void* args[] = {&nbig, &order, &nsz, &moff, &eoff, &H, &T, &Q, &Z, &AR, &AI, &BE, &status, &counter};
    e = cudaLaunchKernel((const void*)k_batch_big, dim3(std::min(nbig, sm_count)), dim3(kBigThreads), args, kBigSmem,
                         st);
    if (e != cudaSuccess) return e;
  }
  count -= nbig;
  order += nbig;
  counter += 1;
  if (count == 0) return cudaSuccess;
  void* args[] = {&count, &order, &nsz, &moff, &eoff, &H, &T, &Q, &Z, &AR, &AI, &BE, &status, &counter, &smem_max};
  return cudaLaunchKernel((const void*)k_batch_qz, dim3(grid), dim3(threads), args, batch_smem_bytes(smem_max), st);
}

int batch_big_count(const int* n, int count) {
  int k = 0;
  for (int i = 0; i < count; ++i) k += n[i] > kBatchSmemMax;
  return k;
}

// ---------------------------------------------------------------------------
// Batched solve that allocates nothing.
//
// For callers that may not allocate device memory themselves: code that
// runs inside another library's memory pool or allocator, hosts that
// reserve the whole device heap up front, or real-time loops where an
// allocation could block.  The per-batch descriptors and the work-queue
// counter live in one fixed array in the library's device memory instead
// of a buffer from cudaMalloc.  Every GPU that loads the library holds the
// array (kNoAllocBytes) until the process exits.
// ---------------------------------------------------------------------------
namespace {

constexpr int kNoAllocMaxPencils = 4096;
// moff, eoff (int64), order, n (int32), two queue counters
constexpr size_t kNoAllocBytes = (size_t)kNoAllocMaxPencils * (2 * sizeof(int64_t) + 2 * sizeof(int)) + 256;

static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocBytes];

constexpr int kNoAllocMaxDevices = 64;
struct NoAllocDev {
  bool ready = false;
  unsigned char* scratch = nullptr;  // device address of g_noalloc_scratch
  int sm_count = 0;
};
NoAllocDev g_noalloc_dev[kNoAllocMaxDevices];
std::mutex g_noalloc_mu;

// Both kernels on an empty queue, waited for.  k_batch_big's frame (its rare
// block swaps in doubled precision, at 128 registers) is larger than the
// per-thread stack a context begins with, and CUDA takes the device memory for
// a larger one, about 78 MB, at the first launch that needs it.
cudaError_t noalloc_first_launches(int* counter) {
  cudaStream_t st;
  cudaError_t e = cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking);
  if (e != cudaSuccess) return e;
  int none = 0, smem_max = kBatchSmemMax;
  const int* ip = nullptr;
  const int64_t* lp = nullptr;
  double* dp = nullptr;
  int* status = nullptr;
  // (as launch_batch passes them)
  void* args[] = {&none, &ip, &ip, &lp, &lp, &dp, &dp, &dp, &dp, &dp, &dp, &dp, &status, &counter, &smem_max};
  e = cudaLaunchKernel((const void*)k_batch_big, dim3(1), dim3(kBigThreads), args, kBigSmem, st);
  if (e == cudaSuccess)
    e = cudaLaunchKernel((const void*)k_batch_qz, dim3(1), dim3(kRoleThreads), args, batch_smem_bytes(smem_max), st);
  const cudaError_t es = cudaStreamSynchronize(st), ed = cudaStreamDestroy(st);
  return e != cudaSuccess ? e : es != cudaSuccess ? es : ed;
}

// Once per device, with that device current: the device address of the
// scratch array (its host-side name is only a stand-in), the SM count, the
// kernels' shared-memory limits and their first launches, so that no later
// call has to take device memory.
int noalloc_setup(int dev, NoAllocDev** out) {
  if (dev < 0 || dev >= kNoAllocMaxDevices) return 10001;
  std::lock_guard<std::mutex> lk(g_noalloc_mu);
  NoAllocDev& d = g_noalloc_dev[dev];
  if (!d.ready) {
    void* p = nullptr;
    if (cudaGetSymbolAddress(&p, g_noalloc_scratch) != cudaSuccess) return 10001;
    if (cudaDeviceGetAttribute(&d.sm_count, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 10001;
    if (batch_init() != cudaSuccess) return 10001;
    if (noalloc_first_launches((int*)((unsigned char*)p + kNoAllocBytes - 256)) != cudaSuccess) return 10001;
    d.scratch = (unsigned char*)p;
    d.ready = true;
  }
  *out = &d;
  return 0;
}

}  // namespace

}  // namespace qz

extern "C" int b200qz_solve_batched_noalloc(int count, const int* n, const long long* moff, const long long* eoff,
                                            double* h, double* t, double* q, double* z, double* alphar,
                                            double* alphai, double* beta, int* info, void* stream) {
  using namespace qz;
  if (count < 0) return -1;
  if (count > kNoAllocMaxPencils) return -2;
  for (int i = 0; i < count; ++i)
    if (n[i] < 1 || n[i] > 46340) return -3;
  if (count == 0) return 0;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 10001;
  NoAllocDev* d = nullptr;
  if (noalloc_setup(dev, &d) != 0) return 10001;
  cudaStream_t st = (cudaStream_t)stream;
  // longest pencils first on the work queue (order held on the stack)
  int order[kNoAllocMaxPencils];
  for (int i = 0; i < count; ++i) order[i] = i;
  std::sort(order, order + count, [&](int a, int b) { return n[a] != n[b] ? n[a] > n[b] : a < b; });
  int64_t* d_moff = (int64_t*)d->scratch;
  int64_t* d_eoff = d_moff + kNoAllocMaxPencils;
  int* d_order = (int*)(d_eoff + kNoAllocMaxPencils);
  int* d_n = d_order + kNoAllocMaxPencils;
  int* d_counter = d_n + kNoAllocMaxPencils;
  // Host-to-device copies from pageable memory (the stack array `order`, and
  // n/moff/eoff when the caller passes ordinary memory) return only after
  // the source has been copied to a staging buffer, as the CUDA runtime
  // documents for cudaMemcpyAsync from pageable memory, so `order` may go
  // out of scope on return.  Page-locked n/moff/eoff are read when the
  // stream reaches the copy: the caller keeps them unchanged until then.
  if (cudaMemcpyAsync(d_moff, moff, count * sizeof(int64_t), cudaMemcpyHostToDevice, st) != cudaSuccess ||
      cudaMemcpyAsync(d_eoff, eoff, count * sizeof(int64_t), cudaMemcpyHostToDevice, st) != cudaSuccess ||
      cudaMemcpyAsync(d_order, order, count * sizeof(int), cudaMemcpyHostToDevice, st) != cudaSuccess ||
      cudaMemcpyAsync(d_n, n, count * sizeof(int), cudaMemcpyHostToDevice, st) != cudaSuccess)
    return 10001;
  // the queue counters are zeroed on the stream before the kernels start
  const cudaError_t e =
      launch_batch(st, d->sm_count, kRoleThreads, kBatchSmemMax, count, batch_big_count(n, count), d->sm_count,
                   d_order, d_n, d_moff, d_eoff, h, t, q, z, alphar, alphai, beta, info, d_counter);
  return e == cudaSuccess ? 0 : 10001;
}

