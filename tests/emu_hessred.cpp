// The Hessenberg-triangular reduction's kernels and the host code that
// launches them (hessred.cu), run on the host: every thread block of a launch
// after another, in an order that the test chooses, each as a block of fibers
// (warp_emu.h).  hessred_host.inc is that file with its launches turned into
// emu_launch calls, its shared memory into emu_shared() and its PTX into plain
// copies.
#include "emu_prims.h"

#include "roles_host.inc"

// the part of the CUDA runtime that it calls
using cudaError_t = int;
using cudaStream_t = void*;
enum { cudaSuccess = 0, cudaErrorLaunchTimeout = 702 };
enum { cudaFuncAttributeMaxDynamicSharedMemorySize, cudaDevAttrMultiProcessorCount, cudaMemcpyDeviceToHost };
inline cudaError_t cudaGetLastError() { return cudaSuccess; }
template <class F>
cudaError_t cudaFuncSetAttribute(F, int, int) { return cudaSuccess; }
inline cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
static int g_sms = 4;
inline cudaError_t cudaDeviceGetAttribute(int* v, int, int) { *v = g_sms; return cudaSuccess; }
inline cudaError_t cudaMallocAsync(double** p, size_t bytes, cudaStream_t) {
  *p = (double*)aligned_alloc(64, (bytes + 63) / 64 * 64);
  memset(*p, 0xff, bytes);  // (NaN: nothing may be read before it is written)
  return cudaSuccess;
}
inline cudaError_t cudaFreeAsync(void* p, cudaStream_t) { free(p); return cudaSuccess; }
inline cudaError_t cudaMemsetAsync(void* p, int v, size_t bytes, cudaStream_t) { memset(p, v, bytes); return cudaSuccess; }
inline cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t bytes, int, cudaStream_t) {
  memcpy(d, s, bytes);
  return cudaSuccess;
}
inline cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }

#define __global__
#define __launch_bounds__(...)
#define blockIdx emu_block_index()
#define gridDim emu_grid_size()
#define blockDim emu_block_size()

constexpr size_t kShared = 227 << 10;
inline double* emu_shared() {
  static double* const p = (double*)aligned_alloc(64, kShared);
  return p;
}
static int g_order = 0;      // blocks of a launch: 0 upwards, 1 downwards
static unsigned g_slow = 0;  // warps held back in every block
static long g_launches = 0;
template <class F>
void emu_launch(const F& body, int grid, int threads, size_t smem, cudaStream_t) {
  ++g_launches;
  if (smem > kShared) abort();
  for (int k = 0; k < grid; ++k) {
    blockIdx.x = g_order ? grid - 1 - k : k;
    gridDim.x = grid;
    blockDim.x = threads;
    memset(emu_shared(), 0xff, kShared);
    emu::run(threads, g_slow, (char*)emu_shared(), [&](int) { body(); });
  }
}

#include "hessred.cuh"
namespace qz {
inline void launch_identity(cudaStream_t, double* M, int64_t ld, int n) {
  for (int j = 0; j < n; ++j)
    for (int i = 0; i < n; ++i) M[i + j * ld] = i == j;
}
}  // namespace qz
// flags between warps: a poll may switch the warp out
#define hr_ld_acq emu::polled
#define hr_st_rel role_st
#include "hessred_host.inc"

extern "C" int emu_gghrd(int n, int ilo, int ihi, double* A, double* B, double* Q, double* Z, int W, int cq, int cz,
                         int qrows, int sms, int order, unsigned slow) {
  g_sms = sms;
  g_order = order;
  g_slow = slow;
  qz::GghrdOut out;
  return qz::gghrd_device(nullptr, cq, cz, qrows != 0, n, ilo, ihi, A, n, B, n, Q, n, Z, n, W, &out);
}
