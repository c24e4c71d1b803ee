// sbp_mdl_device_static: the MDL of a blockmodel that already sits in device
// memory, computed without allocating anything.
//
// Some callers cannot allocate device memory at the point where they need
// the objective: hosts that own all device memory through their own pool and
// do not let a library allocate behind their back, and serving loops that
// forbid the device-wide synchronisation a cudaMalloc or cudaFree can cost.
// For them this entry point keeps its scratch (the per-CTA partial sums) in
// one file-scope device array of fixed size, created when the library is
// loaded and held by every GPU that loads it until the process exits.  The
// caller passes the inputs and the outputs.
//
// Limits and rules of use:
//   * at most kStaticMaxBlocks (65,536) blocks; larger B is rejected;
//   * the first call on a device looks the array's device address up
//     (cudaGetSymbolAddress, with that device current) and caches it for the
//     process; make that first call before any stream capture.  A
//     cudaDeviceReset ends the context the cached address belongs to, and
//     the entry point must not be called on that device afterwards;
//   * every call on a device shares the one array, and the array keeps the
//     last call's contents: calls that overlap on the GPU (different
//     streams, or work still running) race on it and may give wrong values.
//     The CTA ticket of the reduction wraps to zero by itself, so that calls
//     that overlapped spoil no later call.
#include "../../include/sbp.h"
#include "common.cuh"

#include <cmath>
#include <mutex>
#include <string>

namespace sbp {
sbp_status host_fail(sbp_status st, const char* msg);

namespace {

constexpr int kStaticMaxBlocks = 65536;
constexpr int kStaticCtas = 128;
constexpr int kStaticThreads = 256;

struct StaticScratch {
  double sum[kStaticCtas], err[kStaticCtas];
  unsigned ticket;
};

// The whole scratch of sbp_mdl_device_static.
static __device__ __align__(256) unsigned char g_mdl_scratch[sizeof(StaticScratch)];

constexpr int kMaxDevices = 64;
std::mutex g_mu;
StaticScratch* g_addr[kMaxDevices] = {};

// A sum and the rounding errors left out of it (Knuth's two-sum): whatever
// the order of the additions, value() is rounded about once.
struct ExactSum {
  double s = 0.0, e = 0.0;
  __device__ __forceinline__ void add(double x) {
    const double t = __dadd_rn(s, x);
    const double z = __dsub_rn(t, s);
    e = __dadd_rn(e, __dadd_rn(__dsub_rn(s, __dsub_rn(t, z)), __dsub_rn(x, z)));
    s = t;
  }
  __device__ __forceinline__ void add(const ExactSum& o) {
    add(o.s);
    e = __dadd_rn(e, o.e);
  }
  // an infinite term (a count in a column of degree 0) leaves no error term
  __device__ __forceinline__ double value() const { return isfinite(s) ? __dadd_rn(s, e) : s; }
};

__device__ __forceinline__ ExactSum warp_total(ExactSum x) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    ExactSum y;
    y.s = __shfl_xor_sync(kFull, x.s, o);
    y.e = __shfl_xor_sync(kFull, x.e, o);
    x.add(y);
  }
  return x;
}

// data_S = sum over blocks b of sum over out-row b of
//   M (log2 M - log2 d_out[b] - log2 d_in[c])
// (compute_overall_S_transform, kernels.hpp:1066-1093), then
// S = model - data_S (partition.hpp:696-701).  The rows' sums of M are the
// degrees, so the terms are one per entry, whatever its row, and one per
// block: threads stride over both, and no launch waits for the other.  A
// thread per row took 200 us at 350 rows of 350 entries, a chain of dependent
// loads, behind a launch of its own for the logarithms; a call of this takes 9.  CTA sums land in the scratch and the last
// CTA (ticket) adds them; the additions carry their errors, so the result
// does not depend on the split.
__global__ void __launch_bounds__(kStaticThreads) static_mdl_kernel(
    StaticScratch* sc, int32_t B, const int32_t* __restrict__ optr,
    const int32_t* __restrict__ ocol, const uint32_t* __restrict__ ocnt,
    const uint32_t* __restrict__ d_out, const uint32_t* __restrict__ d_in, double model,
    double* S, double* data_S) {
  constexpr int kWarps = kStaticThreads / 32;
  __shared__ ExactSum sh[kWarps];
  __shared__ bool last;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int first = blockIdx.x * kStaticThreads + tid, step = gridDim.x * kStaticThreads;
  ExactSum acc;
  for (int b = first; b < B; b += step) acc.add(-xlog2x(d_out[b]));
  const int end = optr[B];
#pragma unroll 4
  for (long long i = (long long)optr[0] + first; i < end; i += step) {
    const uint32_t m = ocnt[i];
    const double ld = log2((double)d_in[ocol[i]]);
    if (m) acc.add(xlog2x(m) - (double)m * ld);
  }
  acc = warp_total(acc);
  if (lane == 0) sh[wid] = acc;
  __syncthreads();
  if (tid == 0) {
    for (int k = 1; k < kWarps; ++k) acc.add(sh[k]);
    sc->sum[blockIdx.x] = acc.s;
    sc->err[blockIdx.x] = acc.e;
    __threadfence();
    last = atomicInc(&sc->ticket, gridDim.x - 1) == gridDim.x - 1;
  }
  __syncthreads();
  if (last && wid == 0) {
    __threadfence();
    ExactSum t;
    for (int k = lane; k < (int)gridDim.x; k += 32) {
      ExactSum x;
      x.s = ((volatile double*)sc->sum)[k];
      x.e = ((volatile double*)sc->err)[k];
      t.add(x);
    }
    t = warp_total(t);
    if (lane == 0) {
      *data_S = t.value();
      *S = model - t.value();
    }
  }
}

// The scratch's device address on the current device, looked up once.
sbp_status scratch_address(StaticScratch** out) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return host_fail(SBP_ERR_CUDA, cudaGetErrorString(e));
  if (dev < 0 || dev >= kMaxDevices) return host_fail(SBP_ERR_INVALID, "device ordinal too large");
  std::lock_guard<std::mutex> lk(g_mu);
  if (!g_addr[dev]) {
    void* p = nullptr;
    e = cudaGetSymbolAddress(&p, g_mdl_scratch);
    if (e != cudaSuccess) return host_fail(SBP_ERR_CUDA, cudaGetErrorString(e));
    g_addr[dev] = (StaticScratch*)p;
  }
  *out = g_addr[dev];
  return SBP_OK;
}

}  // namespace
}  // namespace sbp

extern "C" sbp_status sbp_mdl_device_static(int32_t N, int32_t E, int32_t B,
                                            const int32_t* out_ptr, const int32_t* out_col,
                                            const uint32_t* out_cnt, const uint32_t* d_out,
                                            const uint32_t* d_in, double* S, double* data_S,
                                            void* stream) {
  using namespace sbp;
  if (N < 1 || E < 1 || B < 1 || !out_ptr || !out_col || !out_cnt || !d_out || !d_in || !S ||
      !data_S)
    return host_fail(SBP_ERR_INVALID, "sbp_mdl_device_static: bad arguments");
  if (B > kStaticMaxBlocks)
    return host_fail(SBP_ERR_INVALID,
                     "sbp_mdl_device_static: B exceeds its static scratch (65536 blocks)");
  StaticScratch* sc = nullptr;
  sbp_status s = scratch_address(&sc);
  if (s != SBP_OK) return s;
  cudaStream_t st = (cudaStream_t)stream;
  const double b = (double)B, x = b * b / (double)E;
  const double model =
      (double)E * (1.0 + x) * std::log(1.0 + x) - x * std::log(x) + (double)N * std::log(b);
  // A launch error left pending by earlier, unrelated work is cleared first
  // so that the status below belongs to this launch (a sticky error,
  // which ends the context, is reported again by the check after it).
  (void)cudaGetLastError();
  static_mdl_kernel<<<kStaticCtas, kStaticThreads, 0, st>>>(sc, B, out_ptr, out_col, out_cnt,
                                                            d_out, d_in, model, S, data_S);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return host_fail(SBP_ERR_CUDA, cudaGetErrorString(e));
  return SBP_OK;
}
