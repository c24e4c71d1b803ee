// Multi-job launches.
//
// Every kernel body of the partitioner is written against a virtual grid:
// Body::run(args, vb, vg) does the work of virtual block vb of a job whose
// virtual grid has vg blocks.  Two kernels are generated from each body:
//
//   single_kernel<Body>  one job, arguments by value, vb = blockIdx.x;
//   multi_kernel<Body>   many jobs in one launch.  Job j owns the virtual
//                        blocks [cta0[j], cta0[j+1]); each CTA takes one
//                        virtual block (grid-striding only past 2^22 of
//                        them), finds its job with one warp-wide search of
//                        cta0 and loads the job's argument record into
//                        shared memory.  The hardware block scheduler
//                        balances the jobs' uneven blocks.
//
// A body's result for a job depends only on the job's arguments and its
// virtual grid, never on which physical CTA ran which virtual block, so a
// job computes the same bits alone and inside any mix of other jobs.
#pragma once

#include "common.cuh"
#include "kernels.h"

#include <algorithm>
#include <cstring>
#include <type_traits>

namespace sbp {

// A body that sets kCluster runs its blocks in clusters of that size: its
// virtual grids are multiples of it, so a cluster's blocks belong to one job
// and are consecutive virtual blocks.
template <class Body, class = void>
struct ClusterOf {
  static constexpr int value = 1;
};
template <class Body>
struct ClusterOf<Body, std::void_t<decltype(Body::kCluster)>> {
  static constexpr int value = Body::kCluster;
};

// Programmatic dependent launch: a kernel may be launched while the one before
// it in its stream still runs (launch_kernel below), so that its blocks sit
// on the SMs when that one ends instead of being scheduled then.  Each kernel
// lets its successor launch at once and then waits until every kernel it
// depends on has completed and its memory is visible, before it reads
// anything but its parameters; a kernel that has completed implies all
// before it, since it has waited for them.  A batch of a small graph is a
// chain of launches of a few microseconds each: 1k LL partitions 16.8 -> 15.3
// ms, 20k HH 55.1 -> 53.2 ms, 200k HH unchanged.
// Read-only loads (__ldg) are for data that stays the same while a kernel is
// resident, which now includes the time its predecessors still write: the
// graph, the x log2 x table and the launch records, nothing that a kernel of
// the loop writes.
__device__ __forceinline__ void begin_kernel() {
  cudaTriggerProgrammaticLaunchCompletion();
  cudaGridDependencySynchronize();
}

// A body that sets kEarly makes the wait itself (wait_kernel), after loading
// what no kernel writes: the graph, the batch lists, its launch records.
// These come by copies that are complete before the first kernel behind them
// starts, so they may be read before the wait.
template <class Body, class = void>
struct IsEarly {
  static constexpr bool value = false;
};
template <class Body>
struct IsEarly<Body, std::void_t<decltype(Body::kEarly)>> {
  static constexpr bool value = Body::kEarly;
};
__device__ __forceinline__ void wait_kernel() { cudaGridDependencySynchronize(); }
template <class Body>
__device__ __forceinline__ void begin_body() {
  if constexpr (IsEarly<Body>::value) cudaTriggerProgrammaticLaunchCompletion();
  else begin_kernel();
}

template <class Body>
__global__ void __launch_bounds__(Body::kThreads, Body::kMinBlocks)
    single_kernel(typename Body::Args a) {
  begin_body<Body>();
  Body::run(a, (int)blockIdx.x, (int)gridDim.x);
}

template <class Body>
__global__ void __launch_bounds__(Body::kThreads, Body::kMinBlocks)
    __cluster_dims__(ClusterOf<Body>::value, 1, 1) single_cluster_kernel(typename Body::Args a) {
  begin_body<Body>();
  Body::run(a, (int)blockIdx.x, (int)gridDim.x);
}

template <class Body>
__device__ __forceinline__ void run_multi(const MultiSpan& sp) {
  using Args = typename Body::Args;
  static_assert(sizeof(Args) % 8 == 0, "argument records are copied in 8-byte words");
  constexpr int kWords = (int)(sizeof(Args) / 8);
  __shared__ unsigned long long raw[kWords];
  __shared__ int s_j, s_vb, s_vg;
  begin_body<Body>();
  const Args& a = *reinterpret_cast<const Args*>(raw);
  int loaded = -1;
  for (int blk = blockIdx.x; blk < sp.total; blk += gridDim.x) {
    if (threadIdx.x < 32) {
      // job = number of job starts cta0[1..njobs-1] at or below blk (the
      // starts increase strictly: jobs without blocks are not listed)
      const int lane = threadIdx.x;
      int cnt = 0;
      for (int i = 1 + lane; i < sp.njobs; i += 32) cnt += __ldg(sp.cta0 + i) <= blk ? 1 : 0;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
      if (lane == 0) {
        const int c0 = __ldg(sp.cta0 + cnt);
        s_j = cnt;
        s_vb = blk - c0;
        s_vg = __ldg(sp.cta0 + cnt + 1) - c0;
      }
    }
    __syncthreads();
    const int j = s_j, vb = s_vb, vg = s_vg;
    if (j != loaded) {
      const unsigned long long* src = reinterpret_cast<const unsigned long long*>(
          static_cast<const char*>(sp.args) + (size_t)j * sizeof(Args));
      for (int k = threadIdx.x; k < kWords; k += blockDim.x) raw[k] = __ldg(src + k);
      loaded = j;
    }
    __syncthreads();
    Body::run(a, vb, vg);
    __syncthreads();
  }
}

template <class Body>
__global__ void __launch_bounds__(Body::kThreads, Body::kMinBlocks) multi_kernel(MultiSpan sp) {
  run_multi<Body>(sp);
}

template <class Body>
__global__ void __launch_bounds__(Body::kThreads, Body::kMinBlocks)
    __cluster_dims__(ClusterOf<Body>::value, 1, 1) multi_cluster_kernel(MultiSpan sp) {
  run_multi<Body>(sp);
}

constexpr int kMaxMultiGrid = 1 << 22;

// Launches a kernel that starts with begin_kernel().
template <class Param>
void launch_kernel(void (*k)(Param), int grid, int threads, size_t smem, cudaStream_t st,
                   const Param& param) {
  ++g_launches;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t c{};
  c.gridDim = dim3((unsigned)grid);
  c.blockDim = dim3((unsigned)threads);
  c.dynamicSmemBytes = smem;
  c.stream = st;
  c.attrs = &at;
  c.numAttrs = 1;
  (void)cudaLaunchKernelEx(&c, k, param);  // an error stays for the caller's check
}

template <class Body>
void launch_multi(const MultiSpan& sp, cudaStream_t st) {
  if (sp.total <= 0) return;
  const int grid = std::min(sp.total, kMaxMultiGrid);
  if constexpr (ClusterOf<Body>::value > 1)
    launch_kernel(&multi_cluster_kernel<Body>, grid, Body::kThreads, Body::kSmem, st, sp);
  else
    launch_kernel(&multi_kernel<Body>, grid, Body::kThreads, Body::kSmem, st, sp);
}

template <class Body>
void launch_single(const typename Body::Args& a, int grid, cudaStream_t st) {
  if (grid <= 0) return;
  if constexpr (ClusterOf<Body>::value > 1)
    launch_kernel(&single_cluster_kernel<Body>, grid, Body::kThreads, Body::kSmem, st, a);
  else
    launch_kernel(&single_kernel<Body>, grid, Body::kThreads, Body::kSmem, st, a);
}

// Opts both kernels of a body in to its dynamic shared memory; once per
// device, before the first launch.
template <class Body>
cudaError_t allow_smem() {
  auto set = [](const void* f) {
    return cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Body::kSmem);
  };
  cudaError_t e, e2;
  if constexpr (ClusterOf<Body>::value > 1) {
    e = set((const void*)single_cluster_kernel<Body>);
    e2 = set((const void*)multi_cluster_kernel<Body>);
  } else {
    e = set((const void*)single_kernel<Body>);
    e2 = set((const void*)multi_kernel<Body>);
  }
  return e != cudaSuccess ? e : e2;
}

// One job's record through the by-value kernel, same virtual grid: a slot
// holding a single job costs no argument loads.
template <class Body>
void launch_one(const void* rec, int32_t vctas, cudaStream_t st) {
  typename Body::Args a;
  std::memcpy(&a, rec, sizeof(a));
  launch_single<Body>(a, vctas, st);
}

template <class Body>
constexpr MultiKernel multi_kernel_desc(const char* name) {
  return MultiKernel{sizeof(typename Body::Args), &launch_multi<Body>, &launch_one<Body>, name};
}

// Appends one job's record to a slot (nothing when it has no virtual blocks).
template <class Args>
void slot_push(Slot& s, const Args& a, int32_t vctas) {
  if (vctas <= 0) return;
  const size_t off = s.recs.size();
  s.recs.resize(off + sizeof(Args));
  std::memcpy(s.recs.data() + off, &a, sizeof(Args));
  s.cta0.push_back(s.cta0.back() + vctas);
}

inline int32_t ceil_div(long long a, long long b) { return (int32_t)((a + b - 1) / b); }

}  // namespace sbp
