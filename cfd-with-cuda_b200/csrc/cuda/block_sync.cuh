// Block-level synchronisation of the persistent PCG kernels (pcg.cu,
// pcg_dia.cu): progress flags between neighbouring blocks and the reduction
// of an iteration's dot products.  Every wait is bounded.
#pragma once
#include "common.cuh"

namespace cfd {
namespace {

// Block-level synchronisation of the pipelined solve (all waits bounded):
//   publish(k)         this block's own rows of phase k are written
//   publish_arrive(k)  the same, and its partials of a reduction are posted
//   wait_nb(k)         every block owning a row this block gathers reached k
//   wait_red           the arrivals of a reduction, then its sums
// A release is one gpu-scope fence by thread 0 after a block barrier, then
// relaxed stores of the flag and the counter; a wait is an acquire by the
// polling warp before a block barrier.  The polls look at the error word and
// the clock only every kPollCheck rounds: either costs as much as the poll.
constexpr int kPollCheck = 32;
struct BlockSync {
  unsigned* cnt;   // monotonic arrival counter
  unsigned* prog;  // phase flag per block
  int lo, hi;
  int* err;
  unsigned long long timeout_ns;

  static __device__ __forceinline__ void fence_gpu() { asm volatile("fence.acq_rel.gpu;" ::: "memory"); }
  __device__ void publish(unsigned k) {
    __syncthreads();
    if (threadIdx.x == 0) {
      fence_gpu();
      asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(prog + blockIdx.x), "r"(k) : "memory");
    }
  }
  // partials already written by thread 0 of this block
  __device__ void publish_arrive(unsigned k) {
    publish(k);
    if (threadIdx.x == 0) asm volatile("red.relaxed.gpu.global.add.u32 [%0], 1;" ::"l"(cnt) : "memory");
  }
  // Whether a wait that began at t0 has to end without its event.
  __device__ __forceinline__ bool give_up(unsigned long long t0) const {
    return ld_volatile_i32(err) != 0 || global_ns() - t0 > timeout_ns;
  }
  // THREADS > 0: called by the block's first THREADS threads only.
  template <int THREADS = 0>
  __device__ bool wait_nb(unsigned k) {
    __shared__ int ok;
    if (threadIdx.x < 32) {
      // one lane per neighbour block, all polled at once
      int good = 1;
      const unsigned long long t0 = global_ns();
      for (int j0 = lo; j0 <= hi; j0 += 32) {
        const int j = j0 + (int)threadIdx.x;
        bool done = j > hi;
        for (int spin = 1;; spin++) {
          if (!done) done = ld_acquire_u32(prog + j) >= k;
          if (__all_sync(0xffffffffu, done)) break;
          // the whole warp gives up together: every lane takes the same
          // sequence of warp-wide votes
          if (spin % kPollCheck == 0 && __any_sync(0xffffffffu, give_up(t0))) {
            good = 0;
            break;
          }
        }
        if (!good) break;
      }
      if (threadIdx.x == 0) {
        if (!good) atomicExch(err, 1);
        ok = good;
      }
    }
    if constexpr (THREADS > 0)
      asm volatile("bar.sync 1, %0;" ::"n"(THREADS) : "memory");
    else
      __syncthreads();
    return ok != 0;
  }
  // Waits until `target` arrivals, then sums the partials in one fixed order
  // (FP64): every block sees identical values, in every lane.  Called by one warp.
  template <int NV>
  __device__ bool warp_red(unsigned target, const double* buf, double (&sum)[NV]) {
    const int G = gridDim.x, lane = threadIdx.x & 31;
    int good = 1;
    const unsigned long long t0 = global_ns();
    for (int spin = 1; ld_acquire_u32(cnt) < target; spin++) {
      if (spin % kPollCheck == 0 && give_up(t0)) {
        good = 0;
        break;
      }
    }
    good = __all_sync(0xffffffffu, good);
#pragma unroll
    for (int k = 0; k < NV; k++) sum[k] = 0;
    if (!good) {
      if (lane == 0) atomicExch(err, 1);
      return false;
    }
#pragma unroll 5
    for (int i = lane; i < G; i += 32)
#pragma unroll
      for (int k = 0; k < NV; k++) sum[k] += __ldcg(buf + (size_t)k * G + i);
#pragma unroll
    for (int k = 0; k < NV; k++) sum[k] = warp_sum(sum[k]);
    return true;
  }
  // The same for the whole block, by its first warp.
  template <int NV>
  __device__ bool wait_red(unsigned target, const double* buf, double (&v)[NV]) {
    __shared__ double res[NV];
    __shared__ int ok;
    if (threadIdx.x < 32) {
      double sum[NV];
      const bool good = warp_red<NV>(target, buf, sum);
      if (threadIdx.x == 0) {
#pragma unroll
        for (int k = 0; k < NV; k++) res[k] = sum[k];
        ok = good;
      }
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < NV; k++) v[k] = res[k];
    const bool r = ok != 0;
    __syncthreads();
    return r;
  }
};

// Writes this block's partial sums of NV values into buf (thread 0).
template <int NV>
__device__ __forceinline__ void block_partials(double (&v)[NV], double* buf) {
  block_sum<NV>(v);
  if (threadIdx.x == 0)
#pragma unroll
    for (int k = 0; k < NV; k++) buf[(size_t)k * gridDim.x + blockIdx.x] = v[k];
}

}  // namespace
}  // namespace cfd
