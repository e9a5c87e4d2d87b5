// Products with a matrix stored by offsets (DiaArgs, kernels.h), for kernels
// whose blocks each own a contiguous range of 32-row slices (pcg_dia.cu, the
// FP64 SpMV of flexible CG).  The work of a block is split
// evenly over its 16 warps in groups of 16 taps, and the coefficients of the
// next group are loaded while the current one multiplies.
#pragma once
#include "common.cuh"
#include "kernels.h"

namespace cfd {
namespace {

constexpr int kDiaWarps = 16, kDiaThreads = 32 * kDiaWarps;
constexpr int kDiaGroup = 16;  // taps per group

// Shared memory of the partial products of a block of `slices` slices.
constexpr size_t dia_slot_bytes(int slices) { return (size_t)(slices + kDiaWarps) * 32 * sizeof(double); }
// Blocks of a one-pass kernel over a matrix of n rows (0: the partial products
// do not fit): one per SM, each owning at least one slice.
inline int dia_blocks(int n, int num_sms) {
  const int ns = (n + 31) / 32, g = ns < num_sms ? ns : num_sms;
  return g > 0 && dia_slot_bytes((ns + g - 1) / g) <= 200 * 1024 ? g : 0;
}

__device__ __forceinline__ double ld_coef(const double* p, unsigned long long policy) {
  double v;
  asm volatile("ld.global.nc.L1::no_allocate.L2::cache_hint.f64 %0, [%1], %2;" : "=d"(v) : "l"(p), "l"(policy));
  return v;
}

// The block's share of the matrix: slices [s0, s0 + ns), ng groups per slice.
// Warp w of nw owns groups [g0, g1) of the ns ng; its part of slice s goes to
// slot[s + w] (distinct for every warp and slice that meet).
struct DiaRows {
  DiaArgs d;
  const int* off;  // shared memory
  double (*slot)[32];
  int nw, s0, ns, ng, g0, g1;
  // the first groups of every warp, keep_bytes over the whole matrix, stay
  // in L2 from one iteration of a solve to the next; the rest passes through
  int gk;
  unsigned long long keep, once;

  __device__ __forceinline__ int owner(int g) const { return (nw * (g + 1) - 1) / (ns * ng); }
  // The coefficients of group g of the block.
  __device__ __forceinline__ void load(int g, int lane, double (&c)[kDiaGroup]) const {
    const int sl = g / ng, t0 = (g - sl * ng) * kDiaGroup;
    const unsigned long long policy = g < gk ? keep : once;
    const double* p = d.coef + ((size_t)(s0 + sl) * d.ntap + t0) * 32 + lane;
#pragma unroll
    for (int k = 0; k < kDiaGroup; k++) c[k] = t0 + k < d.ntap ? ld_coef(p + 32 * k, policy) : 0.0;
  }
  // Partial products of the warp's groups with v; c holds the first group on
  // entry and (the stream being cyclic) again on return.
  __device__ __forceinline__ void multiply(int warp, int lane, const double* v, double (&c)[kDiaGroup]) const {
    if (g0 >= g1) return;
    int sl = g0 / ng;
    double acc[4] = {0, 0, 0, 0};
    for (int g = g0; g < g1; g++) {
      const int t0 = (g - sl * ng) * kDiaGroup;
      double nxt[kDiaGroup];
      load(g + 1 < g1 ? g + 1 : g0, lane, nxt);
      const int row0 = (s0 + sl) * 32, row = row0 + lane;
      double x[kDiaGroup];
      if (row0 >= d.reach && row0 + 31 + d.reach < d.n) {
#pragma unroll
        for (int k = 0; k < kDiaGroup; k++) x[k] = v[row + off[t0 + k]];
      } else {
#pragma unroll
        for (int k = 0; k < kDiaGroup; k++) x[k] = v[min(max(row + off[t0 + k], 0), d.n - 1)];
      }
#pragma unroll
      for (int k = 0; k < kDiaGroup; k++) acc[k & 3] += c[k] * x[k];
      const bool last = g + 1 == g1 || g + 1 == (sl + 1) * ng;
      if (last) {
        slot[sl + warp][lane] = (acc[0] + acc[1]) + (acc[2] + acc[3]);
        acc[0] = acc[1] = acc[2] = acc[3] = 0;
        sl++;
      }
#pragma unroll
      for (int k = 0; k < kDiaGroup; k++) c[k] = nxt[k];
    }
  }
  // The product of row 32 sl + l of the block, after a block barrier.
  __device__ __forceinline__ double row(int sl, int l) const {
    const int w1 = owner(sl * ng + ng - 1);
    double y = 0;
    for (int w = owner(sl * ng); w <= w1; w++) y += slot[sl + w][l];
    return y;
  }
};

// Part of a matrix's coefficients that a persistent solve asks to stay in L2
// (126 MB, shared with the vectors; kernels that pass over the matrix once, or
// between reads of the coarse inverse, ask for none: 2 us slower with it).  Measured per iteration of
// the persistent PCG at 0 / 0.1 / 0.25 / 0.35 / 0.5 of the coefficients: 46.2 /
// 45.2 / 43.5 / 44.1 / 47.1 us for 275 MB (64^3), 22.5 / 21.8 / 21.2 / 20.8 /
// 20.2 for 118 MB (48^3; 19.8 at 0.6, 23.0 at 1): the L2's own rate is not much
// above the copy rate, and past about 70 MB it starts to lose lines.
constexpr double kPcgKeepBytes = 70e6;

// Sets up the block's share and its offsets table (kDiaMaxTaps + kDiaGroup ints
// of shared memory); slot: dia_slot_bytes(its slices); nw <= kDiaWarps.  The caller
// synchronises the block before the first product.
__device__ __forceinline__ DiaRows dia_rows(const DiaArgs& d, int* soff, double* slot, double keep_bytes,
                                            int nw = kDiaWarps) {
  const int nslices = (d.n + 31) >> 5, G = gridDim.x, warp = threadIdx.x >> 5;
  // padding taps: coefficient 0 at offset 0
  for (int k = threadIdx.x; k < kDiaMaxTaps + kDiaGroup; k += kDiaThreads) soff[k] = k < d.ntap ? d.off[k] : 0;
  DiaRows M;
  M.d = d;
  M.off = soff;
  M.s0 = (int)((long long)nslices * blockIdx.x / G);
  M.ns = (int)((long long)nslices * (blockIdx.x + 1) / G) - M.s0;
  M.ng = (d.ntap + kDiaGroup - 1) / kDiaGroup;
  const int T = M.ns * M.ng;
  M.nw = nw;  // the warps from nw on own nothing
  M.g0 = T * min(warp, nw) / nw;
  M.g1 = T * min(warp + 1, nw) / nw;
  M.slot = reinterpret_cast<double(*)[32]>(slot);
  M.keep = l2_evict_last();
  M.once = l2_evict_first();
  const double bytes = 256.0 * (double)nslices * d.ntap;
  M.gk = M.g0 + (bytes <= keep_bytes ? M.g1 - M.g0 : (int)((M.g1 - M.g0) * (keep_bytes / bytes)));
  // with fewer groups than warps some slots between a slice's first and last
  // warp are never written
  for (int k = threadIdx.x; k < (M.ns + kDiaWarps) * 32; k += kDiaThreads) slot[k] = 0.0;
  return M;
}

}  // namespace
}  // namespace cfd
