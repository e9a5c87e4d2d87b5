// Backward pass of the U-Net's 3x3x3 convolutions (stride 1 or 2): data and
// weight gradients in FP32, on the tensor cores.
//
// Weights and stored activations are BF16, so only the gradient g of a
// layer's output needs more than the tensor core's input type.  It is split
// into three BF16 parts by truncation (8 + 8 + 8 = 24 mantissa bits: exact for
// |g| >= 2^-110, below that off by less than 2^-133, BF16's smallest number),
// and every product with it becomes three mma.sync of 16 terms, one per part,
// each from zero.  The tensor core truncates what an addition inside a step shifts
// out, always towards zero, which adds up over the layers where rounding does not;
// so the parts are not chained through its accumulator but added in
// round-to-nearest FP32, lo, mid, hi and then the running sum, and the data
// gradient, whose errors every layer in front inherits, takes the hi part in two
// steps of eight terms.  (A tensor-memory accumulator would carry the whole sum
// through the tensor core's own additions.)  Error of a layer's weight gradient
// against 64 bits from the same stored activations, first / middle / last layer, in
// 1e-7:
//                                        65^3               161 x 25 x 25
//   FP32 on CUDA cores, atomics          1.5 / 1.2 / 1.6    1.1 / 1.8 / 1.1
//   three parts chained                  1.1 / 2.1 / 0.26   1.8 / 2.2 / 0.27
//   parts added apart                    0.62 / 1.3 / 0.26  1.1 / 1.4 / 0.27
//   the same, hi in steps of eight       0.38 / 0.98 / 0.26 0.56 / 0.98 / 0.27
//   (weight gradient in steps of eight too: 0.38 / 0.89 / 0.26, 0.56 / 0.83 / 0.27)
// and the calls, in ms, gradient of 65^3 and batch of 4 on 161 x 25 x 25: chained 1.40
// and 2.68, apart 1.44 and 2.74, hi in steps of eight 1.51 and 2.88, both kernels 1.55
// and 2.95.
//
// Both kernels use the row numbering of the forward convolution: a block
// stages a brick of voxels with a one-voxel halo in shared memory, rows
// hx + HX (hy + HY hz), channels contiguous in a row, so a tap is a constant
// row shift and ldmatrix reads any 16 consecutive rows.  Row pitches are an
// odd multiple of 16 bytes, so the 8 rows of an ldmatrix hit distinct banks.
// The derivative of the leaky ReLU (from the sign of the stored output) is
// applied while g is staged; nothing but the gradients themselves goes to
// memory.
//
// What bounds it: the shared-memory reads of the fragments and the
// latency of staging, at one or two blocks per SM (the layers are small:
// 0.5 to 3.8 GFLOP).  Measured on one sample of a 65^3 grid, against FP32
// CUDA-core kernels with one voxel (data) or one tap (weights) per thread
// row: the whole gradient call 13.0 -> 1.51 ms; a batch of 4 on 161 x 25 x 25
// 21.6 -> 2.88 ms.  Error of the whole gradient against 64 bits (same stored
// activations): 1.5e-7 -> 3.4e-8 relative at 65^3, 1.1e-7 -> 3.2e-8 on
// 161 x 25 x 25.
#include <cuda_bf16.h>

#include <algorithm>

#include "common.cuh"
#include "unet.h"

namespace cfd {

namespace {

struct BwdParams {
  int vd[3];              // grid of the convolution's output (of g)
  int id[3];              // grid of its input
  int cin, cout;
  int b[3], nb[3], h[3];  // brick, bricks per axis, halo box
  int kr;                 // rows of one z plane of a brick, rounded up to 16
  int rows;               // rows reserved for the halo box, lead row and read slack included
  const __nv_bfloat16 *in, *y, *w;  // y: the stored output (null: no activation)
  const float* g;
  const float* add;       // data gradient: added to the result (may be null)
  float* part;            // weight gradient: one record of 27 CI CO + CO sums per block
  float* dx;
};

__device__ __forceinline__ unsigned pack2(unsigned a, unsigned b) { return (a >> 16) | (b & 0xffff0000u); }

// g = hi + mid + lo (three truncations to BF16): exact for |g| >= 2^-110, off by
// less than 2^-133 below; an infinity or NaN stays in hi.  Returned in the upper
// halves.
__device__ __forceinline__ void split3(float g, unsigned& hi, unsigned& mid, unsigned& lo) {
  const unsigned u = __float_as_uint(g);
  if ((u & 0x7f800000u) == 0x7f800000u) {
    hi = (u & 0x007fffffu) ? 0x7fc00000u : u;
    mid = lo = 0u;
    return;
  }
  hi = u & 0xffff0000u;
  const float r1 = g - __uint_as_float(hi);
  mid = __float_as_uint(r1) & 0xffff0000u;
  lo = __float_as_uint(r1 - __uint_as_float(mid)) & 0xffff0000u;
}

// Four channels of g at voxel v (activation derivative applied).
__device__ __forceinline__ float4 load_g4(const BwdParams& p, long long v, int c) {
  float4 g = __ldg(reinterpret_cast<const float4*>(p.g + v * p.cout + c));
  if (p.y) {
    const uint2 q = __ldg(reinterpret_cast<const uint2*>(p.y + v * p.cout + c));
    // y <= 0 for BF16 bits: sign set or zero
    auto neg = [](unsigned bits16) { return __uint_as_float(bits16 << 16) <= 0.f; };
    if (neg(q.x & 0xffffu)) g.x *= kLeaky;
    if (neg(q.x >> 16)) g.y *= kLeaky;
    if (neg(q.y & 0xffffu)) g.z *= kLeaky;
    if (neg(q.y >> 16)) g.w *= kLeaky;
  }
  return g;
}

// The three parts of four channels into a row of part-major channels.
template <int CO>
__device__ __forceinline__ void store_split(unsigned char* row, int c, const float4& g) {
  unsigned h[4], m[4], l[4];
  split3(g.x, h[0], m[0], l[0]);
  split3(g.y, h[1], m[1], l[1]);
  split3(g.z, h[2], m[2], l[2]);
  split3(g.w, h[3], m[3], l[3]);
  *reinterpret_cast<uint2*>(row + 2 * c) = make_uint2(pack2(h[0], h[1]), pack2(h[2], h[3]));
  *reinterpret_cast<uint2*>(row + 2 * (CO + c)) = make_uint2(pack2(m[0], m[1]), pack2(m[2], m[3]));
  *reinterpret_cast<uint2*>(row + 2 * (2 * CO + c)) = make_uint2(pack2(l[0], l[1]), pack2(l[2], l[3]));
}

__device__ __forceinline__ void ldsm4(unsigned addr, unsigned (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr)
               : "memory");
}
__device__ __forceinline__ void ldsm4_t(unsigned addr, unsigned (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr)
               : "memory");
}
// c += A B (16 x 8 x 16, BF16 operands, FP32)
__device__ __forceinline__ void mma16816(float (&c)[4], const unsigned (&a)[4], unsigned b0, unsigned b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
      "{%0, %1, %2, %3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// c += A B (16 x 8 x 8): the first (a0, a1, b0) or second (a2, a3, b1) half of the
// terms of the fragments above
__device__ __forceinline__ void mma1688(float (&c)[4], unsigned a0, unsigned a1, unsigned b0) {
  asm volatile(
      "mma.sync.aligned.m16n8k8.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5}, {%6}, {%0, %1, %2, %3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a0), "r"(a1), "r"(b0));
}

__device__ __forceinline__ void brick_origin(const BwdParams& p, int b, int& x0, int& y0, int& z0) {
  x0 = (b % p.nb[0]) * p.b[0];
  y0 = ((b / p.nb[0]) % p.nb[1]) * p.b[1];
  z0 = (b / (p.nb[0] * p.nb[1])) * p.b[2];
}

// ---- weight gradient: dw[k][ci][co] += sum_v in[s v + d_k][ci] g[v][co] ----
// A GEMM over voxels: M = 16 input channels, N = 8 output channels, K = 16
// consecutive rows of the brick (halo columns and padding rows carry g = 0).
// Nine warps, one per (dy, dz); each keeps its three dx taps' CI x CO sums in
// registers over all bricks of the block and stores them once, in the block's
// record, which k_wgrad_sum adds up.  Stride 2 stages the input by parity phase (tap d reads
// phase d != 0 at coarse index v - (d < 0)).  blockIdx.y = (ci, co) block of
// a layer with more channels.  The blocks of the first ci block also sum the
// bias gradient.
constexpr int kWgWarps = 9;
template <int CI, int CO, int STRIDE>
__global__ void __launch_bounds__(32 * kWgWarps, CI * CO < 512 ? 2 : 1) k_wgrad(const __grid_constant__ BwdParams p) {
  constexpr int NPH = STRIDE == 2 ? 8 : 1, PI = 2 * CI + 16, PG = 6 * CO + 16, MT = CI / 16, NT = CO / 8;
  constexpr int QC = CO / 4;  // channel quads of a row of g
  static_assert(32 % QC == 0, "a thread keeps one channel quad");
  extern __shared__ __align__(128) unsigned char smem[];
  const int nph_rows = NPH * p.rows;
  unsigned char* sI = smem;
  unsigned char* sG = smem + (size_t)nph_rows * PI;
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
  const int nco = p.cout / CO, ci0 = (blockIdx.y / nco) * CI, co0 = (blockIdx.y % nco) * CO;
  const int HX = p.h[0], HY = p.h[1], HZ = p.h[2], KR = p.kr;
  const int nbox = HX * HY * HZ, nbricks = p.nb[0] * p.nb[1] * p.nb[2];
  // the lead row and the read slack of every phase: finite for good
  for (int i = t; i < NPH * (p.rows - nbox) * (PI / 16); i += blockDim.x) {
    const int c = i % (PI / 16), r = (i / (PI / 16)) % (p.rows - nbox), ph = i / ((PI / 16) * (p.rows - nbox));
    const int row = ph * p.rows + (r == 0 ? 0 : nbox + r);
    *reinterpret_cast<uint4*>(sI + (size_t)row * PI + 16 * c) = make_uint4(0, 0, 0, 0);
  }
  float acc[3][MT][NT][4];
#pragma unroll
  for (int a = 0; a < 3; a++)
#pragma unroll
    for (int m = 0; m < MT; m++)
#pragma unroll
      for (int n = 0; n < NT; n++) acc[a][m][n][0] = acc[a][m][n][1] = acc[a][m][n][2] = acc[a][m][n][3] = 0.f;
  float4 bs = make_float4(0.f, 0.f, 0.f, 0.f);
  const int dy = warp % 3 - 1, dz = warp / 3 - 1;
  int toff[3];  // row shift of the warp's taps
#pragma unroll
  for (int a = 0; a < 3; a++) {
    const int dx = a - 1;
    toff[a] = STRIDE == 2
                  ? ((dx != 0) + 2 * (dy != 0) + 4 * (dz != 0)) * p.rows - (dx < 0) - HX * ((dy < 0) + HY * (dz < 0))
                  : dx + HX * (dy + HY * dz);
  }
  const int q = lane >> 3, l8 = lane & 7;
  const unsigned aA = smem_u32(sI) + (unsigned)((l8 + 8 * (q >> 1) + 1) * PI + 16 * (q & 1));
  const unsigned aB = smem_u32(sG) + (unsigned)((l8 + 8 * (q & 1)) * PG + 16 * (q >> 1));

  for (int b = blockIdx.x; b < nbricks; b += gridDim.x) {
    int x0, y0, z0;
    brick_origin(p, b, x0, y0, z0);
    __syncthreads();
    // a warp stages whole x-lines of the box (every phase) and of g
    for (int ln = warp; ln < NPH * HY * HZ; ln += kWgWarps) {
      const int ph = ln / (HY * HZ), hy = ln % HY, hz = (ln / HY) % HZ;
      int y = y0 + hy - 1, z = z0 + hz - 1, xs = x0 - 1;
      if (STRIDE == 2) {
        xs = 2 * xs + (ph & 1);
        y = 2 * y + ((ph >> 1) & 1);
        z = 2 * z + (ph >> 2);
      }
      const bool line = y >= 0 && z >= 0 && y < p.id[1] && z < p.id[2];
      const __nv_bfloat16* src = p.in + ((long long)p.id[0] * (y + (long long)p.id[1] * z)) * p.cin + ci0;
      unsigned char* dst = sI + (size_t)(ph * p.rows + 1 + HX * (hy + HY * hz)) * PI;
#pragma unroll 4
      for (int i = lane; i < HX * (CI / 8); i += 32) {
        const int c = i % (CI / 8), hx = i / (CI / 8), x = xs + STRIDE * hx;
        uint4 u = make_uint4(0, 0, 0, 0);
        if (line && x >= 0 && x < p.id[0]) u = __ldg(reinterpret_cast<const uint4*>(src + (long long)x * p.cin + 8 * c));
        *reinterpret_cast<uint4*>(dst + (size_t)hx * PI + 16 * c) = u;
      }
    }
    for (int ln = warp; ln < p.b[2] * (p.b[1] + 1); ln += kWgWarps) {
      // line b[1] of a plane: its padding rows up to KR
      const int hy = ln % (p.b[1] + 1), zz = ln / (p.b[1] + 1), y = y0 + hy, z = z0 + zz;
      const bool line = hy < p.b[1] && y < p.vd[1] && z < p.vd[2];
      const int n = hy < p.b[1] ? HX : KR - HX * p.b[1];
      const long long v0 = (long long)p.vd[0] * (y + (long long)p.vd[1] * z);
      unsigned char* dst = sG + (size_t)(zz * KR + hy * HX) * PG;
#pragma unroll 4
      for (int i = lane; i < n * QC; i += 32) {
        const int c = 4 * (i % QC), hx = i / QC, x = x0 + hx - 1;
        float4 g = make_float4(0.f, 0.f, 0.f, 0.f);
        if (line && hx >= 1 && hx <= p.b[0] && x < p.vd[0]) g = load_g4(p, v0 + x, co0 + c);
        bs.x += g.x;
        bs.y += g.y;
        bs.z += g.z;
        bs.w += g.w;
        store_split<CO>(dst + (size_t)hx * PG, c, g);
      }
    }
    __syncthreads();
    for (int zz = 0; zz < p.b[2]; zz++) {
      const int row0 = ((zz + 1) * HY + 1) * HX;
      for (int s = 0; s < KR; s += 16) {
        const unsigned ab = aB + (unsigned)((zz * KR + s) * PG);
#pragma unroll
        for (int n2 = 0; n2 < NT / 2; n2++) {
          unsigned bf[3][4];
#pragma unroll
          for (int part = 0; part < 3; part++) ldsm4_t(ab + 2 * (part * CO + 16 * n2), bf[part]);
#pragma unroll
          for (int a = 0; a < 3; a++) {
#pragma unroll
            for (int m = 0; m < MT; m++) {
              unsigned af[4];
              ldsm4_t(aA + (unsigned)((row0 + s + toff[a]) * PI + 32 * m), af);
#pragma unroll
              for (int n = 0; n < 2; n++) {
                float v[4];
#pragma unroll
                for (int part = 2; part >= 0; part--) {
                  float c[4] = {0.f, 0.f, 0.f, 0.f};
                  mma16816(c, af, bf[part][2 * n], bf[part][2 * n + 1]);
#pragma unroll
                  for (int e = 0; e < 4; e++) v[e] = part == 2 ? c[e] : v[e] + c[e];
                }
#pragma unroll
                for (int e = 0; e < 4; e++) acc[a][m][2 * n2 + n][e] += v[e];
              }
            }
          }
        }
      }
    }
  }
  // the block's record: [27][CI][CO] sums, then the CO bias sums.  Lane pairs
  // exchange halves so that each lane stores four consecutive output
  // channels: even lanes row l / 4, odd lanes row l / 4 + 8
  float* rec = p.part + ((size_t)blockIdx.y * gridDim.x + blockIdx.x) * (27 * CI * CO + CO);
  const int odd = lane & 1;
#pragma unroll
  for (int a = 0; a < 3; a++) {
#pragma unroll
    for (int m = 0; m < MT; m++)
#pragma unroll
      for (int n = 0; n < NT; n++) {
        float(&v)[4] = acc[a][m][n];
        const float r0 = __shfl_xor_sync(0xffffffffu, odd ? v[0] : v[2], 1);
        const float r1 = __shfl_xor_sync(0xffffffffu, odd ? v[1] : v[3], 1);
        const int ci = 16 * m + (lane >> 2) + 8 * odd, co = 8 * n + 2 * ((lane & 3) - odd);
        *reinterpret_cast<float4*>(rec + ((a + 3 * warp) * CI + ci) * CO + co) =
            odd ? make_float4(r0, r1, v[2], v[3]) : make_float4(v[0], v[1], r0, r1);
      }
  }
  if (ci0 == 0) {
    float4* sb = reinterpret_cast<float4*>(smem);
    __syncthreads();
    sb[t] = bs;
    __syncthreads();
    if (t < QC) {
      float4 v = sb[t];
      for (int i = t + QC; i < (int)blockDim.x; i += QC) {
        v.x += sb[i].x;
        v.y += sb[i].y;
        v.z += sb[i].z;
        v.w += sb[i].w;
      }
      *reinterpret_cast<float4*>(rec + 27 * CI * CO + 4 * t) = v;
    }
  }
}

// dw += the sum of the blocks' records, in FP64 and in block order: the same
// bits every time, and no loss from adding many partial sums.  A block takes
// 16 channel quads of a record, 32 threads each over every 32nd record (few
// dependent rounds of loads: the records are in L2 and latency is the bound).
// blockIdx.y = (ci, co) block of the layer; nbias: bias sums of a record in use.
constexpr int kRedQ = 16, kRedS = 32;
__global__ void __launch_bounds__(kRedQ* kRedS) k_wgrad_sum(const float* __restrict__ part, int nrec, int ci_n,
                                                            int co_n, int cin, int cout, int nbias, float* dw,
                                                            float* db) {
  __shared__ double sh[kRedS][kRedQ][4];
  const int reclen = 27 * ci_n * co_n + co_n, q = threadIdx.x % kRedQ, sl = threadIdx.x / kRedQ;
  const int i = 4 * (blockIdx.x * kRedQ + q);  // first of four entries of the record
  const int nco = cout / co_n, ci0 = ((int)blockIdx.y / nco) * ci_n, co0 = ((int)blockIdx.y % nco) * co_n;
  const bool bias = i >= 27 * ci_n * co_n, use = i < reclen && !(bias && ci0 != 0);
  double v[4] = {0, 0, 0, 0};
  if (use) {
    const float* src = part + (size_t)blockIdx.y * nrec * reclen + i;
#pragma unroll 5
    for (int r = sl; r < nrec; r += kRedS) {
      const float4 f = __ldcg(reinterpret_cast<const float4*>(src + (size_t)r * reclen));
      v[0] += f.x;
      v[1] += f.y;
      v[2] += f.z;
      v[3] += f.w;
    }
  }
#pragma unroll
  for (int e = 0; e < 4; e++) sh[sl][q][e] = v[e];
  __syncthreads();
  if (sl != 0 || !use) return;
  float* d;
  int n = 4;
  if (bias) {
    d = db + co0 + (i - 27 * ci_n * co_n);
    n = min(4, nbias - (i - 27 * ci_n * co_n));
  } else {
    const int co = i % co_n, ci = (i / co_n) % ci_n, k = i / (co_n * ci_n);
    d = dw + ((size_t)k * cin + ci0 + ci) * cout + co0 + co;
  }
  for (int e = 0; e < n; e++) {
    double x = 0;
    for (int k = 0; k < kRedS; k++) x += sh[k][q][e];
    d[e] = (float)((double)d[e] + x);
  }
}

// ---- data gradient: dx[u][ci] = add[u][ci] + sum over taps of g[(u - d) / s] . w[d][ci] ----
// M = 16 consecutive rows of the brick, N = 8 input channels, K = 16 output
// channels; the block's weights (27 taps x CI x cout) stay in shared memory
// over its bricks.  A warp takes (16 rows, 16 input channels) units.  Stride
// 2: the brick is of g's grid, and each of the 8 parity classes of the fine
// voxel 2 i + p has its own taps (per axis: p = 0 the centre at i; p = 1 the
// tap +1 at i and the tap -1 at i + 1).  blockIdx.y = ci block.
constexpr int kDgThreads = 512;
template <int CI, int CO, int STRIDE>
__global__ void __launch_bounds__(kDgThreads, 2) k_dgrad(const __grid_constant__ BwdParams p) {
  constexpr int PG = 6 * CO + 16, PW = 2 * CO + 16, QC = CO / 4, NCLS = STRIDE == 2 ? 8 : 1;
  extern __shared__ __align__(128) unsigned char smem[];
  unsigned char* sW = smem;
  unsigned char* sG = smem + 27 * CI * PW;
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31, ci0 = blockIdx.y * CI;
  const int HX = p.h[0], HY = p.h[1], HZ = p.h[2], KR = p.kr;
  const int nbox = HX * HY * HZ, nbricks = p.nb[0] * p.nb[1] * p.nb[2];
  for (int i = t; i < 27 * CI * (CO / 8); i += kDgThreads) {
    const int c = i % (CO / 8), kc = i / (CO / 8), ci = kc % CI, k = kc / CI;
    *reinterpret_cast<uint4*>(sW + (size_t)kc * PW + 16 * c) =
        __ldg(reinterpret_cast<const uint4*>(p.w + ((size_t)k * p.cin + ci0 + ci) * CO + 8 * c));
  }
  for (int i = t; i < (p.rows - nbox) * (PG / 16); i += kDgThreads) {
    const int c = i % (PG / 16), r = i / (PG / 16), row = r == 0 ? 0 : nbox + r;
    *reinterpret_cast<uint4*>(sG + (size_t)row * PG + 16 * c) = make_uint4(0, 0, 0, 0);
  }
  const int q = lane >> 3, l8 = lane & 7;
  const unsigned aA = smem_u32(sG) + (unsigned)((l8 + 8 * (q & 1) + 1) * PG + 16 * (q >> 1));
  const unsigned aB = smem_u32(sW) + (unsigned)((l8 + 8 * (q >> 1)) * PW + 16 * (q & 1));
  const int tiles = p.b[2] * (KR / 16), units = tiles * NCLS * (CI / 16);
  for (int b = blockIdx.x; b < nbricks; b += gridDim.x) {
    int x0, y0, z0;
    brick_origin(p, b, x0, y0, z0);
    __syncthreads();
    for (int ln = warp; ln < HY * HZ; ln += kDgThreads / 32) {
      const int hy = ln % HY, hz = ln / HY, y = y0 + hy - 1, z = z0 + hz - 1;
      const bool line = y >= 0 && z >= 0 && y < p.vd[1] && z < p.vd[2];
      const long long v0 = (long long)p.vd[0] * (y + (long long)p.vd[1] * z);
      unsigned char* dst = sG + (size_t)(1 + HX * ln) * PG;
#pragma unroll 4
      for (int i = lane; i < HX * QC; i += 32) {
        const int c = 4 * (i % QC), hx = i / QC, x = x0 + hx - 1;
        float4 g = make_float4(0.f, 0.f, 0.f, 0.f);
        if (line && x >= 0 && x < p.vd[0]) g = load_g4(p, v0 + x, c);
        store_split<CO>(dst + (size_t)hx * PG, c, g);
      }
    }
    __syncthreads();
    for (int un = warp; un < units; un += kDgThreads / 32) {
      // stride 2: the parity classes with most taps first
      const int cb = un % (CI / 16), tile = (un / (CI / 16)) % tiles;
      const int cls = STRIDE == 2 ? (0x04216537 >> (4 * (un / ((CI / 16) * tiles)))) & 7 : 0;
      const int zz = tile / (KR / 16), s = 16 * (tile % (KR / 16));
      const int row0 = ((zz + 1) * HY + 1) * HX + s;
      const int px = cls & 1, py = (cls >> 1) & 1, pz = cls >> 2;
      float acc[2][4] = {};
      auto tap = [&](int k, int off) {
        const unsigned ra = aA + (unsigned)((row0 + off) * PG), rb = aB + (unsigned)((k * CI + 16 * cb) * PW);
#pragma unroll
        for (int kc = 0; kc < CO / 16; kc++) {
          unsigned bw[4];
          ldsm4(rb + 32 * kc, bw);
          float v[2][4];
#pragma unroll
          for (int part = 2; part >= 0; part--) {
            unsigned af[4];
            ldsm4(ra + 2 * part * CO + 32 * kc, af);
#pragma unroll
            for (int n = 0; n < 2; n++) {
              float c[4] = {0.f, 0.f, 0.f, 0.f};
              if (part == 0) {
                float d[4] = {0.f, 0.f, 0.f, 0.f};
                mma1688(c, af[0], af[1], bw[2 * n]);
                mma1688(d, af[2], af[3], bw[2 * n + 1]);
#pragma unroll
                for (int e = 0; e < 4; e++) c[e] += d[e];
              } else {
                mma16816(c, af, bw[2 * n], bw[2 * n + 1]);
              }
#pragma unroll
              for (int e = 0; e < 4; e++) v[n][e] = part == 2 ? c[e] : v[n][e] + c[e];
            }
          }
#pragma unroll
          for (int n = 0; n < 2; n++)
#pragma unroll
            for (int e = 0; e < 4; e++) acc[n][e] += v[n][e];
        }
      };
      if constexpr (STRIDE == 2) {
        const int ntap = 1 << (px + py + pz);
        for (int j = 0; j < ntap; j++) {
          // bit j of the odd axes: 0 the tap +1 at i, 1 the tap -1 at i + 1
          const int jx = px ? j & 1 : 0, jy = py ? (j >> px) & 1 : 0, jz = pz ? (j >> (px + py)) & 1 : 0;
          const int k = (px ? 2 - 2 * jx : 1) + 3 * (py ? 2 - 2 * jy : 1) + 9 * (pz ? 2 - 2 * jz : 1);
          tap(k, jx + HX * (jy + HY * jz));
        }
      } else {
#pragma unroll 1
        for (int yz = 0; yz < 9; yz++) {
          const int off = -HX * ((yz % 3 - 1) + HY * (yz / 3 - 1));
          tap(3 * yz, off + 1);
          tap(3 * yz + 1, off);
          tap(3 * yz + 2, off - 1);
        }
      }
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const int r = s + (lane >> 2) + 8 * h, hy = r / HX, hx = r - hy * HX;
        int x = x0 + hx - 1, y = y0 + hy, z = z0 + zz;
        if (hx < 1 || hx > p.b[0] || hy >= p.b[1]) continue;
        if (STRIDE == 2) {
          x = 2 * x + px;
          y = 2 * y + py;
          z = 2 * z + pz;
        }
        if (x >= p.id[0] || y >= p.id[1] || z >= p.id[2]) continue;
        const long long o =
            (x + (long long)p.id[0] * (y + (long long)p.id[1] * z)) * p.cin + ci0 + 16 * cb + 2 * (lane & 3);
#pragma unroll
        for (int n = 0; n < 2; n++) {
          float2 v = make_float2(acc[n][2 * h], acc[n][2 * h + 1]);
          if (p.add) {
            const float2 a = __ldg(reinterpret_cast<const float2*>(p.add + o + 8 * n));
            v.x += a.x;
            v.y += a.y;
          }
          *reinterpret_cast<float2*>(p.dx + o + 8 * n) = v;
        }
      }
    }
  }
}

// ---- the layers with one channel on one side (16 on the other), CUDA cores ----
constexpr int kOX = 16, kOY = 4, kOZ = 4;

// Data gradient of the last layer (16 -> 1): one thread per voxel, the
// tile's g with its halo and the 27 x 16 weights in shared memory.
__global__ void __launch_bounds__(kOX* kOY* kOZ) k_dgrad_1(const __grid_constant__ BwdParams p) {
  constexpr int HX = kOX + 2, HY = kOY + 2, HZ = kOZ + 2;
  __shared__ float tile[HX * HY * HZ];
  __shared__ float4 sw[27 * 4];
  for (int i = threadIdx.x; i < 27 * 16; i += blockDim.x) ((float*)sw)[i] = __bfloat162float(p.w[i]);
  const int nx = p.vd[0], ny = p.vd[1], nz = p.vd[2];
  const int tbx = (nx + kOX - 1) / kOX, tby = (ny + kOY - 1) / kOY;
  const int x0 = kOX * (blockIdx.x % tbx), y0 = kOY * ((blockIdx.x / tbx) % tby), z0 = kOZ * (blockIdx.x / (tbx * tby));
  for (int i = threadIdx.x; i < HX * HY * HZ; i += blockDim.x) {
    const int x = x0 - 1 + i % HX, y = y0 - 1 + (i / HX) % HY, z = z0 - 1 + i / (HX * HY);
    float g = 0.f;
    if (x >= 0 && y >= 0 && z >= 0 && x < nx && y < ny && z < nz) g = __ldg(p.g + x + (size_t)nx * (y + (size_t)ny * z));
    tile[i] = g;
  }
  __syncthreads();
  const int tx = threadIdx.x % kOX, ty = (threadIdx.x / kOX) % kOY, tz = threadIdx.x / (kOX * kOY);
  const int x = x0 + tx, y = y0 + ty, z = z0 + tz;
  if (x >= nx || y >= ny || z >= nz) return;
  float acc[16] = {};
#pragma unroll 3
  for (int k = 0; k < 27; k++) {
    const float a = tile[(tx + 2 - k % 3) + HX * ((ty + 2 - (k / 3) % 3) + HY * (tz + 2 - k / 9))];
#pragma unroll
    for (int c = 0; c < 4; c++) {
      const float4 w = sw[4 * k + c];
      acc[4 * c] += a * w.x;
      acc[4 * c + 1] += a * w.y;
      acc[4 * c + 2] += a * w.z;
      acc[4 * c + 3] += a * w.w;
    }
  }
  float4* d = reinterpret_cast<float4*>(p.dx + (x + (size_t)nx * (y + (size_t)ny * z)) * 16);
#pragma unroll
  for (int c = 0; c < 4; c++) d[c] = make_float4(acc[4 * c], acc[4 * c + 1], acc[4 * c + 2], acc[4 * c + 3]);
}

// Weight gradient of the first (1 -> 16) and last (16 -> 1) layer, both
// dw[k][c] = sum_v s[v + sign d_k] q[v][c] with a scalar field s and a
// 16-channel field q (FIRST: s the input, q the output gradient; else s the
// output gradient, q the input).  A thread owns a (dy, dz) pair and four
// channels and walks an x-row with the three dx values of s in registers:
// 12 multiply-adds per two shared-memory reads.  Eight rows of a tile at a
// time, sums kept over all tiles of the block.
constexpr int kW1Groups = 8, kW1Threads = 36 * kW1Groups;
template <bool FIRST>
__global__ void __launch_bounds__(kW1Threads) k_wgrad_1(const __grid_constant__ BwdParams p) {
  constexpr int HX = kOX + 2, HY = kOY + 2, HZ = kOZ + 2, SG = FIRST ? 1 : -1;
  __shared__ float s[HX * HY * HZ];
  __shared__ float4 qv[kOX * kOY * kOZ * 4];
  __shared__ __align__(16) float red[kW1Threads * 12];  // read and written as float4 too
  const int t = threadIdx.x, cq = t & 3, yz = (t >> 2) % 9, grp = t / 36;
  const int dy = SG * (yz % 3 - 1), dz = SG * (yz / 3 - 1);
  const int nx = p.vd[0], ny = p.vd[1], nz = p.vd[2];
  const int tbx = (nx + kOX - 1) / kOX, tby = (ny + kOY - 1) / kOY, tbz = (nz + kOZ - 1) / kOZ;
  float acc[3][4] = {};
  float4 bs = make_float4(0.f, 0.f, 0.f, 0.f);
  for (int b = blockIdx.x; b < tbx * tby * tbz; b += gridDim.x) {
    const int x0 = kOX * (b % tbx), y0 = kOY * ((b / tbx) % tby), z0 = kOZ * (b / (tbx * tby));
    __syncthreads();
    for (int i = t; i < HX * HY * HZ; i += kW1Threads) {
      const int x = x0 - 1 + i % HX, y = y0 - 1 + (i / HX) % HY, z = z0 - 1 + i / (HX * HY);
      float v = 0.f;
      if (x >= 0 && y >= 0 && z >= 0 && x < nx && y < ny && z < nz) {
        const size_t u = x + (size_t)nx * (y + (size_t)ny * z);
        v = FIRST ? __bfloat162float(p.in[u]) : __ldg(p.g + u);
      }
      s[i] = v;
    }
    for (int i = t; i < kOX * kOY * kOZ * 4; i += kW1Threads) {
      const int c = i & 3, r = i >> 2;
      const int x = x0 + r % kOX, y = y0 + (r / kOX) % kOY, z = z0 + r / (kOX * kOY);
      float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
      if (x < nx && y < ny && z < nz) {
        const long long u = x + (long long)nx * (y + (long long)ny * z);
        if (FIRST) {
          v = load_g4(p, u, 4 * c);
        } else {
          const uint2 a = __ldg(reinterpret_cast<const uint2*>(p.in + u * 16 + 4 * c));
          v = make_float4(__uint_as_float(a.x << 16), __uint_as_float(a.x & 0xffff0000u), __uint_as_float(a.y << 16),
                          __uint_as_float(a.y & 0xffff0000u));
        }
      }
      qv[i] = v;
      if (FIRST) {
        bs.x += v.x;
        bs.y += v.y;
        bs.z += v.z;
        bs.w += v.w;
      }
    }
    __syncthreads();
    if (!FIRST)
      for (int i = t; i < kOX * kOY * kOZ; i += kW1Threads)
        bs.x += s[1 + i % kOX + HX * (1 + (i / kOX) % kOY + HY * (1 + i / (kOX * kOY)))];
    for (int r = grp; r < kOY * kOZ; r += kW1Groups) {
      float ra[3][4] = {};
      const float* sr = s + 1 + HX * (r % kOY + 1 + dy + HY * (r / kOY + 1 + dz));
      const float4* qr = qv + r * kOX * 4 + cq;
      float a = sr[-1], m = sr[0];
#pragma unroll
      for (int x = 0; x < kOX; x++) {
        const float c = sr[x + 1];
        const float4 v = qr[4 * x];
        const float sv[3] = {FIRST ? a : c, m, FIRST ? c : a};
#pragma unroll
        for (int k = 0; k < 3; k++) {
          ra[k][0] += sv[k] * v.x;
          ra[k][1] += sv[k] * v.y;
          ra[k][2] += sv[k] * v.z;
          ra[k][3] += sv[k] * v.w;
        }
        a = m;
        m = c;
      }
#pragma unroll
      for (int k = 0; k < 3; k++)
#pragma unroll
        for (int e = 0; e < 4; e++) acc[k][e] += ra[k][e];
    }
  }
#pragma unroll
  for (int k = 0; k < 3; k++)
#pragma unroll
    for (int e = 0; e < 4; e++) red[t * 12 + 4 * k + e] = acc[k][e];
  __syncthreads();
  // the block's record: [27][16] sums, then the bias sums (16, or 1 and padding)
  float* rec = p.part + (size_t)blockIdx.x * (27 * 16 + 16);
  for (int i = t; i < 36 * 12; i += kW1Threads) {
    float v = 0.f;
    for (int g = 0; g < kW1Groups; g++) v += red[g * 36 * 12 + i];
    const int th = i / 12, k = (i % 12) / 4, e = i % 4;
    rec[(3 * (th >> 2) + k) * 16 + 4 * (th & 3) + e] = v;
  }
  __syncthreads();
  // a thread staged one channel quad of q (kW1Threads is a multiple of 4), or
  // with FIRST = false summed s over its voxels
  *reinterpret_cast<float4*>(red + 4 * t) = bs;
  __syncthreads();
  if (t < 16) {
    float v = 0.f;
    if (FIRST)
      for (int i = t >> 2; i < kW1Threads; i += 4) v += red[4 * i + (t & 3)];
    else if (t == 0)
      for (int i = 0; i < kW1Threads; i++) v += red[4 * i];
    rec[27 * 16 + t] = v;
  }
}

int ceil_div(int a, int b) { return (a + b - 1) / b; }

constexpr int kSmemMax = 227 * 1024;

BwdParams bwd_params(const ConvDesc& d, const float* g, const __nv_bfloat16* y) {
  BwdParams p{};
  for (int a = 0; a < 3; a++) {
    p.vd[a] = d.out_dims[a];
    p.id[a] = d.in_dims[a];
  }
  p.cin = d.ca;
  p.cout = d.cout;
  p.in = d.inA;
  p.w = d.w;
  p.g = g;
  p.y = y;
  return p;
}

// Brick of a block: x-rows of at most 33 voxels (the coarser grids' whole
// rows) and the y-z extent with the least estimated time: waves of bricks
// over the blocks that run at once, times the rows a brick multiplies (a
// block of W warps takes W tiles of 16 rows at a time) plus the rows it
// stages.  hi: halo rows on the high side (0 or 1); smem_of(p) gives the
// bytes of a brick, per_sm(bytes) the blocks an SM holds (1 or 2).  False when no
// brick fits.
template <class F, class S>
bool pick_brick(BwdParams& p, int hi, int warps, int blocks_y, int num_sms, F smem_of, S per_sm, size_t& smem) {
  BwdParams best = p;
  double least = -1;
  for (int nbx = ceil_div(p.vd[0], 33); least < 0 && nbx <= p.vd[0]; nbx++)
    for (int by = 1; by <= std::min(6, p.vd[1]); by++)
      for (int bz = 1; bz <= std::min(4, p.vd[2]); bz++) {
        p.b[0] = ceil_div(p.vd[0], nbx);
        p.b[1] = by;
        p.b[2] = bz;
        for (int a = 0; a < 3; a++) {
          p.nb[a] = ceil_div(p.vd[a], p.b[a]);
          p.h[a] = p.b[a] + 1 + hi;
        }
        const int HX = p.h[0], HY = p.h[1], box = HX * HY * p.h[2], reach = 1 + HX + HX * HY;
        p.kr = 16 * ceil_div(by * HX, 16);
        // last row an operand can start in, and the lead row
        p.rows = std::max(box, (bz * HY + 1) * HX + p.kr + (hi ? reach : 0)) + 2;
        const size_t need = smem_of(p);
        if (need > (size_t)kSmemMax) continue;
        const int waves = ceil_div(p.nb[0] * p.nb[1] * p.nb[2], std::max(1, per_sm(need) * num_sms / blocks_y));
        // two blocks on an SM share it, but overlap staging and products
        const double t = waves * (per_sm(need) == 1 ? 1.0 : 1.6) *
                         (16.0 * warps * ceil_div(bz * p.kr / 16, warps) + 0.5 * box + 64.0);
        if (least < 0 || t < least) {
          least = t;
          best = p;
          smem = need;
        }
      }
  p = best;
  return least >= 0;
}

// Records of the weight gradient's blocks: at most two blocks per SM.
constexpr int kWgPerSm = 2;

cudaError_t sum_records(const float* part, int nrec, int ci_n, int co_n, int cin, int cout, int nbias, float* dw,
                        float* db, cudaStream_t s) {
  const int quads = (27 * ci_n * co_n + co_n) / 4, by = (cin / ci_n) * (cout / co_n);
  k_wgrad_sum<<<dim3(ceil_div(quads, kRedQ), by), kRedQ * kRedS, 0, s>>>(part, nrec, ci_n, co_n, cin, cout, nbias, dw,
                                                                         db);
  return cudaGetLastError();
}

template <int CI, int CO, int STRIDE>
cudaError_t launch_wgrad(BwdParams p, float* dw, float* db, int num_sms, cudaStream_t s) {
  const int by = (p.cin / CI) * (p.cout / CO);
  size_t smem = 0;
  auto bytes = [](const BwdParams& q) {
    return std::max((size_t)(STRIDE == 2 ? 8 : 1) * q.rows * (2 * CI + 16) + (size_t)q.b[2] * q.kr * (6 * CO + 16),
                    sizeof(float4) * 32 * kWgWarps);
  };
  auto k = k_wgrad<CI, CO, STRIDE>;
  cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemMax);
  if (e != cudaSuccess) return e;
  // two blocks per SM where shared memory and the accumulators leave room
  auto per_sm = [](size_t need) { return CI * CO < 512 && 2 * (need + 1024) <= (size_t)kSmemMax ? kWgPerSm : 1; };
  if (p.cin % CI || p.cout % CO || !pick_brick(p, STRIDE == 1 ? 1 : 0, 1, by, num_sms, bytes, per_sm, smem))
    return cudaErrorInvalidValue;
  const int nrec = std::min(p.nb[0] * p.nb[1] * p.nb[2], std::max(1, per_sm(smem) * num_sms / by));
  k<<<dim3(nrec, by), 32 * kWgWarps, smem, s>>>(p);
  e = cudaGetLastError();
  return e != cudaSuccess ? e : sum_records(p.part, nrec, CI, CO, p.cin, p.cout, CO, dw, db, s);
}

template <int CI, int CO, int STRIDE>
cudaError_t launch_dgrad(BwdParams p, int num_sms, cudaStream_t s) {
  const int by = p.cin / CI;
  size_t smem = 0;
  auto bytes = [](const BwdParams& q) { return (size_t)27 * CI * (2 * CO + 16) + (size_t)q.rows * (6 * CO + 16); };
  auto per_sm = [](size_t need) { return 2 * (need + 1024) <= (size_t)kSmemMax ? 2 : 1; };
  if (p.cin % CI || p.cout != CO ||
      !pick_brick(p, 1, kDgThreads / 32 / (CI / 16), by, num_sms, bytes, per_sm, smem))
    return cudaErrorInvalidValue;
  auto k = k_dgrad<CI, CO, STRIDE>;
  cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemMax);
  if (e != cudaSuccess) return e;
  k<<<dim3(std::min(p.nb[0] * p.nb[1] * p.nb[2], std::max(1, per_sm(smem) * num_sms / by)), by), kDgThreads, smem,
      s>>>(p);
  return cudaGetLastError();
}

int tiles_1(const BwdParams& p) {
  return ceil_div(p.vd[0], kOX) * ceil_div(p.vd[1], kOY) * ceil_div(p.vd[2], kOZ);
}

}  // namespace

cudaError_t conv3_dgrad(const ConvDesc& d, const float* dout, const __nv_bfloat16* y, const float* add, float* dx,
                        int num_sms, cudaStream_t s) {
  BwdParams p = bwd_params(d, dout, y);
  p.add = add;
  p.dx = dx;
  if (d.cb != 0) return cudaErrorInvalidValue;
  if (d.cout == 1 && d.ca == 16 && d.stride == 1 && !y && !add) {
    k_dgrad_1<<<tiles_1(p), kOX * kOY * kOZ, 0, s>>>(p);
    return cudaGetLastError();
  }
  if (d.stride == 1) {
    if (d.ca == 16 && d.cout == 16) return launch_dgrad<16, 16, 1>(p, num_sms, s);
    if (d.ca % 32 == 0 && d.cout == 16) return launch_dgrad<32, 16, 1>(p, num_sms, s);
    if (d.ca % 32 == 0 && d.cout == 32) return launch_dgrad<32, 32, 1>(p, num_sms, s);
    if (d.ca % 32 == 0 && d.cout == 64) return launch_dgrad<32, 64, 1>(p, num_sms, s);
  } else if (d.stride == 2) {
    if (d.ca == 16 && d.cout == 32) return launch_dgrad<16, 32, 2>(p, num_sms, s);
    if (d.ca % 32 == 0 && d.cout == 64) return launch_dgrad<32, 64, 2>(p, num_sms, s);
  }
  return cudaErrorInvalidValue;
}

long long conv3_wgrad_words(int num_sms) {
  return (long long)kWgPerSm * num_sms * (27 * 32 * 32 + 32);
}

cudaError_t conv3_wgrad(const ConvDesc& d, const float* dout, const __nv_bfloat16* y, float* dw, float* db,
                        float* work, int num_sms, cudaStream_t s) {
  BwdParams p = bwd_params(d, dout, y);
  p.part = work;
  if (d.cb != 0 || !db) return cudaErrorInvalidValue;
  const bool first = d.ca == 1 && d.cout == 16, last = d.ca == 16 && d.cout == 1 && !y;
  if (d.stride == 1 && (first || last)) {
    const int nrec = std::min(tiles_1(p), kWgPerSm * num_sms);
    if (first)
      k_wgrad_1<true><<<nrec, kW1Threads, 0, s>>>(p);
    else
      k_wgrad_1<false><<<nrec, kW1Threads, 0, s>>>(p);
    const cudaError_t e = cudaGetLastError();
    // both layers' weights are [27][16]
    return e != cudaSuccess ? e : sum_records(p.part, nrec, 1, 16, 1, 16, d.cout, dw, db, s);
  }
  if (d.stride == 1) {
    if (d.ca == 16 && d.cout == 16) return launch_wgrad<16, 16, 1>(p, dw, db, num_sms, s);
    if (d.ca % 32 == 0 && d.cout == 16) return launch_wgrad<32, 16, 1>(p, dw, db, num_sms, s);
    if (d.ca % 32 == 0 && d.cout % 32 == 0) return launch_wgrad<32, 32, 1>(p, dw, db, num_sms, s);
  } else if (d.stride == 2) {
    if (d.ca % 16 == 0 && d.cout % 32 == 0) return launch_wgrad<16, 32, 2>(p, dw, db, num_sms, s);
  }
  return cudaErrorInvalidValue;
}

}  // namespace cfd
