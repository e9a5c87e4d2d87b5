// Jacobi-PCG on the pressure operator stored by offsets: the pipelined
// iteration of pcg.cu (Ghysels & Vanroose 2014) as one persistent cooperative
// kernel per solve, FP64, for matrices whose entries lie on at most
// kDiaMaxTaps diagonals (pressure nodes numbered along the axes of a structured
// grid: 125 diagonals).
//
// - No column indices: 8 bytes per entry instead of 12, and the gathers of the
//   vector are contiguous across a warp.
// - One block of 16 warps per SM owns a contiguous range of 32-row slices, and
//   all ten vectors of its rows stay in shared memory; only m, which other
//   blocks gather, is published to global memory.
// - The products are split evenly over the block's warps in groups of 16 taps,
//   whatever the number of slices: a warp owns a contiguous run of groups, and
//   a slice that several warps share has a partial sum from each, added in
//   warp order.  So a grid of one slice per block (729 rows) still has 8 warps
//   at work on it.  The coefficients of the next group are loaded while the
//   current one multiplies, and those of the first while the block waits for
//   its neighbours.
// - The dot products of an iteration are posted before its SpMV and
//   collected after it; blocks wait only for the blocks whose rows they
//   gather.  Every wait is bounded.
//
// What bounds it: the coefficient stream on large grids; the latency of the
// two waits, the gathers and the block sums on small ones.  Measured per
// iteration on cavities of n^3 elements, against k_pcg on the SELL-32 form (us):
//   n          4     8     16    24    32    48    64
//   k_pcg      15.8  17.0  19.9  20.4  21.2  42    77.5
//   k_pcg_dia  4.7   5.1   6.5   8.4   10.6  19.6  43.7
// of which L2 residence of part of the coefficients (dia.cuh) gave 13.0 -> 10.6
// at n = 32 and 46 -> 43.7 at 64: 0.98 of the copy rate on the 275 MB.  Half
// the coefficients (Z is symmetric) would halve that, but the mirror reads of
// other blocks' rows come from L2 at about the same rate.  Keeping the
// coefficients of small grids in the L1 changed nothing there and cost the
// large ones 20 us (the loads no longer run ahead).
#include <algorithm>

#include "block_sync.cuh"
#include "dia.cuh"
#include "kernels.h"

namespace cfd {

namespace {

constexpr int kDiaVecs = 10;   // r u w z q s p x m dinv
constexpr int kDiaMaxSmem = 224 * 1024;

size_t dia_smem(int slices) {
  return (size_t)slices * 32 * kDiaVecs * sizeof(double) + dia_slot_bytes(slices);
}

__global__ void __launch_bounds__(kDiaThreads, 1) k_pcg_dia(PcgDiaArgs a) {
  extern __shared__ double sv[];
  __shared__ int soff[kDiaMaxTaps + kDiaGroup];
  const int n = a.d.n, nslices = (n + 31) >> 5, G = gridDim.x;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int R = 32 * ((int)((long long)nslices * (blockIdx.x + 1) / G) - (int)((long long)nslices * blockIdx.x / G));
  double *r = sv, *u = r + R, *w = u + R, *z = w + R, *q = z + R, *s = q + R, *p = s + R, *x = p + R, *m = x + R,
         *dinv = m + R;
  const DiaRows M = dia_rows(a.d, soff, dinv + R, kPcgKeepBytes);
  const int r0 = 32 * M.s0, nr = min(R, n - r0), reach = a.d.reach;

  auto block_of = [&](int row) { return (int)(((long long)G * ((row >> 5) + 1) - 1) / nslices); };
  BlockSync bs;
  bs.cnt = a.sync;
  bs.prog = a.sync + 1;
  bs.lo = block_of(max(r0 - reach, 0));
  bs.hi = block_of(min(r0 + nr - 1 + reach, n - 1));
  bs.err = a.err;
  bs.timeout_ns = a.timeout_ns;
  double* mb[2] = {a.mb, a.mb + n};

  double c[kDiaGroup];
  if (M.g0 < M.g1) M.load(M.g0, lane, c);
  __syncthreads();  // soff, slots
  // r = b - Z x0, u = D^-1 r (published in mb[1])
  if (a.warm) {
    M.multiply(warp, lane, a.x, c);
    __syncthreads();
  }
  double bb = 0;
  for (int i = threadIdx.x; i < nr; i += kDiaThreads) {
    const double bi = a.b[r0 + i], di = a.dinv[r0 + i];
    const double ri = a.warm ? bi - M.row(i >> 5, i & 31) : bi;
    r[i] = ri;
    dinv[i] = di;
    u[i] = ri * di;
    x[i] = a.warm ? a.x[r0 + i] : 0.0;
    z[i] = q[i] = s[i] = p[i] = 0.0;
    mb[1][r0 + i] = ri * di;
    bb += bi * bi;
  }
  bs.publish(1);
  bool alive = bs.wait_nb(1);
  // w = Z u, m0 = D^-1 w, dots of iteration 0
  if (alive) M.multiply(warp, lane, mb[1], c);
  __syncthreads();
  double v[4] = {0, 0, 0, bb};
  for (int i = threadIdx.x; i < nr; i += kDiaThreads) {
    const double wi = alive ? M.row(i >> 5, i & 31) : 0.0, mi = wi * dinv[i];
    w[i] = wi;
    m[i] = mi;
    mb[0][r0 + i] = mi;
    v[0] += r[i] * u[i];
    v[1] += wi * u[i];
    v[2] += r[i] * r[i];
  }
  block_partials<4>(v, a.part);
  bs.publish_arrive(2);

  double bnorm = 0, tol = 0, rn = 0, gam_old = 1, alpha_old = 1;
  int its = 0, status = 1;
  for (int i = 0;; i++) {
    // n_i = Z m_i  (neighbours' m_i published at phase i + 2)
    if (alive) alive = bs.wait_nb((unsigned)i + 2);
    if (alive) M.multiply(warp, lane, mb[i & 1], c);
    // reduction of iteration i (posted before the SpMV); its barriers also
    // order the slots' writes before the reads below
    double red[4];
    if (!alive || !bs.wait_red<4>((unsigned)(i + 1) * (unsigned)G, a.part + (size_t)(i & 1) * 4 * G, red)) {
      status = 3;
      break;
    }
    if (i == 0) {
      bnorm = sqrt(red[3]);
      tol = a.rtol * bnorm;
    }
    rn = sqrt(red[2]);
    if (!isfinite(bnorm) || !isfinite(rn)) { status = 2; break; }
    if (bnorm == 0.0) {
      for (int k = threadIdx.x; k < nr; k += kDiaThreads) x[k] = 0.0;
      rn = 0;
      status = 0;
      break;
    }
    if (rn <= tol) { status = 0; break; }
    if (its >= a.maxit) { status = 1; break; }
    const double gam = red[0], del = red[1];
    const double beta = i > 0 ? gam / gam_old : 0.0;
    const double alpha = i > 0 ? gam / (del - beta * gam / alpha_old) : gam / del;
    gam_old = gam;
    alpha_old = alpha;
    double* mnext = mb[(i + 1) & 1];
    double d[4] = {0, 0, 0, 0};
    for (int k = threadIdx.x; k < nr; k += kDiaThreads) {
      const double zi = M.row(k >> 5, k & 31) + beta * z[k];
      const double qi = m[k] + beta * q[k];
      const double si = w[k] + beta * s[k];
      const double pi = u[k] + beta * p[k];
      const double ri = r[k] - alpha * si;
      const double ui = u[k] - alpha * qi;
      const double wi = w[k] - alpha * zi;
      const double mi = wi * dinv[k];
      z[k] = zi;
      q[k] = qi;
      s[k] = si;
      p[k] = pi;
      x[k] += alpha * pi;
      r[k] = ri;
      u[k] = ui;
      w[k] = wi;
      m[k] = mi;
      mnext[r0 + k] = mi;
      d[0] += ri * ui;
      d[1] += wi * ui;
      d[2] += ri * ri;
    }
    its++;
    block_partials<4>(d, a.part + (size_t)((i + 1) & 1) * 4 * G);
    bs.publish_arrive((unsigned)i + 3);
  }
  __syncthreads();
  for (int k = threadIdx.x; k < nr; k += kDiaThreads) a.x[r0 + k] = x[k];
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    a.result[0] = its;
    a.result[1] = bnorm > 0 ? rn / bnorm : 0.0;
    a.result[2] = status;
    a.result[3] = bnorm;
  }
}

// r = b - Z x in FP64, rf = (float) r, per-block partial of r^2: one pass over
// the coefficients, bound by their stream (us on the 64^3 cavity: 68 on the
// SELL-32 form, 47 here).
__global__ void __launch_bounds__(kDiaThreads, 1) k_residual_dia(DiaArgs d, const double* __restrict__ b,
                                                                 const double* __restrict__ x, double* r, float* rf,
                                                                 double* part, const int* when) {
  if (when && *when == 0) return;
  extern __shared__ double sv[];
  __shared__ int soff[kDiaMaxTaps + kDiaGroup];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const DiaRows M = dia_rows(d, soff, sv, 0.0);
  double c[kDiaGroup];
  if (M.g0 < M.g1) M.load(M.g0, lane, c);
  __syncthreads();
  M.multiply(warp, lane, x, c);
  __syncthreads();
  const int r0 = 32 * M.s0, nr = min(32 * M.ns, d.n - r0);
  double v[1] = {0};
  for (int i = threadIdx.x; i < nr; i += kDiaThreads) {
    const double ri = b[r0 + i] - M.row(i >> 5, i & 31);
    r[r0 + i] = ri;
    if (rf) rf[r0 + i] = (float)ri;
    v[0] += ri * ri;
  }
  block_sum<1>(v);
  if (threadIdx.x == 0) part[blockIdx.x] = v[0];
}

__global__ void k_dia_mark(int n, const int* __restrict__ rp, const int* __restrict__ col, unsigned char* mark) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    for (int k = rp[i]; k < rp[i + 1]; k++) {
      unsigned char* p = mark + (col[k] - i + n - 1);
      if (!*p) *p = 1;
    }
}

__global__ void k_dia_fill(DiaArgs d, const int* __restrict__ rp, const int* __restrict__ col,
                           const double* __restrict__ val, double* coef) {
  __shared__ int soff[kDiaMaxTaps];
  for (int k = threadIdx.x; k < d.ntap; k += blockDim.x) soff[k] = d.off[k];
  __syncthreads();
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < d.n; i += gridDim.x * blockDim.x) {
    int t = 0;  // columns ascend, so the taps do too
    for (int k = rp[i]; k < rp[i + 1]; k++) {
      const int o = col[k] - i;
      while (t < d.ntap && soff[t] < o) t++;
      if (t < d.ntap && soff[t] == o) coef[((size_t)(i >> 5) * d.ntap + t) * 32 + (i & 31)] = val[k];
    }
  }
}

}  // namespace

int pcg_dia_grid(int n, int device) {
  int sms = 0;
  if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess || sms < 1) return 0;
  // one slice per block up to 96 slices, then three until every SM has a block:
  // fewer blocks wait on fewer neighbours and arrivals (16^3, 154 slices: 8.0 us
  // per iteration on 148 blocks, 6.7 on 51; 20^3, 290 slices: 9.2 on 148, 7.8 on
  // 96; 12^3, 69 slices: 5.4 on 69, 6.0 on 23)
  const int ns = (n + 31) / 32, grid = ns <= 96 ? std::min(sms, ns) : std::min(sms, (ns + 2) / 3);
  return dia_smem((ns + grid - 1) / grid) <= (size_t)kDiaMaxSmem ? grid : 0;
}

cudaError_t launch_pcg_dia(const PcgDiaArgs& a, int grid, cudaStream_t s) {
  const int ns = (a.d.n + 31) / 32;
  if (grid < 1 || grid > ns || a.d.ntap < 1 || a.d.ntap > kDiaMaxTaps) return cudaErrorInvalidValue;
  cudaError_t e = cudaFuncSetAttribute(k_pcg_dia, cudaFuncAttributeMaxDynamicSharedMemorySize, kDiaMaxSmem);
  if (e != cudaSuccess) return e;
  PcgDiaArgs args = a;
  void* params[] = {&args};
  return cudaLaunchCooperativeKernel((const void*)k_pcg_dia, dim3(grid), dim3(kDiaThreads), params,
                                     dia_smem((ns + grid - 1) / grid), s);
}

int dia_apply_grid(int n, int num_sms) { return dia_blocks(n, num_sms); }

cudaError_t launch_residual_dia(const DiaArgs& d, const double* b, const double* x, double* r, float* rf, double* part,
                                int grid, const int* when, cudaStream_t s) {
  const int ns = (d.n + 31) / 32;
  if (grid < 1 || grid > ns || d.ntap < 1 || d.ntap > kDiaMaxTaps) return cudaErrorInvalidValue;
  cudaError_t e = cudaFuncSetAttribute(k_residual_dia, cudaFuncAttributeMaxDynamicSharedMemorySize, kDiaMaxSmem);
  if (e != cudaSuccess) return e;
  k_residual_dia<<<grid, kDiaThreads, dia_slot_bytes((ns + grid - 1) / grid), s>>>(d, b, x, r, rf, part,
                                                                                       when);
  return cudaGetLastError();
}

cudaError_t launch_dia_mark(int n, const int* rp, const int* col, unsigned char* mark, cudaStream_t s) {
  k_dia_mark<<<std::max(1, std::min((n + 255) / 256, 148 * 8)), 256, 0, s>>>(n, rp, col, mark);
  return cudaGetLastError();
}

cudaError_t launch_dia_fill(const DiaArgs& d, const int* rp, const int* col, const double* val, double* coef,
                            cudaStream_t s) {
  cudaError_t e = cudaMemsetAsync(coef, 0, dia_elems(d.n, d.ntap) * sizeof(double), s);
  if (e != cudaSuccess) return e;
  k_dia_fill<<<std::max(1, std::min((d.n + 127) / 128, 148 * 16)), 128, 0, s>>>(d, rp, col, val, coef);
  return cudaGetLastError();
}

}  // namespace cfd
