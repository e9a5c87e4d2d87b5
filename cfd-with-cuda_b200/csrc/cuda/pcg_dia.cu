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
// - The products are split evenly over the block's warps in groups of 16
//   taps, whatever the number of slices: a warp owns a contiguous run of groups,
//   and a slice that several warps share has a partial sum from each, added in
//   warp order.  The coefficients of the next group are loaded while the current
//   one multiplies, and those of the first while the block waits for its
//   neighbours.
// - The dot products of an iteration are posted before its SpMV.  One warp
//   collects them and forms alpha and beta: beside the SpMV, which it then takes
//   no part in, up to 12 slices per block (BESIDE), after it above that, where a
//   sixteenth of the loads in flight is worth more (the first form below / after /
//   beside: 40^3, 14.5 slices, 14.5 / - / 15.2, 48^3 20.3 / 19.6 / 19.1 to 19.6, 64^3
//   41.0 / 40.0 / 44.1 on one device).  The other warps wait only for
//   the blocks whose rows they gather.  Every wait of this form is bounded.
//
// What bounds it: the coefficient stream on large grids; the latency of the
// wait for the neighbours, the gathers and the block sums on small ones.  Measured
// per iteration on cavities of n^3 elements, against k_pcg on the SELL-32 form (us):
//   n                     12    14    16    20    24    28    32    40    48    64
//   k_pcg                             19.9        20.4        21.2        42    77.5
//   sums after the SpMV,
//   scalars by all        5.7   6.4   6.6   7.1   8.4   9.7   10.4  15.0  19.9  44.0
//   k_pcg_dia             5.9   5.8   6.1   6.0   7.8   8.1   9.4         19.6  43
// of which L2 residence of part of the coefficients (dia.cuh) gave 13.0 -> 10.6
// at n = 32 and 46 -> 43.7 at 64: the copy rate on the 275 MB.  Half
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
constexpr int kBesideSlices = 12;  // slices of a block up to which one of its warps only reduces

size_t dia_smem(int slices) {
  return (size_t)slices * 32 * kDiaVecs * sizeof(double) + dia_slot_bytes(slices);
}

// BESIDE: the last warp only reduces, beside the SpMV; else the first one does, after it.
template <bool BESIDE>
__global__ void __launch_bounds__(kDiaThreads, 1) k_pcg_dia(PcgDiaArgs a) {
  constexpr int PROD = BESIDE ? kDiaWarps - 1 : kDiaWarps;  // warps of the products and the rows
  extern __shared__ double sv[];
  __shared__ int soff[kDiaMaxTaps + kDiaGroup];
  __shared__ double sred[4];  // alpha, beta, ||r||, ||b||
  __shared__ int sstat, sdead;
  const int n = a.d.n, nslices = (n + 31) >> 5, G = gridDim.x;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const bool sums = warp == (BESIDE ? PROD : 0);  // the warp of the reductions
  const bool rows = warp < PROD;
  const int R = 32 * ((int)((long long)nslices * (blockIdx.x + 1) / G) - (int)((long long)nslices * blockIdx.x / G));
  double *r = sv, *u = r + R, *w = u + R, *z = w + R, *q = z + R, *s = q + R, *p = s + R, *x = p + R, *m = x + R,
         *dinv = m + R;
  const DiaRows M = dia_rows(a.d, soff, dinv + R, kPcgKeepBytes, PROD);
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
  if (threadIdx.x == 0) sdead = 0;
  double bb = 0;
  for (int i = threadIdx.x; i < nr && rows; i += 32 * PROD) {
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
  for (int i = threadIdx.x; i < nr && rows; i += 32 * PROD) {
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

  double bnorm = 0, tol = 0, gam_old = 1, alpha_old = 1;  // the reductions' warp
  int its = 0, status;
  for (int i = 0;; i++) {
    if (rows) {
      // n_i = Z m_i  (neighbours' m_i published at phase i + 2)
      if (alive) alive = bs.wait_nb<BESIDE ? 32 * PROD : 0>((unsigned)i + 2 + a.nb_extra);
      if (alive)
        M.multiply(warp, lane, mb[i & 1], c);
      else if (threadIdx.x == 0)
        sdead = 1;
    }
    if (sums) {
      // reduction of iteration i, posted before the SpMV
      double red[4];
      const bool ok = bs.warp_red<4>((unsigned)(i + 1) * (unsigned)G + a.red_extra, a.part + (size_t)(i & 1) * 4 * G, red);
      if (i == 0) {
        bnorm = sqrt(red[3]);
        tol = a.rtol * bnorm;
      }
      const double rn = sqrt(red[2]);
      int st = -1;
      if (!ok)
        st = 3;
      else if (!isfinite(bnorm) || !isfinite(rn))
        st = 2;
      else if (bnorm == 0.0 || rn <= tol)
        st = 0;
      else if (i >= a.maxit)
        st = 1;
      const double gam = red[0], del = red[1];
      const double beta = i > 0 ? gam / gam_old : 0.0;
      const double alpha = i > 0 ? gam / (del - beta * gam / alpha_old) : gam / del;
      gam_old = gam;
      alpha_old = alpha;
      if (lane == 0) {
        sred[0] = alpha;
        sred[1] = beta;
        sred[2] = bnorm == 0.0 ? 0.0 : rn;
        sred[3] = bnorm;
        sstat = st;
      }
    }
    __syncthreads();
    status = sdead ? 3 : sstat;
    if (status >= 0) break;
    const double alpha = sred[0], beta = sred[1];
    double* mnext = mb[(i + 1) & 1];
    double d[4] = {0, 0, 0, 0};
    for (int k = threadIdx.x; k < nr && rows; k += 32 * PROD) {
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
  const bool zero = status == 0 && sred[3] == 0.0;
  for (int k = threadIdx.x; k < nr && rows; k += 32 * PROD) a.x[r0 + k] = zero ? 0.0 : x[k];
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    a.result[0] = its;
    a.result[1] = sred[3] > 0 ? sred[2] / sred[3] : 0.0;
    a.result[2] = status;
    a.result[3] = sred[3];
  }
}

// ---- small grids: the same iteration in one cluster of up to 16 blocks ----
// Block k of C owns slices as above, one row per thread with its ten vector
// entries in registers; the whole matrix stays in the cluster, in registers where
// a warp has one group of taps (ONE), else in shared memory.  Each block keeps the
// m it gathers (double buffered) in shared memory: a block writes its rows of m
// straight into the copies of the blocks that gather them, and its partial sums
// into every block, and one hardware cluster barrier per iteration covers both.
// No flag, no poll, no trip to L2.  That barrier has no time limit: the blocks of a
// cluster are on the chip together, each arrives at every barrier (all take the same
// decisions, from the same sums in the same order), and the iterations are limited.  A seventeenth warp adds the partials (in the
// same order in every block, so all take the same decisions) and forms alpha and
// beta beside the product.  Bound by latency: the product's chain, the row sums,
// the block's sums and the barrier.  us per iteration, launch included, on cavities of
// n^3 elements (the matrix of 12^3 no longer fits the shared memory of 16 blocks;
// with part of it streamed from L2 13^3 took 5.8 against 5.3, 16^3 8.1 against 7.1):
//   n              2    4    6    8    10   11
//   k_pcg_dia      4.6  5.0  4.7  4.9  5.7  5.1
//   k_pcg_cluster  2.4  2.3  2.4  2.5  2.9  3.1
// Vectors in shared memory and the scalars in every thread instead: 3.4 to 4.5.
__device__ __forceinline__ unsigned cluster_addr(const void* p, int rank) {
  unsigned r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_u32(p)), "r"(rank));
  return r;
}
__device__ __forceinline__ void st_cluster(unsigned addr, double v) {
  asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(addr), "d"(v) : "memory");
}
__device__ __forceinline__ void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}
constexpr int kClMax = 16;                      // blocks of a cluster at most
constexpr int kClThreads = kDiaThreads + 32;    // the product's warps and the scalars' one

// Groups of taps of a warp at most.
int cluster_groups(int slices, int ntap) {
  return (slices * ((ntap + kDiaGroup - 1) / kDiaGroup) + kDiaWarps - 1) / kDiaWarps;
}
// Shared memory of a block: slots of its slices, two copies of m, the
// coefficients where a warp has more than one group.
size_t cluster_smem(int n, int slices, int ntap) {
  const int groups = cluster_groups(slices, ntap);
  return dia_slot_bytes(slices) + 2 * (size_t)n * sizeof(double) +
         (groups > 1 ? (size_t)groups * kDiaWarps * kDiaGroup * 32 * sizeof(double) : 0);
}

template <bool ONE>
__global__ void __launch_bounds__(kClThreads, 1) k_pcg_cluster(PcgDiaArgs a, int groups) {
  extern __shared__ double sv[];
  __shared__ __align__(16) int soff[kDiaMaxTaps + kDiaGroup];
  __shared__ double spart[2][kClMax][4], swarp[kDiaWarps][4], sred[4];
  __shared__ int sstat;
  const int n = a.d.n, nslices = (n + 31) >> 5, C = gridDim.x, rank = blockIdx.x;
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
  const int s0 = (int)((long long)nslices * rank / C), ns = (int)((long long)nslices * (rank + 1) / C) - s0;
  const int ng = (a.d.ntap + kDiaGroup - 1) / kDiaGroup, T = ns * ng;
  const int g0 = T * min(warp, kDiaWarps) / kDiaWarps, g1 = T * min(warp + 1, kDiaWarps) / kDiaWarps;
  // the copies of m lie at the same place in every block
  double* const mb[2] = {sv, sv + n};
  double(*const slot)[32] = reinterpret_cast<double(*)[32]>(sv + 2 * n);
  double* const res = sv + 2 * n + (ns + kDiaWarps) * 32 + (size_t)warp * groups * kDiaGroup * 32 + lane;
  const int r0 = 32 * s0, nr = min(32 * ns, n - r0), reach = a.d.reach;
  const bool mine = t < nr;
  const int row = r0 + t;
  auto block_of = [&](int i) { return (int)(((long long)C * ((i >> 5) + 1) - 1) / nslices); };
  const int lo = block_of(max(r0 - reach, 0)), hi = block_of(min(r0 + nr - 1 + reach, n - 1));
  // warps that share the thread's row
  const int w0 = warp < ns ? (kDiaWarps * (warp * ng + 1) - 1) / T : 0;
  const int w1 = warp < ns ? (kDiaWarps * (warp + 1) * ng - 1) / T : -1;

  for (int k = t; k < kDiaMaxTaps + kDiaGroup; k += kClThreads) soff[k] = k < a.d.ntap ? a.d.off[k] : 0;
  for (int k = t; k < n; k += kClThreads) {
    mb[0][k] = a.warm ? a.x[k] : 0.0;
    mb[1][k] = 0.0;
  }
  // with fewer groups than warps some slots are never written
  for (int k = t; k < (ns + kDiaWarps) * 32; k += kClThreads) slot[0][k] = 0.0;
  double c[kDiaGroup];
  for (int g = g0; g < g1; g++) {
    const int sl = g / ng, t0 = (g - sl * ng) * kDiaGroup;
    const double* p = a.d.coef + ((size_t)(s0 + sl) * a.d.ntap + t0) * 32 + lane;
#pragma unroll
    for (int k = 0; k < kDiaGroup; k++) {
      c[k] = t0 + k < a.d.ntap ? __ldg(p + 32 * k) : 0.0;
      if (!ONE) res[((g - g0) * kDiaGroup + k) * 32] = c[k];
    }
  }
  __syncthreads();

  auto product = [&](const double* v) {
    if (g0 >= g1) return;
    int sl = g0 / ng;
    double acc[4] = {0, 0, 0, 0};
    for (int g = g0; g < g1; g++) {
      const int t0 = (g - sl * ng) * kDiaGroup, i0 = (s0 + sl) * 32, i = i0 + lane;
      const double* rs = res + (g - g0) * kDiaGroup * 32;
      const bool inside = i0 >= reach && i0 + 31 + reach < n;
      double x[kDiaGroup];
#pragma unroll
      for (int k = 0; k < kDiaGroup; k += 4) {
        const int4 o = *reinterpret_cast<const int4*>(soff + t0 + k);
        const int j[4] = {i + o.x, i + o.y, i + o.z, i + o.w};
#pragma unroll
        for (int e = 0; e < 4; e++) x[k + e] = v[inside ? j[e] : min(max(j[e], 0), n - 1)];
      }
#pragma unroll
      for (int k = 0; k < kDiaGroup; k++) acc[k & 3] += (ONE ? c[k] : rs[k * 32]) * x[k];
      if (g + 1 == g1 || g + 1 == (sl + 1) * ng) {
        slot[sl + warp][lane] = (acc[0] + acc[1]) + (acc[2] + acc[3]);
        acc[0] = acc[1] = acc[2] = acc[3] = 0;
        sl++;
      }
    }
  };
  auto row_sum = [&]() {
    double y[4] = {0, 0, 0, 0};
    for (int w = w0; w <= w1; w += 4)
#pragma unroll
      for (int e = 0; e < 4; e++)
        if (w + e <= w1) y[e] += slot[warp + w + e][lane];
    return (y[0] + y[1]) + (y[2] + y[3]);
  };
  auto send = [&](double* copy, double v) {  // the thread's m into the copies that gather it
    for (int k = lo; k <= hi; k++) st_cluster(cluster_addr(copy + row, k), v);
  };
  // Sum over k < count of the four values at v[k]: lane l holds that of value l & 3.
  auto sum4 = [&](const double (*v)[4], int count) {
    const int k = lane >> 2;
    double y = (k < count ? v[k][lane & 3] : 0.0) + (k + 8 < count ? v[k + 8][lane & 3] : 0.0);
#pragma unroll
    for (int o = 4; o < 32; o <<= 1) y += __shfl_xor_sync(0xffffffffu, y, o);
    return y;
  };
  auto post = [&](double (&v)[4], int buf) {  // the block's partial sums into every block
    if (warp < ns) {
#pragma unroll
      for (int k = 0; k < 4; k++) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v[k] += __shfl_xor_sync(0xffffffffu, v[k], o);
        if (lane == 0) swarp[warp][k] = v[k];
      }
    }
    __syncthreads();
    if (warp == kDiaWarps) {
      const double y = sum4(swarp, ns);
      for (int k = lane >> 2; k < C; k += 8) st_cluster(cluster_addr(&spart[buf][rank][lane & 3], k), y);
    }
  };

  if (a.warm) product(mb[0]);
  cluster_barrier();  // every block runs and has set up its copies
  double r = 0, u = 0, w = 0, z = 0, q = 0, s = 0, p = 0, x = 0, m = 0, dinv = 0;
  double v[4] = {0, 0, 0, 0};
  if (mine) {
    const double bi = a.b[row];
    dinv = a.dinv[row];
    r = a.warm ? bi - row_sum() : bi;
    u = r * dinv;
    x = a.warm ? mb[0][row] : 0.0;
    send(mb[1], u);
    v[3] = bi * bi;
  }
  cluster_barrier();
  product(mb[1]);
  __syncthreads();
  if (mine) {
    w = row_sum();
    m = w * dinv;
    send(mb[0], m);
    v[0] = r * u;
    v[1] = w * u;
    v[2] = r * r;
  }
  post(v, 0);
  cluster_barrier();

  // the scalars' warp; the reciprocals are formed off the critical path
  double bnorm = 0, tol = 0, gam_old = 1, igam = 0, ialpha = 0;
  int its = 0;
  for (int i = 0;; i++) {
    if (warp == kDiaWarps) {
      const double y = sum4(spart[i & 1], C);
      const double gam = __shfl_sync(0xffffffffu, y, 0), del = __shfl_sync(0xffffffffu, y, 1);
      const double rn = sqrt(__shfl_sync(0xffffffffu, y, 2));
      if (i == 0) {
        bnorm = sqrt(__shfl_sync(0xffffffffu, y, 3));
        tol = a.rtol * bnorm;
      }
      int st = -1;
      if (!isfinite(bnorm) || !isfinite(rn))
        st = 2;
      else if (bnorm == 0.0 || rn <= tol)
        st = 0;
      else if (i >= a.maxit)
        st = 1;
      // i = 0: igam = 0; the reciprocal of a gam near the smallest numbers overflows
      const double beta = gam_old > 1e-290 ? gam * igam : gam / gam_old;
      const double alpha = gam / (del - beta * gam * ialpha);
      if (lane == 0) {
        sred[0] = alpha;
        sred[1] = beta;
        sred[2] = bnorm == 0.0 ? 0.0 : rn;
        sred[3] = bnorm;
        sstat = st;
      }
      gam_old = gam;
      igam = 1.0 / gam;
      ialpha = 1.0 / alpha;
    } else {
      product(mb[i & 1]);
    }
    __syncthreads();
    if (sstat >= 0) break;
    double d[4] = {0, 0, 0, 0};
    if (mine) {
      const double alpha = sred[0], beta = sred[1];
      z = row_sum() + beta * z;
      q = m + beta * q;
      s = w + beta * s;
      p = u + beta * p;
      x += alpha * p;
      r -= alpha * s;
      u -= alpha * q;
      w -= alpha * z;
      m = w * dinv;
      send(mb[(i + 1) & 1], m);
      d[0] = r * u;
      d[1] = w * u;
      d[2] = r * r;
    }
    its++;
    post(d, (i + 1) & 1);
    cluster_barrier();
  }
  if (mine) a.x[row] = sstat == 0 && sred[3] == 0.0 ? 0.0 : x;
  if (rank == 0 && t == 0) {
    a.result[0] = its;
    a.result[1] = sred[3] > 0 ? sred[2] / sred[3] : 0.0;
    a.result[2] = sstat;
    a.result[3] = sred[3];
  }
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
  // three slices per block until every SM has one: fewer blocks wait on fewer
  // neighbours and arrivals.  us per iteration with 1 / 2 / 3 / 4 slices: 12^3 (69
  // slices) 7.5 / 6.2 / 5.9 / 6.8, 13^3 5.3 / 5.4 / 5.6 / 6.1, 14^3 6.9 / 6.1 / 5.8 /
  // 6.9, 16^3 8.0 / 6.2 / 6.6 / 7.6, 20^3 6.4 / 6.3 / 5.5 / 6.6, 22^3 7.6 / 7.5 / 6.4 /
  // 8.4.  Smaller grids, where no cluster is to be had: one slice per block (729 rows
  // on 23 blocks).
  const int ns = (n + 31) / 32, grid = std::min(sms, ns <= 64 ? ns : (ns + 2) / 3);
  return dia_smem((ns + grid - 1) / grid) <= (size_t)kDiaMaxSmem ? grid : 0;
}

namespace {
using ClusterKernel = void (*)(PcgDiaArgs, int);
// Launch of a cluster of C blocks; false when they cannot hold the matrix.
bool cluster_config(int n, int ntap, int C, ClusterKernel& k, int& groups, cudaLaunchConfig_t& cfg,
                    cudaLaunchAttribute& attr) {
  const int ns = (n + 31) / 32, slices = (ns + C - 1) / C;
  groups = cluster_groups(slices, ntap);
  k = groups == 1 ? k_pcg_cluster<true> : k_pcg_cluster<false>;
  cfg = cudaLaunchConfig_t{};
  cfg.gridDim = dim3(C);
  cfg.blockDim = dim3(kClThreads);
  cfg.dynamicSmemBytes = cluster_smem(n, slices, ntap);
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = C;
  attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  // a row per thread of the product's warps, and the shared memory of a block
  return C <= ns && slices <= kDiaWarps && cfg.dynamicSmemBytes <= (size_t)kDiaMaxSmem &&
         cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, kDiaMaxSmem) == cudaSuccess &&
         cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess;
}
}  // namespace

int pcg_cluster_blocks(int n, int ntap) {
  if (n < 1 || ntap < 1 || ntap > kDiaMaxTaps) return 0;
  const int ns = (n + 31) / 32;
  int C = kClMax;
  while (C > ns) C /= 2;
  ClusterKernel k;
  int groups = 0, active = 0;
  cudaLaunchConfig_t cfg;
  cudaLaunchAttribute attr;
  // not every device (or partition of one) has room for a cluster of 16
  const bool ok = cluster_config(n, ntap, C, k, groups, cfg, attr) &&
                  cudaOccupancyMaxActiveClusters(&active, k, &cfg) == cudaSuccess && active >= 1;
  if (!ok) cudaGetLastError();
  return ok ? C : 0;
}

cudaError_t launch_pcg_dia(const PcgDiaArgs& a, int grid, int cluster, cudaStream_t s) {
  const int ns = (a.d.n + 31) / 32;
  if (cluster > 0) {
    ClusterKernel k;
    int groups = 0;
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute attr;
    if (cluster > kClMax || a.d.ntap < 1 || a.d.ntap > kDiaMaxTaps ||
        !cluster_config(a.d.n, a.d.ntap, cluster, k, groups, cfg, attr))
      return cudaErrorInvalidValue;
    cfg.stream = s;
    return cudaLaunchKernelEx(&cfg, k, a, groups);
  }
  if (grid < 1 || grid > ns || a.d.ntap < 1 || a.d.ntap > kDiaMaxTaps) return cudaErrorInvalidValue;
  const int slices = (ns + grid - 1) / grid;
  const void* k = slices <= kBesideSlices ? (const void*)k_pcg_dia<true> : (const void*)k_pcg_dia<false>;
  cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, kDiaMaxSmem);
  if (e != cudaSuccess) return e;
  PcgDiaArgs args = a;
  void* params[] = {&args};
  return cudaLaunchCooperativeKernel(k, dim3(grid), dim3(kDiaThreads), params, dia_smem(slices), s);
}

int dia_apply_grid(int n, int num_sms) { return dia_blocks(n, num_sms); }

cudaError_t launch_dia_mark(int n, const int* rp, const int* col, unsigned char* mark, int num_sms, cudaStream_t s) {
  k_dia_mark<<<std::max(1, std::min((n + 255) / 256, 8 * num_sms)), 256, 0, s>>>(n, rp, col, mark);
  return cudaGetLastError();
}

cudaError_t launch_dia_fill(const DiaArgs& d, const int* rp, const int* col, const double* val, double* coef,
                            int num_sms, cudaStream_t s) {
  cudaError_t e = cudaMemsetAsync(coef, 0, dia_elems(d.n, d.ntap) * sizeof(double), s);
  if (e != cudaSuccess) return e;
  k_dia_fill<<<std::max(1, std::min((d.n + 127) / 128, 16 * num_sms)), 128, 0, s>>>(d, rp, col, val, coef);
  return cudaGetLastError();
}

}  // namespace cfd
