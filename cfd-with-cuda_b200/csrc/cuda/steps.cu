// Fractional-step stage kernels (step1GPUpart, step2GPU, step3GPU,
// calculate_KtimesAcc_prevGPU and the convergence norms of CUDAcodes.cu:
// 946-1121).  Each stage is one pass over its SELL-32 operator(s) with the
// elementwise work fused into the epilogue, replacing the reference's 3-6
// library SpMVs plus 2-4 elementwise kernels and the temporary
// cudaMalloc/cudaFree of every call.
//
// A warp owns a 32-row slice, lane = row, so the entry loop has a
// warp-uniform trip count, needs no shuffles, and every load of the matrix is
// a contiguous warp-wide segment.  With few slices that leaves most of the
// chip idle and each warp a serial chain of up to 125 dependent rounds of
// loads, so SPLIT warps (one block) share a slice.  FP64: warp k sums entries
// k, k + SPLIT, ..., and the partial sums are added in warp order.  FP32: the
// warps load entries and gather vector values side by side into shared
// memory, and the first warp runs the multiply-adds in entry order from
// there, so that the FP32 sums keep every bit of the unsplit row (the pressure
// of a step is sensitive to their rounding: a reordered G^T d moved it by
// 1e-6).  row_split below has the rule and the measurements.  Matrix values
// and columns are
// read with streaming (evict-first) loads so the gathered vectors stay in
// L2.  Matrix values are VT (double or float, accumulated in VT); vectors
// stay FP64.
#include <type_traits>

#include "kernels.h"

namespace cfd {

namespace {

constexpr int kRowThreads = 256;

inline int rows_grid(long long rows) {
  long long g = (rows + kRowThreads - 1) / kRowThreads;
  return (int)(g < 1 ? 1 : g);
}

// Warps per slice: the largest of 1, 2, 4, 8 with at most the rule's warps per SM over
// all slices.  Splitting pays while the chip is short of warps (a wave is 148
// x 64) or a few long rows are its tail; it costs where the epilogue, which
// one warp of the SPLIT runs, weighs as much as the row, and in FP32 where the
// trip through shared memory does.  Measured in us at SPLIT 1 / 2 / 4 / 8 on
// cavities of n^3 elements (velocity slices: 154, 1123, 3676, 8582, 16 600,
// 22 000 and 67 000 for n = 8, 16, 24, 32, 40, 44, 64; pressure slices: 23,
// 154, 489, 1124, 2154, 2848, 8583):
//                n = 8                n = 16              n = 24              n = 32 (40 FP32)    n = 44 (64 FP32)
//   FP64
//   k_step1      23 / 17 / 11 / 7.1   47 / 36 / 21 / 15   59 / 48 / 39 / 41   80 / 82 / 80 / 93   185/200/204/237
//   with K Acc   36 / 20 / 12 / 9.4   54 / 43 / 29 / 23   85 / 69 / 59 / 62   114/132/126/142     280/326/315/356
//   k_spmv_k3    18 / 18 / 10 / 6.3   38 / 37 / 20 / 14   45 / 42 / 30 / 30   63 / 62 / 60 / 63   137/143/146/152
//   k_step3      9.1/ 7.0/ 5.1/ 4.4   19 / 13 / 8.1/ 6.7  24 / 18 / 15 / 20   36 / 32 / 35 / 46   70/ 71/ 81/108
//   k_gt         44 / 22 / 12 / 7.2   81 / 41 / 22 / 12   103/ 50 / 28 / 17   104/ 55 / 33 / 26   109/ 67/ 73/ 62
//   FP32
//   k_step1      20 / 11 / 8.1/ 7.5   39 / 21 / 15 / 16   45 / 33 / 35 / 51   95 /126/144/227     373/495/583/929
//   with K Acc   19 / 16 / 11 / 10    37 / 30 / 22 / 22   46 / 52 / 54 / 68   118/197/218/297     474/758/850/1190
//   k_spmv_k3    16 / 9.9/ 7.3/ 6.2   35 / 19 / 12 / 11   39 / 26 / 24 / 33   60 / 92 / 96 /140   223/346/373/556
//   k_step3      8.4/ 6.2/ 4.9/ 4.4   15 / 9.7/ 7.2/ 11   19 / 14 / 18 / 26   39 / 51 / 67 /107   160/197/257/424
//   k_gt         26 / 23 / 13 / 7.8   55 / 46 / 24 / 14   65 / 52 / 28 / 16   67 / 57 / 36 / 37   112/126/127/129
// and k_gt in FP64 at n = 64 180 / 174 / 173 / 172, in FP32 on the duct of 24
// x 24 x 160 (3145 slices) 70 / 60 / 61 / 52.  One rule serves step 1 with and without K
// Acc_prev; with it the FP64 line would lie a little lower (n = 32: 114 unsplit, 132
// as chosen).
struct SplitRule {
  int fp64, fp32;  // warps per SM
  int least32;     // least FP32 split that pays (below it: 1)
};
constexpr SplitRule kStep1Rule{128, 32, 2}, kSpmvK3Rule{256, 100, 2}, kStep3Rule{128, 50, 2}, kGtRule{512, 192, 8};
template <class VT>
inline int row_split(long long rows, const SplitRule& rule, int num_sms) {
  const long long ns = (rows + 31) / 32, warps = (long long)num_sms * (sizeof(VT) == 8 ? rule.fp64 : rule.fp32);
  int sp = 1;
  while (sp < 8 && 2 * sp * ns <= warps) sp *= 2;
  return sizeof(VT) == 4 && sp < rule.least32 ? 1 : sp;
}
constexpr int block_threads(int split) { return split == 1 ? kRowThreads : 32 * split; }
inline int split_grid(long long rows, int sp) { return sp == 1 ? rows_grid(rows) : (int)((rows + 31) / 32); }

// What is read in order for one entry: the value(s) and the column.
template <class T>
struct KEntry {
  int c;
  T v;
};
template <class T>
struct GEntry {
  int c;
  T x, y, z;
};
// One entry of a row and the vector values it multiplies.
template <class T>
struct alignas(4 * sizeof(T)) Entry {
  T a, b, c, d;
};
// The same for two vectors.
template <class T>
struct Entry2 {
  T a, b, c, d, x, y, z;
};
// Shared memory of a split slice: FP32 entries on their way to the first
// warp, or NV FP64 partial sums of every warp.
template <class VT, class E, int NV, int SPLIT>
struct alignas(32) SplitBuf {  // an Entry2 buffer is read as one of Entry too
  static constexpr bool ordered = sizeof(VT) == 4;
  union {
    E e[ordered ? 4 * SPLIT : 1][32];
    VT v[ordered ? 1 : SPLIT][NV][32];
  };
};
// Entries of a slice's rows, w of them: stream(j) reads entry j of the thread's
// row, gather its vector values, use consumes both, in order.  FP32 with SPLIT
// > 1: each of the block's warps loads four of the next 4 SPLIT entries (the
// loads of the next group are in flight while the first warp consumes the
// current one).
//
// SPLIT = 1, one thread per row: every entry is a chain of column -> gather ->
// FMA, and what bounds a launch is how many chains its warps keep in flight
// against how much of the gathered vector the L1 keeps between them.  D = 0
// leaves the order to the compiler (unrolled by four); D > 0 gathers D entries
// together while the next D are read.  More D means more registers, fewer warps
// and a wider front of columns, so the best is small and differs by kernel (us
// on the 64^3 cavity, duct of 24 x 24 x 160 in brackets; K / G loop of step 1):
//   FP32  step 1 D = 0/0 369..456 (135..167)   0/2 373 (135)    2/2 458  4/4 389  8/8 454
//         with K Acc_prev  0/0 704 (261)  2/2 523 (191)  3/2 494 (181)  3/3 474 (174)  4/4 491  8/8 636
//         step 3  0 160  1 187  2 163  4 174  8 196     K v  0 228  1 303  2 229  3 293  8 340
//         G^T  0 113  1 131  2 116  3 122  4 149
//   FP64  step 1 0/0 637  2/0 550  2/2 576  3/3 627  4/4 700  8/8 847
//         with K Acc_prev  0/0 880  0/2 841  2/2 890  4/4 961
//         step 3  0 217  1 211  2 213  4 219  8 373     K v  0 414  1 462  2 404  4 418  8 498
// The column is read before the value where it is the head of the chain (split
// slices, K v FP32 on 24^3 elements 29 -> 24, G^T FP64 at 64^3 191 -> 175, FP32 on
// the duct 56 -> 52); in step 1's FP32 K loop the value goes first (3/3 with K
// Acc_prev 488 -> 474).
template <int SPLIT, int D, class B, class S, class G, class U>
__device__ __forceinline__ void for_entries(B& buf, int w, S stream, G gather, U use) {
  auto load = [&](int j) { return gather(stream(j)); };
  if constexpr (SPLIT == 1 && D == 0) {
#pragma unroll 4
    for (int j = 0; j < w; j++) use(load(j));
  } else if constexpr (SPLIT == 1) {
    decltype(stream(0)) st[D];
#pragma unroll
    for (int i = 0; i < D; i++)
      if (i < w) st[i] = stream(i);
    for (int j0 = 0; j0 < w; j0 += D) {
      decltype(load(0)) e[D];
#pragma unroll
      for (int i = 0; i < D; i++)
        if (j0 + i < w) e[i] = gather(st[i]);
#pragma unroll
      for (int i = 0; i < D; i++)
        if (j0 + D + i < w) st[i] = stream(j0 + D + i);
#pragma unroll
      for (int i = 0; i < D; i++)
        if (j0 + i < w) use(e[i]);
    }
  } else if constexpr (!B::ordered) {
#pragma unroll 4
    for (int j = threadIdx.x >> 5; j < w; j += SPLIT) use(load(j));
  } else {
    const int k = threadIdx.x >> 5, l = threadIdx.x & 31;
    decltype(load(0)) e[4];
    auto fetch = [&](int c0) {
#pragma unroll
      for (int i = 0; i < 4; i++)
        if (c0 + 4 * k + i < w) e[i] = load(c0 + 4 * k + i);
    };
    fetch(0);
    for (int c0 = 0; c0 < w; c0 += 4 * SPLIT) {
      __syncthreads();
#pragma unroll
      for (int i = 0; i < 4; i++) buf.e[4 * k + i][l] = e[i];
      __syncthreads();
      fetch(c0 + 4 * SPLIT);
      if (k == 0) {
        const int n = min(4 * SPLIT, w - c0);
#pragma unroll 4
        for (int j = 0; j < n; j++) use(buf.e[j][l]);
      }
    }
  }
}
// FP64 with SPLIT > 1: the warps' partial sums, added in warp order in the
// first warp.  Called by every thread of the block.
template <int SPLIT, class B, class VT, int NV>
__device__ __forceinline__ void split_sum(B& buf, VT (&v)[NV]) {
  if constexpr (SPLIT > 1 && !B::ordered) {
    const int k = threadIdx.x >> 5, l = threadIdx.x & 31;
    if (k != 0)
#pragma unroll
      for (int i = 0; i < NV; i++) buf.v[k][i][l] = v[i];
    __syncthreads();
    if (k == 0)
#pragma unroll
      for (int j = 1; j < SPLIT; j++)
#pragma unroll
        for (int i = 0; i < NV; i++) v[i] += buf.v[j][i][l];
  }
}

// step1: R1 = R1conv - K UnpHalf_prev - G Pn (blascoCodinaHuerta.cpp:
// 3745-3758), R1 = 0 at Dirichlet nodes (applyBC_Step1(2)),
// UnpHalf = Un + dt R1 MdInv (:3781-3783) -- the Dirichlet zeroing is the
// zero in minv_free.  Also writes d = UnpHalf/dt^2 - [iter>1] MdOrigInv KAcc,
// the input of step2 (blascoCodinaHuerta.cpp:3821-3832).
//
// ACC (iter > 1 inside cfd_run): the K Acc_prev of calculate_KtimesAcc_prev in
// the same pass over K, one read of its values and columns instead of two (us
// of step 1 and K Acc_prev: 64^3 FP64 1044 -> 841, FP32 597 -> 474, duct FP32
// 219 -> 174, 32^3 FP64 142 -> 131, 8^3 FP64 13.2 -> 9.5; 24^3 FP32 72 -> 46,
// 16^3 FP32 27 -> 22).
template <class VT, int SPLIT, bool ACC>
__global__ void __launch_bounds__(block_threads(SPLIT)) k_step1(Step1Args<VT> a) {
  __shared__ SplitBuf<VT, std::conditional_t<ACC, Entry2<VT>, Entry<VT>>, ACC ? 9 : 6, SPLIT> buf;
  constexpr bool fp32 = sizeof(VT) == 4;
  const int l = threadIdx.x & 31;
  const int row = SPLIT == 1 ? blockIdx.x * blockDim.x + threadIdx.x : 32 * blockIdx.x + l;
  if (SPLIT == 1 && row >= a.NN) return;
  const int s = row >> 5;
  const double inv_dt2 = 1.0000000000000000 / (a.dt * a.dt);
  VT kx = 0, ky = 0, kz = 0, gx = 0, gy = 0, gz = 0, ax = 0, ay = 0, az = 0;
  {
    const int b = __ldg(a.k_off + s), w = (__ldg(a.k_off + s + 1) - b) >> 5, bl = b + l;
    // order of the two loads as in the table at for_entries
    auto stream = [&](int j) {
      KEntry<VT> k;
      if constexpr (fp32 && SPLIT == 1) {
        k.v = __ldcs(a.kval + bl + 32 * j);
        k.c = __ldcs(a.k_col + bl + 32 * j);
      } else {
        k.c = __ldcs(a.k_col + bl + 32 * j);
        k.v = __ldcs(a.kval + bl + 32 * j);
      }
      return k;
    };
    if constexpr (ACC) {
      for_entries<SPLIT, fp32 ? 3 : 0>(
          buf, w, stream,
          [&](const KEntry<VT>& k) {
            const auto x = ldgv(a.uprev + k.c);
            const auto y = ldgv(a.accprev + k.c);
            return Entry2<VT>{k.v, (VT)x.x, (VT)x.y, (VT)x.z, (VT)y.x, (VT)y.y, (VT)y.z};
          },
          [&](const Entry2<VT>& e) {
            kx += e.a * e.b;
            ky += e.a * e.c;
            kz += e.a * e.d;
            ax += e.a * e.x;
            ay += e.a * e.y;
            az += e.a * e.z;
          });
    } else {
      for_entries<SPLIT, fp32 ? 0 : 2>(
          buf, w, stream,
          [&](const KEntry<VT>& k) {
            const auto x = ldgv(a.uprev + k.c);
            return Entry<VT>{k.v, (VT)x.x, (VT)x.y, (VT)x.z};
          },
          [&](const Entry<VT>& e) {
            kx += e.a * e.b;
            ky += e.a * e.c;
            kz += e.a * e.d;
          });
    }
  }
  {
    const int b = __ldg(a.g_off + s), w = (__ldg(a.g_off + s + 1) - b) >> 5, bl = b + l;
    auto& gbuf = reinterpret_cast<SplitBuf<VT, Entry<VT>, 6, SPLIT>&>(buf);
    for_entries<SPLIT, fp32 ? (ACC ? 3 : 2) : ACC ? 2 : 0>(
        gbuf, w,
        [&](int j) {
          const int e = bl + 32 * j;
          return GEntry<VT>{__ldcs(a.g_col + e), __ldcs(a.g1 + e), __ldcs(a.g2 + e), __ldcs(a.g3 + e)};
        },
        [&](const GEntry<VT>& g) { return Entry<VT>{g.x, g.y, g.z, (VT)__ldg(a.pn + g.c)}; },
        [&](const Entry<VT>& e) {
          gx += e.a * e.d;
          gy += e.b * e.d;
          gz += e.c * e.d;
        });
  }
  if constexpr (SPLIT > 1) {
    if constexpr (ACC) {
      VT v[9] = {kx, ky, kz, gx, gy, gz, ax, ay, az};
      split_sum<SPLIT>(buf, v);
      kx = v[0], ky = v[1], kz = v[2], gx = v[3], gy = v[4], gz = v[5], ax = v[6], ay = v[7], az = v[8];
    } else {
      VT v[6] = {kx, ky, kz, gx, gy, gz};
      split_sum<SPLIT>(buf, v);
      kx = v[0], ky = v[1], kz = v[2], gx = v[3], gy = v[4], gz = v[5];
    }
    if (threadIdx.x >= 32 || row >= a.NN) return;
  }
  double4 rc;
  if (a.r1conv32) {
    const float4 f = a.r1conv32[row];
    rc = make_double4(f.x, f.y, f.z, 0.0);
  } else {
    rc = a.r1conv[row];
  }
  const double mf = a.minv_free[row];
  double rx = (rc.x - (double)kx) - (double)gx;
  double ry = (rc.y - (double)ky) - (double)gy;
  double rz = (rc.z - (double)kz) - (double)gz;
  if (mf == 0.0) rx = ry = rz = 0.0;  // Dirichlet node
  const double4 u = a.un[row];
  double4 h;
  h.x = u.x + a.dt * rx * mf;
  h.y = u.y + a.dt * ry * mf;
  h.z = u.z + a.dt * rz * mf;
  h.w = 0.0;
  a.unphalf[row] = h;
  if constexpr (sizeof(VT) == 4) a.unphalf_g[row] = to_f4(h);
  double4 d;
  d.x = inv_dt2 * h.x;
  d.y = inv_dt2 * h.y;
  d.z = inv_dt2 * h.z;
  d.w = 0.0;
  if (a.iter != 1) {
    const double mo = a.minv_orig[row];
    double4 ka;
    if constexpr (ACC) {
      ka = make_double4((double)ax, (double)ay, (double)az, 0.0);
      a.kacc[row] = ka;
    } else {
      ka = a.kacc[row];
    }
    d.x = d.x - mo * ka.x;
    d.y = d.y - mo * ka.y;
    d.z = d.z - mo * ka.z;
  }
  a.d[row] = d;
  if constexpr (sizeof(VT) == 4) a.d_g[row] = to_f4(d);
  if (a.r1out) a.r1out[row] = make_double4(rx, ry, rz, 0.0);
}

// out[p] = sum_d (G_d^T d_d)[p]; out[pin] = 0 when pin > 0
// (step2GPU's three transposed csrmv calls + applyPresBC, CUDAcodes.cu:1006-1011).
template <class VT, int SPLIT>
__global__ void __launch_bounds__(block_threads(SPLIT)) k_gt(GtArgs<VT> a) {
  __shared__ SplitBuf<VT, VT, 1, SPLIT> buf;
  const int l = threadIdx.x & 31;
  const int row = SPLIT == 1 ? blockIdx.x * blockDim.x + threadIdx.x : 32 * blockIdx.x + l;
  if (SPLIT == 1 && row >= a.NNp) return;
  const int s = row >> 5;
  const int b = __ldg(a.gt_off + s) + l, w = (__ldg(a.gt_off + s + 1) - __ldg(a.gt_off + s)) >> 5;
  VT acc[1] = {0};
  for_entries<SPLIT, 0>(
      buf, w,
      [&](int j) {
        const int e = b + 32 * j;
        return GEntry<VT>{__ldcs(a.gt_col + e), __ldcs(a.gt1 + e), __ldcs(a.gt2 + e), __ldcs(a.gt3 + e)};
      },
      [&](const GEntry<VT>& g) {
        const auto d = ldgv(a.d + g.c);
        return g.x * (VT)d.x + g.y * (VT)d.y + g.z * (VT)d.z;
      },
      [&](VT t) { acc[0] += t; });
  split_sum<SPLIT>(buf, acc);
  if (SPLIT > 1 && (threadIdx.x >= 32 || row >= a.NNp)) return;
  a.out[row] = (a.pin > 0 && row == a.pin) ? 0.0 : (double)acc[0];
}

// step3: R3 = -dt G Pdot - [iter>1] dt KAcc, R3 = 0 at Dirichlet nodes,
// Acc = R3 MdInv, Unp1 = UnpHalf + dt Acc (blascoCodinaHuerta.cpp:3920-3967)
// plus the partial sums of the convergence test (:2936-2961) and of the
// steady-state test (:3052-3057).
template <class VT, int SPLIT>
__global__ void __launch_bounds__(block_threads(SPLIT)) k_step3(Step3Args<VT> a) {
  __shared__ SplitBuf<VT, Entry<VT>, 3, SPLIT> buf;
  const int l = threadIdx.x & 31;
  const int row = SPLIT == 1 ? blockIdx.x * blockDim.x + threadIdx.x : 32 * blockIdx.x + l;
  const double inv_dt = 1.0000000000000000 / a.dt;
  double s_u2 = 0, s_du2 = 0, m_acc = 0;
  VT gx = 0, gy = 0, gz = 0;
  auto products = [&]() {
    const int s = row >> 5;
    const int b = __ldg(a.g_off + s) + l, w = (__ldg(a.g_off + s + 1) - __ldg(a.g_off + s)) >> 5;
    for_entries<SPLIT, sizeof(VT) == 8 ? 1 : 0>(
        buf, w,
        [&](int j) {
          const int e = b + 32 * j;
          return GEntry<VT>{__ldcs(a.g_col + e), __ldcs(a.g1 + e), __ldcs(a.g2 + e), __ldcs(a.g3 + e)};
        },
        [&](const GEntry<VT>& g) { return Entry<VT>{g.x, g.y, g.z, (VT)__ldg(a.pdot + g.c)}; },
        [&](const Entry<VT>& e) {
          gx += e.a * e.d;
          gy += e.b * e.d;
          gz += e.c * e.d;
        });
  };
  auto epilogue = [&]() {
    double rx = -a.dt * (double)gx, ry = -a.dt * (double)gy, rz = -a.dt * (double)gz;
    if (a.iter != 1) {
      const double4 ka = a.kacc[row];
      rx = rx - a.dt * ka.x;
      ry = ry - a.dt * ka.y;
      rz = rz - a.dt * ka.z;
    }
    const double mf = a.minv_free[row];
    if (mf == 0.0) rx = ry = rz = 0.0;  // Dirichlet node
    const double4 acc = make_double4(rx * mf, ry * mf, rz * mf, 0.0);
    const double4 h = a.unphalf[row];
    const double4 u1 = make_double4(h.x + a.dt * acc.x, h.y + a.dt * acc.y, h.z + a.dt * acc.z, 0.0);
    a.acc[row] = acc;
    if constexpr (sizeof(VT) == 4) a.acc_g[row] = to_f4(acc);
    a.unp1[row] = u1;
    if (a.r3out) a.r3out[row] = make_double4(rx, ry, rz, 0.0);
    const double4 pv = a.unp1_prev[row];
    const double4 un = a.un[row];
    s_u2 = u1.x * u1.x + u1.y * u1.y + u1.z * u1.z;
    const double dx = u1.x - pv.x, dy = u1.y - pv.y, dz = u1.z - pv.z;
    s_du2 = dx * dx + dy * dy + dz * dz;
    m_acc = fmax(fabs((u1.x - un.x) * inv_dt), fmax(fabs((u1.y - un.y) * inv_dt), fabs((u1.z - un.z) * inv_dt)));
  };
  if constexpr (SPLIT == 1) {
    if (row < a.NN) {
      products();
      epilogue();
    }
  } else {
    products();
    VT v[3] = {gx, gy, gz};
    split_sum<SPLIT>(buf, v);
    gx = v[0], gy = v[1], gz = v[2];
    if (threadIdx.x < 32 && row < a.NN) epilogue();
  }
  double v[2] = {s_u2, s_du2};
  m_acc = warp_max(m_acc);
  __shared__ double smax[32];
  if ((threadIdx.x & 31) == 0) smax[threadIdx.x >> 5] = m_acc;
  block_sum<2>(v);
  if (threadIdx.x == 0) {
    double m = 0;
    for (int w = 0; w < (int)(blockDim.x >> 5); w++) m = fmax(m, smax[w]);
    a.part[blockIdx.x] = v[0];
    a.part[a.nblocks + blockIdx.x] = v[1];
    a.part[2 * a.nblocks + blockIdx.x] = m;
  }
}

template <class VT, int SPLIT>
__global__ void __launch_bounds__(block_threads(SPLIT)) k_spmv_k3(SpmvK3Args<VT> a) {
  __shared__ SplitBuf<VT, Entry<VT>, 3, SPLIT> buf;
  const int l = threadIdx.x & 31;
  const int row = SPLIT == 1 ? blockIdx.x * blockDim.x + threadIdx.x : 32 * blockIdx.x + l;
  if (SPLIT == 1 && row >= a.NN) return;
  const int s = row >> 5;
  const int b = __ldg(a.off + s) + l, w = (__ldg(a.off + s + 1) - __ldg(a.off + s)) >> 5;
  VT sx = 0, sy = 0, sz = 0;
  for_entries<SPLIT, sizeof(VT) == 8 ? 2 : 0>(
      buf, w,
      [&](int j) {
        const int e = b + 32 * j;
        return KEntry<VT>{__ldcs(a.col + e), __ldcs(a.val + e)};
      },
      [&](const KEntry<VT>& k) {
        const auto x = ldgv(a.x + k.c);
        return Entry<VT>{k.v, (VT)x.x, (VT)x.y, (VT)x.z};
      },
      [&](const Entry<VT>& e) {
        sx += e.a * e.b;
        sy += e.a * e.c;
        sz += e.a * e.d;
      });
  VT v[3] = {sx, sy, sz};
  split_sum<SPLIT>(buf, v);
  if (SPLIT > 1 && (threadIdx.x >= 32 || row >= a.NN)) return;
  a.y[row] = make_double4((double)v[0], (double)v[1], (double)v[2], 0.0);
}

__global__ void __launch_bounds__(kRowThreads) k_pressure_update(int n, double dt, const double* __restrict__ pn,
                                                                 const double* __restrict__ pdot,
                                                                 const double* __restrict__ pprev, double* pnp1,
                                                                 double* part, int nblocks) {
  double v[2] = {0, 0};
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    double p = pn[i] + dt * pdot[i];
    pnp1[i] = p;
    v[0] += p * p;
    double d = p - pprev[i];
    v[1] += d * d;
  }
  block_sum<2>(v);
  if (threadIdx.x == 0) {
    part[blockIdx.x] = v[0];
    part[nblocks + blockIdx.x] = v[1];
  }
}

// Fixed-order reduction of the per-block partials (deterministic).
__global__ void k_reduce_norms(const double* __restrict__ up, int nub, const double* __restrict__ pp, int npb,
                               double* out) {
  double v[4] = {0, 0, 0, 0};
  double m = 0;
  for (int i = threadIdx.x; i < nub; i += blockDim.x) {
    v[0] += up[i];
    v[1] += up[nub + i];
    m = fmax(m, up[2 * nub + i]);
  }
  for (int i = threadIdx.x; i < npb; i += blockDim.x) {
    v[2] += pp[i];
    v[3] += pp[npb + i];
  }
  m = warp_max(m);
  __shared__ double smax[32];
  if ((threadIdx.x & 31) == 0) smax[threadIdx.x >> 5] = m;
  block_sum<4>(v);
  if (threadIdx.x == 0) {
    double mm = 0;
    for (int w = 0; w < (int)(blockDim.x >> 5); w++) mm = fmax(mm, smax[w]);
    out[0] = v[0]; out[1] = v[1]; out[2] = v[2]; out[3] = v[3]; out[4] = mm;
  }
}

template <class T>
__global__ void k_csr_to_sell(int nrows, const int* __restrict__ rp, const double* __restrict__ csr,
                              const int* __restrict__ off, T* sell) {
  const int row = blockIdx.x * blockDim.x + threadIdx.x;
  const int nslices = (nrows + 31) >> 5;
  if (row >= nslices * 32) return;
  const int s = row >> 5, l = row & 31;
  const int b = off[s] + l, w = (off[s + 1] - off[s]) >> 5;
  const int cb = row < nrows ? rp[row] : 0, len = row < nrows ? rp[row + 1] - cb : 0;
  for (int j = 0; j < w; j++) sell[b + 32 * j] = j < len ? (T)csr[cb + j] : (T)0;
}

// SELL-32 pattern of a CSR pattern: slice widths (longest row of each
// 32-row slice), then the columns slice-column-major, a row shorter than its
// slice padded with its last column (0 for an empty row or a row past the
// end).
__global__ void k_sell_widths(int nrows, const int* __restrict__ rp, int* __restrict__ width) {
  const int ns = (nrows + 31) >> 5;
  for (int sl = blockIdx.x * blockDim.x + threadIdx.x; sl < ns; sl += gridDim.x * blockDim.x) {
    int w = 0;
    for (int r = 32 * sl; r < min(nrows, 32 * sl + 32); r++) w = max(w, rp[r + 1] - rp[r]);
    width[sl] = w;
  }
}
__global__ void k_sell_cols(int nrows, const int* __restrict__ rp, const int* __restrict__ col,
                            const int* __restrict__ off, int* __restrict__ scol) {
  const int row = blockIdx.x * blockDim.x + threadIdx.x;
  const int nslices = (nrows + 31) >> 5;
  if (row >= nslices * 32) return;
  const int sl = row >> 5, l = row & 31;
  const int b = off[sl] + l, w = (off[sl + 1] - off[sl]) >> 5;
  const int cb = row < nrows ? rp[row] : 0, len = row < nrows ? rp[row + 1] - cb : 0;
  const int padc = len > 0 ? col[cb + len - 1] : 0;
  for (int j = 0; j < w; j++) scol[b + 32 * j] = j < len ? col[cb + j] : padc;
}

__global__ void k_blocks_to_vec4(int NN, const double* __restrict__ b, double4* v) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < NN; i += gridDim.x * blockDim.x)
    v[i] = make_double4(b[i], b[(size_t)NN + i], b[2 * (size_t)NN + i], 0.0);
}
__global__ void k_vec4_to_blocks(int NN, const double4* __restrict__ v, double* b) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < NN; i += gridDim.x * blockDim.x) {
    double4 x = v[i];
    b[i] = x.x;
    b[(size_t)NN + i] = x.y;
    b[2 * (size_t)NN + i] = x.z;
  }
}
__global__ void k_apply_bc(int n, const int* __restrict__ nodes, const double* __restrict__ uvw, double4* u) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    u[nodes[i]] = make_double4(uvw[3 * (size_t)i], uvw[3 * (size_t)i + 1], uvw[3 * (size_t)i + 2], 0.0);
}

inline int ew_grid(long long n) {
  long long g = (n + 255) / 256;
  if (g > 148 * 16) g = 148 * 16;
  if (g < 1) g = 1;
  return (int)g;
}

}  // namespace

// Launches kernel<VT, SPLIT, ...> with the SPLIT of the row count.
#define SPLIT_LAUNCH(kernel, rows, rule, ...)                                                              \
  do {                                                                                                     \
    const int sp_ = row_split<VT>(rows, rule, num_sms), g_ = split_grid(rows, sp_);                        \
    switch (sp_) {                                                                                         \
      case 1: kernel<VT, 1 __VA_OPT__(, ) __VA_ARGS__><<<g_, kRowThreads, 0, s>>>(a); break;               \
      case 2: kernel<VT, 2 __VA_OPT__(, ) __VA_ARGS__><<<g_, block_threads(2), 0, s>>>(a); break;          \
      case 4: kernel<VT, 4 __VA_OPT__(, ) __VA_ARGS__><<<g_, block_threads(4), 0, s>>>(a); break;          \
      default: kernel<VT, 8 __VA_OPT__(, ) __VA_ARGS__><<<g_, block_threads(8), 0, s>>>(a); break;         \
    }                                                                                                      \
    return cudaGetLastError();                                                                             \
  } while (0)

template <class VT>
cudaError_t launch_step1(const Step1Args<VT>& a, int num_sms, cudaStream_t s) {
  if (a.accprev) SPLIT_LAUNCH(k_step1, a.NN, kStep1Rule, true);
  SPLIT_LAUNCH(k_step1, a.NN, kStep1Rule, false);
}
template <class VT>
cudaError_t launch_gt(const GtArgs<VT>& a, int num_sms, cudaStream_t s) {
  SPLIT_LAUNCH(k_gt, a.NNp, kGtRule);
}
template <class VT>
cudaError_t launch_step3(const Step3Args<VT>& a, int num_sms, cudaStream_t s) {
  SPLIT_LAUNCH(k_step3, a.NN, kStep3Rule);
}
template <class VT>
cudaError_t launch_spmv_k3(const SpmvK3Args<VT>& a, int num_sms, cudaStream_t s) {
  SPLIT_LAUNCH(k_spmv_k3, a.NN, kSpmvK3Rule);
}
template <class VT>
int step3_blocks(int NN, int num_sms) {
  return split_grid(NN, row_split<VT>(NN, kStep3Rule, num_sms));
}
template int step3_blocks<double>(int, int);
template int step3_blocks<float>(int, int);
int pupdate_blocks(int NNp, int num_sms) { return ew_grid(NNp) < num_sms * 4 ? ew_grid(NNp) : num_sms * 4; }
cudaError_t launch_pressure_update(int NNp, double dt, const double* pn, const double* pdot, const double* pprev,
                                   double* pnp1, double* part, int nblocks, cudaStream_t s) {
  k_pressure_update<<<nblocks, kRowThreads, 0, s>>>(NNp, dt, pn, pdot, pprev, pnp1, part, nblocks);
  return cudaGetLastError();
}
cudaError_t launch_reduce_norms(const double* upart, int nub, const double* ppart, int npb, double* out,
                                cudaStream_t s) {
  k_reduce_norms<<<1, 1024, 0, s>>>(upart, nub, ppart, npb, out);
  return cudaGetLastError();
}
cudaError_t launch_sell_widths(int nrows, const int* rp, int* width, cudaStream_t s) {
  const int ns = (nrows + 31) / 32;
  k_sell_widths<<<rows_grid(ns) < 4096 ? rows_grid(ns) : 4096, kRowThreads, 0, s>>>(nrows, rp, width);
  return cudaGetLastError();
}
cudaError_t launch_sell_cols(int nrows, const int* rp, const int* col, const int* off, int* scol, cudaStream_t s) {
  const int nslices = (nrows + 31) / 32;
  k_sell_cols<<<rows_grid((long long)nslices * 32), kRowThreads, 0, s>>>(nrows, rp, col, off, scol);
  return cudaGetLastError();
}
template <class T>
cudaError_t launch_csr_to_sell(int nrows, const int* rp, const double* csr, const int* off, T* sell, cudaStream_t s) {
  const int nslices = (nrows + 31) / 32;
  k_csr_to_sell<T><<<rows_grid((long long)nslices * 32), kRowThreads, 0, s>>>(nrows, rp, csr, off, sell);
  return cudaGetLastError();
}
__global__ void k_vec4_to_f32(int NN, const double4* __restrict__ v, float4* a, float4* b) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < NN; i += gridDim.x * blockDim.x) {
    const float4 f = to_f4(v[i]);
    a[i] = f;
    b[i] = f;
  }
}

cudaError_t launch_vec4_to_f32(int NN, const double4* v, float4* a, float4* b, cudaStream_t s) {
  k_vec4_to_f32<<<rows_grid(NN), kRowThreads, 0, s>>>(NN, v, a, b);
  return cudaGetLastError();
}

cudaError_t launch_blocks_to_vec4(int NN, const double* blocks, double4* v, cudaStream_t s) {
  k_blocks_to_vec4<<<ew_grid(NN), 256, 0, s>>>(NN, blocks, v);
  return cudaGetLastError();
}
cudaError_t launch_vec4_to_blocks(int NN, const double4* v, double* blocks, cudaStream_t s) {
  k_vec4_to_blocks<<<ew_grid(NN), 256, 0, s>>>(NN, v, blocks);
  return cudaGetLastError();
}
cudaError_t launch_apply_bc(int n, const int* nodes, const double* uvw, double4* u, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  k_apply_bc<<<ew_grid(n), 256, 0, s>>>(n, nodes, uvw, u);
  return cudaGetLastError();
}

template cudaError_t launch_step1<double>(const Step1Args<double>&, int, cudaStream_t);
template cudaError_t launch_step1<float>(const Step1Args<float>&, int, cudaStream_t);
template cudaError_t launch_gt<double>(const GtArgs<double>&, int, cudaStream_t);
template cudaError_t launch_gt<float>(const GtArgs<float>&, int, cudaStream_t);
template cudaError_t launch_step3<double>(const Step3Args<double>&, int, cudaStream_t);
template cudaError_t launch_step3<float>(const Step3Args<float>&, int, cudaStream_t);
template cudaError_t launch_spmv_k3<double>(const SpmvK3Args<double>&, int, cudaStream_t);
template cudaError_t launch_spmv_k3<float>(const SpmvK3Args<float>&, int, cudaStream_t);
template cudaError_t launch_csr_to_sell<double>(int, const int*, const double*, const int*, double*, cudaStream_t);
template cudaError_t launch_csr_to_sell<float>(int, const int*, const double*, const int*, float*, cudaStream_t);

}  // namespace cfd
