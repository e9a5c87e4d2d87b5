// One-time operator assembly on the device (step0 and calculateZ_CUSP of the
// reference, blascoCodinaHuerta.cpp:3127-3315 and CUDAcodes.cu:281-411).
//
// k_assemble: one element per block iteration.  The Jacobian of the
//   trilinear corner map, its adjugate inverse and detJ are recomputed per
//   Gauss point from the 8 corner coordinates (blascoCodinaHuerta.cpp:
//   2566-2615), so no per-Gauss-point geometry is stored in HBM.  Element
//   blocks Ke (27x27), Ge_d (27x8) and the row sums of Me are added into
//   their CSR slots with FP64 atomics; the slot is found by binary search in
//   the sorted CSR row, so no element colouring and no slot map is needed.
//   In deterministic mode the host launches one colour at a time (no two
//   elements of a colour share a node) and the blocks add without atomics,
//   in the same order every run.
// k_build_z: Z = sum_d G_d^T diag(MdOrigInv) G_d in gather form, one warp
//   per Z row: for every velocity node v of G^T row p (ascending), the lanes
//   take the columns q of G row v and add (G_d[v][q]*Minv[v]) * G_d[v][p] to
//   a shared accumulator of row p.  Lanes of one v never collide, so the
//   accumulation order is fixed (deterministic, ascending v as in the oracle).
//   Bound by the chain of gathers and searches per v; reading the next v's row
//   meanwhile: 30^3 elements 1.37 -> 1.12 ms.
#include <cstdio>

#include "kernels.h"

namespace cfd {

namespace {

// Jacobian data of Gauss point k from corner coordinates X[8][3]:
// J[i][j] = sum_m dSp[i][k][m] X[m][j]; returns detJ, writes adj(J)/detJ.
template <class T>
__device__ __forceinline__ T jacobian_inv(const T (*X)[3], const Basis* __restrict__ B, int k, T iJ[3][3]) {
  T J[3][3];
#pragma unroll
  for (int i = 0; i < 3; i++)
#pragma unroll
    for (int j = 0; j < 3; j++) {
      T s = 0;
#pragma unroll
      for (int m = 0; m < 8; m++) s += (T)B->dSp[i][k][m] * X[m][j];
      J[i][j] = s;
    }
  T det = J[0][0] * (J[1][1] * J[2][2] - J[2][1] * J[1][2]) + J[0][1] * (J[1][2] * J[2][0] - J[1][0] * J[2][2]) +
          J[0][2] * (J[1][0] * J[2][1] - J[1][1] * J[2][0]);
  T inv = T(1) / det;
  iJ[0][0] = (J[1][1] * J[2][2] - J[2][1] * J[1][2]) * inv;
  iJ[0][1] = -(J[0][1] * J[2][2] - J[0][2] * J[2][1]) * inv;
  iJ[0][2] = (J[0][1] * J[1][2] - J[1][1] * J[0][2]) * inv;
  iJ[1][0] = -(J[1][0] * J[2][2] - J[1][2] * J[2][0]) * inv;
  iJ[1][1] = (J[2][2] * J[0][0] - J[2][0] * J[0][2]) * inv;
  iJ[1][2] = -(J[1][2] * J[0][0] - J[1][0] * J[0][2]) * inv;
  iJ[2][0] = (J[1][0] * J[2][1] - J[2][0] * J[1][1]) * inv;
  iJ[2][1] = -(J[2][1] * J[0][0] - J[2][0] * J[0][1]) * inv;
  iJ[2][2] = (J[1][1] * J[0][0] - J[1][0] * J[0][1]) * inv;
  return det;
}

constexpr int kAsmThreads = 128;

// Slots of three columns in one sorted CSR row, or -1; the three searches run in
// step, so that a round of loads costs one latency.
__device__ __forceinline__ void search3(const int* __restrict__ col, int b, int e, const int* key, int (&slot)[3]) {
  int lo[3] = {b, b, b};
  for (int n = e - b; n > 1;) {
    const int h = n >> 1;
#pragma unroll
    for (int q = 0; q < 3; q++)
      if (__ldg(col + lo[q] + h) <= key[q]) lo[q] += h;
    n -= h;
  }
#pragma unroll
  for (int q = 0; q < 3; q++) slot[q] = b < e && __ldg(col + lo[q]) == key[q] ? lo[q] : -1;
}

// Threads 0 .. 80 own a 3 x 3 tile of Ke each, threads 96 .. 122 a row of the
// Ge_d (8 corners) and of Me: 2.1 shared-memory reads per entry and Gauss point
// of Ke instead of 7, 9 searches in 3 chains instead of 6 x 1.  The tiles of Me go
// with those of Ke, and a row's 27 entries are then added in order (a serial 729 of one
// warp before).  The order is kept because a lumped mass that differs in its last
// bit changes the rounding of a mixed run's FP32 velocities: with the row sum as
// sum_k Sv_i (sum_j Sv_j) wd its pressure moved by up to 3.5e-8.  30^3 elements, 27 Gauss
// points: 1.80 -> 0.80 ms, 8 points 0.70 -> 0.52 (0.83 and 0.46 with that sum).
__global__ void __launch_bounds__(kAsmThreads) k_assemble(AsmArgs a) {
  __shared__ double sSv[kMaxNGP][27];
  __shared__ double sSp[kMaxNGP][8];
  __shared__ double sM[27][27];  // Me
  __shared__ double X[8][3];
  __shared__ int lt[27];
  __shared__ double iJ[kMaxNGP][3][3];
  __shared__ double wd[kMaxNGP];
  __shared__ double gd[kMaxNGP][27][3];
  const int t = threadIdx.x, ngp = a.ngp;
  const Basis* B = a.basis;
  for (int i = t; i < ngp * 27; i += blockDim.x) sSv[i / 27][i % 27] = B->Sv[i / 27][i % 27];
  for (int i = t; i < ngp * 8; i += blockDim.x) sSp[i / 8][i % 8] = B->Sp[i / 8][i % 8];
  for (int pos = a.e_begin + blockIdx.x; pos < a.e_end; pos += gridDim.x) {
    const int e = a.elist ? a.elist[pos] : pos;
    __syncthreads();
    if (t < 27) lt[t] = a.ltog[(size_t)e * 27 + t];
    __syncthreads();
    if (t < 24) X[t / 3][t % 3] = a.coord[3 * (size_t)lt[t / 3] + t % 3];
    __syncthreads();
    if (t < ngp) {
      double J[3][3];
      double det = jacobian_inv<double>(X, B, t, J);
      for (int i = 0; i < 3; i++)
        for (int j = 0; j < 3; j++) iJ[t][i][j] = J[i][j];
      wd[t] = det * B->w[t];
    }
    __syncthreads();
    for (int idx = t; idx < ngp * 27; idx += blockDim.x) {
      int k = idx / 27, j = idx % 27;
      double r0 = B->dSv[0][k][j], r1 = B->dSv[1][k][j], r2 = B->dSv[2][k][j];
      for (int i = 0; i < 3; i++) gd[k][j][i] = iJ[k][i][0] * r0 + iJ[k][i][1] * r1 + iJ[k][i][2] * r2;
    }
    __syncthreads();
    auto add = [&](double* to, double s) {
      if (a.plain)
        *to += s;
      else
        atomicAdd(to, s);
    };
    if (t < 81) {
      const int i0 = 3 * (t / 9), j0 = 3 * (t % 9);
      double s[3][3] = {}, me[3][3] = {};
      for (int k = 0; k < ngp; k++) {
        double u[3][3], v[3][3];
#pragma unroll
        for (int m = 0; m < 3; m++)
#pragma unroll
          for (int d = 0; d < 3; d++) {
            u[m][d] = gd[k][i0 + m][d];
            v[m][d] = gd[k][j0 + m][d];
          }
        const double w = wd[k];
#pragma unroll
        for (int m = 0; m < 3; m++)
#pragma unroll
          for (int n = 0; n < 3; n++) {
            s[m][n] += a.viscosity * (u[m][0] * v[n][0] + u[m][1] * v[n][1] + u[m][2] * v[n][2]) * w;
            me[m][n] += sSv[k][i0 + m] * sSv[k][j0 + n] * w;
          }
      }
#pragma unroll
      for (int m = 0; m < 3; m++)
#pragma unroll
        for (int n = 0; n < 3; n++) sM[i0 + m][j0 + n] = me[m][n];
#pragma unroll
      for (int m = 0; m < 3; m++) {
        const int row = lt[i0 + m];
        int slot[3];
        search3(a.k_col, a.k_rp[row], a.k_rp[row + 1], lt + j0, slot);
#pragma unroll
        for (int n = 0; n < 3; n++)
          if (slot[n] >= 0) add(a.kval + slot[n], s[m][n]);
      }
    } else if (t >= 96 && t < 96 + 27) {
      // Ge_d[i][m] = -(1/rho) sum_k Sp[k][m] dSv_i/dx_d detJ w
      const int i = t - 96, row = lt[i];
      double s[8][3] = {};
      for (int k = 0; k < ngp; k++) {
        const double w = wd[k], g0 = gd[k][i][0], g1 = gd[k][i][1], g2 = gd[k][i][2];
#pragma unroll
        for (int m = 0; m < 8; m++) {
          const double f = a.inv_density * sSp[k][m];
          s[m][0] -= f * g0 * w;
          s[m][1] -= f * g1 * w;
          s[m][2] -= f * g2 * w;
        }
      }
      const int b = a.g_rp[row], end = a.g_rp[row + 1];
#pragma unroll
      for (int m0 = 0; m0 < 9; m0 += 3) {
        const int key[3] = {lt[m0], lt[m0 + 1], m0 + 2 < 8 ? lt[m0 + 2] : lt[m0]};
        int slot[3];
        search3(a.g_col, b, end, key, slot);
#pragma unroll
        for (int n = 0; n < 3; n++)
          if (m0 + n < 8 && slot[n] >= 0) {
            add(a.g1 + slot[n], s[m0 + n][0]);
            add(a.g2 + slot[n], s[m0 + n][1]);
            add(a.g3 + slot[n], s[m0 + n][2]);
          }
      }
    }
    __syncthreads();
    if (t >= 96 && t < 96 + 27) {
      double ms = 0;
      for (int j = 0; j < 27; j++) ms += sM[t - 96][j];
      add(a.msum + lt[t - 96], ms);
    }
  }
}

__global__ void k_fill_gt(long long nnz, const int* __restrict__ pos, const double* __restrict__ g1,
                          const double* __restrict__ g2, const double* __restrict__ g3, double* gt1, double* gt2,
                          double* gt3) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < nnz; i += (long long)gridDim.x * blockDim.x) {
    int p = pos[i];
    gt1[i] = g1[p];
    gt2[i] = g2[p];
    gt3[i] = g3[p];
  }
}

__global__ void k_md_finalize(int NN, const double* __restrict__ msum, const unsigned char* __restrict__ bc,
                              double* minv_orig, double* minv_free) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < NN; i += gridDim.x * blockDim.x) {
    double inv = 1.0 / msum[i];
    minv_orig[i] = inv;
    minv_free[i] = bc[i] ? 0.0 : inv;
  }
}

__device__ __forceinline__ int bsearch_smem(const int* col, int n, int key) {
  int lo = 0, hi = n - 1;
  while (lo <= hi) {
    int mid = (lo + hi) >> 1;
    int c = col[mid];
    if (c == key) return mid;
    if (c < key) lo = mid + 1; else hi = mid - 1;
  }
  return -1;
}

constexpr int kZWarps = 4;

__global__ void __launch_bounds__(32 * kZWarps) k_build_z(ZArgs a) {
  extern __shared__ unsigned char smem[];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int stride = a.maxrow;
  double* acc = reinterpret_cast<double*>(smem) + (size_t)w * 3 * stride;
  int* cols = reinterpret_cast<int*>(reinterpret_cast<double*>(smem) + (size_t)kZWarps * 3 * stride) + (size_t)w * stride;
  for (int p = blockIdx.x * kZWarps + w; p < a.NNp; p += gridDim.x * kZWarps) {
    const int zb = a.z_rp[p], len = a.z_rp[p + 1] - zb;
    for (int i = lane; i < len; i += 32) {
      cols[i] = a.z_col[zb + i];
      acc[i] = 0.0;
      acc[stride + i] = 0.0;
      acc[2 * stride + i] = 0.0;
    }
    __syncwarp();
    const int t1 = a.gt_rp[p + 1];
    for (int tc = a.gt_rp[p]; tc < t1; tc += 32) {
      // lane l holds entry tc + l of G^T; the G row of the next one is read
      // while the current one is added
      const int nt = min(32, t1 - tc);
      int jb = 0, je = 0;
      double lm = 0, l1 = 0, l2 = 0, l3 = 0;
      if (lane < nt) {
        const int v = a.gt_col[tc + lane];
        lm = a.minv_orig[v];
        l1 = a.gt1[tc + lane];
        l2 = a.gt2[tc + lane];
        l3 = a.gt3[tc + lane];
        jb = a.g_rp[v];
        je = a.g_rp[v + 1];
      }
      int j = 0, e = 0, c = -1;
      double x1 = 0, x2 = 0, x3 = 0;
      auto fetch = [&](int q) {
        j = __shfl_sync(0xffffffffu, jb, q) + lane;
        e = __shfl_sync(0xffffffffu, je, q);
        c = -1;
        if (j < e) {
          c = a.g_col[j];
          x1 = a.g1[j];
          x2 = a.g2[j];
          x3 = a.g3[j];
        }
      };
      fetch(0);
      for (int q = 0; q < nt; q++) {
        const double m = __shfl_sync(0xffffffffu, lm, q), p1 = __shfl_sync(0xffffffffu, l1, q);
        const double p2 = __shfl_sync(0xffffffffu, l2, q), p3 = __shfl_sync(0xffffffffu, l3, q);
        int jj = j, cc = c;
        const int ee = e;
        double y1 = x1, y2 = x2, y3 = x3;
        if (q + 1 < nt) fetch(q + 1);
        while (cc >= 0) {
          const int pos = bsearch_smem(cols, len, cc);
          if (pos >= 0) {
            acc[pos] += (y1 * m) * p1;
            acc[stride + pos] += (y2 * m) * p2;
            acc[2 * stride + pos] += (y3 * m) * p3;
          }
          jj += 32;  // rows longer than a warp
          cc = -1;
          if (jj < ee) {
            cc = a.g_col[jj];
            y1 = a.g1[jj];
            y2 = a.g2[jj];
            y3 = a.g3[jj];
          }
        }
        __syncwarp();
      }
    }
    for (int i = lane; i < len; i += 32) {
      double z = (acc[i] + acc[stride + i]) + acc[2 * stride + i];
      if (cols[i] == p) {
        if (p == a.zeroP && a.zeroP > 0) z *= 1000.0;  // blascoCodinaHuerta.cpp:4167-4180
        a.zdiag[p] = z;
      }
      a.zval[zb + i] = z;
    }
    __syncwarp();
  }
}

__global__ void k_to_float(long long n, const double* __restrict__ in, float* out) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    out[i] = (float)in[i];
}

__global__ void k_recip(long long n, const double* __restrict__ in, double* out64, float* out32) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    double r = 1.0 / in[i];
    if (out64) out64[i] = r;
    if (out32) out32[i] = (float)r;
  }
}

inline int grid_for(long long n, int threads, int cap = 148 * 32) {
  long long g = (n + threads - 1) / threads;
  if (g < 1) g = 1;
  if (g > cap) g = cap;
  return (int)g;
}

}  // namespace

cudaError_t launch_assemble(const AsmArgs& a, int num_sms, cudaStream_t s) {
  const int ne = a.e_end - a.e_begin;
  if (ne <= 0) return cudaSuccess;
  int grid = ne < num_sms * 16 ? ne : num_sms * 16;
  k_assemble<<<grid, kAsmThreads, 0, s>>>(a);
  return cudaGetLastError();
}

cudaError_t launch_fill_gt(long long nnz, const int* pos, const double* g1, const double* g2, const double* g3,
                           double* gt1, double* gt2, double* gt3, cudaStream_t s) {
  k_fill_gt<<<grid_for(nnz, 256), 256, 0, s>>>(nnz, pos, g1, g2, g3, gt1, gt2, gt3);
  return cudaGetLastError();
}

cudaError_t launch_md_finalize(int NN, const double* msum, const unsigned char* bcmask, double* minv_orig,
                               double* minv_free, cudaStream_t s) {
  k_md_finalize<<<grid_for(NN, 256), 256, 0, s>>>(NN, msum, bcmask, minv_orig, minv_free);
  return cudaGetLastError();
}

cudaError_t launch_build_z(const ZArgs& a, cudaStream_t s) {
  size_t smem = (size_t)kZWarps * a.maxrow * (3 * sizeof(double) + sizeof(int));
  if (smem > 200 * 1024) return cudaErrorInvalidValue;
  if (smem > 48 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(k_build_z, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
  }
  int grid = grid_for(a.NNp, kZWarps, 148 * 64);
  k_build_z<<<grid, 32 * kZWarps, smem, s>>>(a);
  return cudaGetLastError();
}

cudaError_t launch_to_float(long long n, const double* in, float* out, cudaStream_t s) {
  k_to_float<<<grid_for(n, 256), 256, 0, s>>>(n, in, out);
  return cudaGetLastError();
}

cudaError_t launch_recip(long long n, const double* in, double* out64, float* out32, cudaStream_t s) {
  k_recip<<<grid_for(n, 256), 256, 0, s>>>(n, in, out64, out32);
  return cudaGetLastError();
}

}  // namespace cfd
