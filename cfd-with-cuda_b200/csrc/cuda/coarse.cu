// Device side of the two-level pressure preconditioners (the coarse space is
// built by galerkin.cu and dense_chol.cu, or on the host by coarse.cpp):
// restriction c = P^T r onto the coarse
// lattice, the coarse solve e = Zc^-1 c as a dense matrix-vector product,
// and the combined preconditioner
//
//   z[p(v)] = D^-1 r[p(v)] + (P e)[v] + s/d * y[v]
//
// (Jacobi step, coarse correction, optional network correction y scaled by
// the residual's RMS s = sqrt(rr / n) and the median diagonal d).  Every
// kernel returns at once while the solve's done flag is set, so the sequence
// can sit inside a captured flexible-CG iteration.
#include <algorithm>

#include "common.cuh"
#include "kernels.h"

namespace cfd {

namespace {

// c = P^T r, separably: one block per coarse (iy, iz) pair and range of coarse
// x-nodes (blockIdx.y of nxs ranges).  The block's fine x-lines (the y-z support of
// the pair, weights wy wz kept in shared memory, set up before the wait for the
// previous kernel) are summed by G groups of threads, each thread one fine x
// over every G-th line (kRestrictBatch loads in flight), the group partials are
// added, and warps restrict the resulting fine x-line onto the coarse x-nodes.  G
// goes with the whole line's length, not with the range's, so that the order of a
// sum, and with it the last bit that decides how c rounds to FP32, is the same
// however the line is cut.  us per launch on the 24 x 24 x 160 duct, wait for the
// previous kernel included, batches of 4 / 8 / 16: 11.3 / 10.7 / 10.9; the loop
// unrolled by the compiler 14.1.
constexpr int kRestrictThreads = 512;
constexpr int kRestrictLines = 1024;  // y-z support lines per coarse pair at most
constexpr int kRestrictBatch = 8;
template <class VT>
__global__ void __launch_bounds__(kRestrictThreads) k_restrict(CoarseArgs<VT> a, const VT* r, float* c,
                                                               const int* done) {
  pdl_trigger();  // the coarse solve reads only constants before its wait
  extern __shared__ double sline[];  // G x W partial sums
  __shared__ double swt[kRestrictLines];
  __shared__ int sbase[kRestrictLines];
  const int cx = a.cd[0], cy = a.cd[1];
  const int iy = blockIdx.x % cy, iz = blockIdx.x / cy;
  const int ix0 = cx * blockIdx.y / gridDim.y, ix1 = cx * (blockIdx.y + 1) / gridDim.y;
  const int xb = a.rx[2 * ix0], W = a.rx[2 * (ix1 - 1) + 1] - xb + 1;  // fine x-range
  const int y0 = a.ry[2 * iy], ny = a.ry[2 * iy + 1] - y0 + 1;
  const int z0 = a.rz[2 * iz], nz = a.rz[2 * iz + 1] - z0 + 1;
  const int fx = a.fd[0], fxy = a.fd[0] * a.fd[1];
  const int nl = ny * nz;
  for (int l = threadIdx.x; l < nl; l += blockDim.x) {
    const int y = y0 + l % ny, z = z0 + l / ny;
    const double wy = a.i0y[y] == iy ? 1.0 - a.fy[y] : (a.i0y[y] + 1 == iy ? a.fy[y] : 0.0);
    const double wz = a.i0z[z] == iz ? 1.0 - a.fz[z] : (a.i0z[z] + 1 == iz ? a.fz[z] : 0.0);
    swt[l] = wy * wz;
    sbase[l] = xb + fx * y + fxy * z;
  }
  pdl_wait();
  if (done && *done) return;
  __syncthreads();
  const int G = fx <= (int)blockDim.x ? (int)blockDim.x / fx : 1;
  const int g = threadIdx.x / W;
  for (int x = threadIdx.x % W; g < G && x < W; x += (G == 1 ? (int)blockDim.x : W)) {
    double acc = 0.0;
    for (int l0 = g; l0 < nl; l0 += kRestrictBatch * G) {
      VT rv[kRestrictBatch];
#pragma unroll
      for (int u = 0; u < kRestrictBatch; u++) {
        const int l = l0 + u * G, v = l < nl ? sbase[l] + x : 0;
        rv[u] = l < nl ? r[a.pmap ? a.pmap[v] : v] : VT(0);
      }
#pragma unroll
      for (int u = 0; u < kRestrictBatch; u++) {
        const int l = l0 + u * G;
        if (l < nl) acc += swt[l] * (double)rv[u];
      }
    }
    sline[g * W + x] = acc;
    if (G != 1) break;
  }
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int ix = ix0 + warp; ix < ix1; ix += blockDim.x >> 5) {
    const int x0 = a.rx[2 * ix], x1 = a.rx[2 * ix + 1];
    double acc = 0.0;
    for (int x = x0 + lane; x <= x1; x += 32) {
      const double wx = a.i0x[x] == ix ? 1.0 - a.fx[x] : (a.i0x[x] + 1 == ix ? a.fx[x] : 0.0);
      double sx = 0.0;
      for (int gg = 0; gg < G; gg++) sx += sline[gg * W + x - xb];
      acc += wx * sx;
    }
    acc = warp_sum(acc);
    if (lane == 0) c[ix + cx * (iy + cy * iz)] = (float)acc;
  }
}

// sum_i h[i] c[i] over 8 FP16 entries packed in q and 8 FP32 values at c
__device__ __forceinline__ float dot8(const uint4& q, const float* c) {
  const __half2* h = reinterpret_cast<const __half2*>(&q);
  const float4 c0 = reinterpret_cast<const float4*>(c)[0], c1 = reinterpret_cast<const float4*>(c)[1];
  float2 f0 = __half22float2(h[0]), f1 = __half22float2(h[1]), f2 = __half22float2(h[2]), f3 = __half22float2(h[3]);
  return (f0.x * c0.x + f0.y * c0.y) + (f1.x * c0.z + f1.y * c0.w) + (f2.x * c1.x + f2.y * c1.y) +
         (f3.x * c1.z + f3.y * c1.w);
}

// e = inv c: one block of four warps per row, every thread with its share
// of the row's 16-byte loads (8 FP16 entries each) in flight at once and
// requested before the wait for c, FP32 products with c (read through L1),
// block sum.  The inverse is read with an evict-last L2 policy (the SpMV's
// matrix stream is evict-first), so it stays in L2 from one flexible-CG
// iteration to the next.
constexpr int kMvThreads = 128, kMvLoads = 6;  // 6 x 128 x 8 entries >= kCoarseMaxNodes of the solver
template <class VT>
__global__ void __launch_bounds__(kMvThreads) k_coarse_mv(int nc, int ld, const __half* __restrict__ inv, float rscale,
                                                          const float* c, VT* e, const int* done) {
  const int row = blockIdx.x;
  const int nv8 = nc >> 3, tail = nc & 7;  // whole 8-entry groups inside the row, then a tail
  const uint4* ir = reinterpret_cast<const uint4*>(inv + (size_t)row * ld);
  const unsigned long long keep = l2_evict_last();
  const int k = threadIdx.x;
  uint4 q[kMvLoads];
#pragma unroll
  for (int u = 0; u < kMvLoads; u++)
    if (k + u * kMvThreads < nv8) q[u] = ldg_hint(ir + k + u * kMvThreads, keep);
  pdl_wait();
  pdl_trigger();
  if (done && *done) return;
  // four chains over the first four loads where a thread has them all, one
  // chain otherwise and for the rest
  float s[4] = {0.f, 0.f, 0.f, 0.f};
  const bool four = k + 3 * kMvThreads < nv8;
#pragma unroll
  for (int u = 0; u < kMvLoads; u++)
    if (k + u * kMvThreads < nv8) s[four && u < 4 ? u : 0] += dot8(q[u], c + 8 * (k + u * kMvThreads));
  for (int kk = k + kMvLoads * kMvThreads; kk < nv8; kk += kMvThreads) s[0] += dot8(ldg_hint(ir + kk, keep), c + 8 * kk);
  if (threadIdx.x < tail) s[1] += __half2float(inv[(size_t)row * ld + 8 * nv8 + threadIdx.x]) * c[8 * nv8 + threadIdx.x];
  float t = warp_sum((s[0] + s[1]) + (s[2] + s[3]));
  __shared__ float sw[kMvThreads / 32];
  if ((threadIdx.x & 31) == 0) sw[threadIdx.x >> 5] = t;
  __syncthreads();
  if (threadIdx.x == 0) {
    float tot = 0.f;
#pragma unroll
    for (int w = 0; w < kMvThreads / 32; w++) tot += sw[w];
    e[row] = (VT)(tot * rscale);
  }
}

// z from r, dinv, e and y.  Only e is written by the kernel before, so all
// the rest of a thread's first voxel is loaded before the wait for it.
template <class VT>
__global__ void __launch_bounds__(256) k_precond(CoarseArgs<VT> a, int nv, const VT* __restrict__ r,
                                                 const VT* __restrict__ dinv, const VT* e,
                                                 const float* __restrict__ y, const double* rr, double dscale,
                                                 VT* z, const int* done) {
  pdl_trigger();  // the SpMV reads only the matrix before its wait
  const int cx = a.cd[0], cxy = a.cd[0] * a.cd[1];
  const int bx = a.cd[0] > 1, by = a.cd[1] > 1, bz = a.cd[2] > 1;
  int p = 0, e0 = 0;
  VT jac = 0, fx = 0, fy = 0, fz = 0, net = 0;
  auto load = [&](int v) {
    p = a.pmap ? a.pmap[v] : v;
    jac = dinv[p] * r[p];
    if (e) {
      const int x = v % a.fd[0], yy = (v / a.fd[0]) % a.fd[1], zz = v / (a.fd[0] * a.fd[1]);
      e0 = a.i0x[x] + cx * a.i0y[yy] + cxy * a.i0z[zz];
      fx = (VT)a.fx[x], fy = (VT)a.fy[yy], fz = (VT)a.fz[zz];
    }
    if (y) net = (VT)y[v];
  };
  int v = blockIdx.x * blockDim.x + threadIdx.x;
  bool loaded = v < nv;
  if (loaded) load(v);
  pdl_wait();
  if (done && *done) return;
  VT ys = 0;
  if (y) ys = (VT)(rr[0] > 0.0 ? sqrt(rr[0] / (double)nv) / dscale : 0.0);
  for (; v < nv; v += gridDim.x * blockDim.x) {
    if (!loaded) load(v);
    loaded = false;
    VT zi = jac;
    if (e) {
      VT s = 0;
#pragma unroll
      for (int cnr = 0; cnr < 8; cnr++) {
        const int dx = cnr & 1, dy = (cnr >> 1) & 1, dz = cnr >> 2;
        if ((dx && !bx) || (dy && !by) || (dz && !bz)) continue;
        const VT w = (dx ? fx : 1 - fx) * (dy ? fy : 1 - fy) * (dz ? fz : 1 - fz);
        s += w * e[e0 + dx + cx * dy + cxy * dz];
      }
      zi += s;
    }
    if (y) zi += net * ys;
    z[p] = zi;
  }
}

int grid_of(long long n, int threads) {
  long long g = (n + threads - 1) / threads;
  return (int)(g < 148 * 16 ? (g < 1 ? 1 : g) : 148 * 16);
}

}  // namespace

template <class VT>
cudaError_t launch_coarse_restrict(const CoarseArgs<VT>& a, const VT* r, float* c, const int* done, cudaStream_t s) {
  // shared memory: G groups x W partials (G = 1 once the range exceeds the block)
  if (a.fd[0] > 4096) return cudaErrorInvalidValue;
  for (int ax = 1; ax < 3; ax++) {  // support lines of a coarse pair: at most (2 h + 1)^2
    const double h = a.cd[ax] > 1 ? (double)(a.fd[ax] - 1) / (a.cd[ax] - 1) : 1.0;
    if (h > 15.0) return cudaErrorInvalidValue;
  }
  // ranges of coarse x-nodes: two blocks per SM, at least eight nodes each (the
  // fine ranges of neighbours overlap by a support); 49 pairs of the 24 x 24 x 160
  // duct: 10.3 us in one range, 5.3 in five (each launched alone)
  const int pairs = a.cd[1] * a.cd[2];
  const int nxs = std::max(1, std::min((2 * a.num_sms + pairs - 1) / pairs, a.cd[0] / 8));
  const size_t sm = (size_t)std::max(kRestrictThreads, a.fd[0]) * sizeof(double);
  return launch_k(a.pdl != 0, k_restrict<VT>, dim3(pairs, nxs), dim3(kRestrictThreads), sm, s, a, r, c, done);
}

template <class VT>
cudaError_t launch_coarse_solve(const CoarseArgs<VT>& a, const float* c, VT* e, const int* done, cudaStream_t s) {
  if (a.ldinv % 8 || a.ldinv < a.nc) return cudaErrorInvalidValue;
  return launch_k(a.pdl != 0, k_coarse_mv<VT>, dim3(a.nc), dim3(kMvThreads), 0, s, a.nc, a.ldinv, a.inv16,
                  (float)(1.0 / a.inv_scale), c, e, done);
}

template <class VT>
cudaError_t launch_precond(const CoarseArgs<VT>& a, int nv, const VT* r, const VT* dinv, const VT* e, const float* y,
                           const double* rr, double dscale, VT* z, const int* done, cudaStream_t s) {
  return launch_k(a.pdl != 0, k_precond<VT>, dim3(grid_of(nv, 256)), dim3(256), 0, s, a, nv, r, dinv, e, y, rr,
                  dscale, z, done);
}

template cudaError_t launch_coarse_restrict<float>(const CoarseArgs<float>&, const float*, float*, const int*,
                                                   cudaStream_t);
template cudaError_t launch_coarse_restrict<double>(const CoarseArgs<double>&, const double*, float*, const int*,
                                                    cudaStream_t);
template cudaError_t launch_coarse_solve<float>(const CoarseArgs<float>&, const float*, float*, const int*,
                                                cudaStream_t);
template cudaError_t launch_coarse_solve<double>(const CoarseArgs<double>&, const float*, double*, const int*,
                                                 cudaStream_t);
template cudaError_t launch_precond<float>(const CoarseArgs<float>&, int, const float*, const float*, const float*,
                                           const float*, const double*, double, float*, const int*, cudaStream_t);
template cudaError_t launch_precond<double>(const CoarseArgs<double>&, int, const double*, const double*,
                                            const double*, const float*, const double*, double, double*, const int*,
                                            cudaStream_t);

}  // namespace cfd
