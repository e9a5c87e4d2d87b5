// Jacobi-preconditioned CG on a caller-provided CSR system that allocates
// no device memory: cfd_pcg_solve_noalloc.
//
// Who needs it: callers that cannot call cudaMalloc/cudaFree while they run
// the pressure solve.  A coupled multi-physics code that keeps other streams
// busy cannot afford cudaFree, which synchronizes the whole device; a host
// application that reserves all of its device memory up front through its
// own pool allocator cannot let a library allocate at solve time, where an
// allocation could fail in the middle of a run.  Such callers own the matrix,
// right-hand side and solution buffers and pass them in; the published work
// vector, per-block partial sums, the barrier words and the result live in
// one file-scope static device array of fixed size.
//
// Limits and rules:
//   - n <= CFD_NOALLOC_MAX_N (524288 rows, a 80^3 pressure grid); larger
//     systems are rejected with CFD_E_BADARG and a message.
//   - every GPU that calls it holds the array (4.1 MiB; with fewer than 103 SMs 12 MiB
//     more) until the process exits;
//   - the first call on a device looks the array's device address up
//     (cudaGetSymbolAddress, once per device, with that device current); make
//     that first call before any stream capture;
//   - all calls share the array and it keeps the last call's contents; the
//     barrier words and the error flag are cleared on every call, the work
//     vector is fully rewritten before use.  Calls that overlap on the GPU
//     (two streams, or two host threads) race on the array and must not be
//     issued.
// The algorithm is the solver's FP64 Jacobi-PCG: x0 = 0, stop when
// ||r||_2 <= rtol ||b||_2, one persistent cooperative kernel with bounded
// grid barriers.
//
// The iteration is Chronopoulos and Gear's form of CG (1989; the same
// iterates as the textbook form): with u = D^-1 r and w = A u, the step
// lengths come from (r, u) and (w, u) of the same iteration, so one reduction
// and one publication of u are the only grid-wide waits.  Everything but u
// is used by the block that owns the rows only and stays in its shared
// memory: r, p, s, w and x.  A device or partition whose SMs cannot hold them (fewer
// than 103 for the largest n) keeps p, s and w in a second array (pcg_noalloc_spill.cu),
// x in the caller's vector, and publishes r, from which u = D^-1 r is formed
// where it is read.
//
// What bounds it: the matrix stream (12 bytes per non-zero; up to about 9 M
// non-zeros it stays in L2 between iterations) and the two waits.  One block
// of 1024 threads per SM keeps the waits short (148 arrivals, 148 partial
// sums).  A block owns a contiguous range of rows, so the gathers of u stay
// in its L1; a row is summed by a group of G lanes, G chosen from the mean row
// length so that a row takes about four loads per lane, all in flight at
// once.  Measured on a 27-point operator with 65 x 63 x 61 rows (rtol 1e-8,
// 273 iterations): 82 us per iteration with a warp per row, 1184 blocks, all
// vectors in L2 and three waits; 34 us with the row groups and 148 blocks; 31
// us in this form; 27 us with two rows per group at once and the row extents
// read ahead.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <mutex>

#include "../../../include/cfdfs.h"
#include "common.cuh"

namespace cfd {

// Device address of 3 CFD_NOALLOC_MAX_N doubles, placed on the device by the first
// call (pcg_noalloc_spill.cu).
cudaError_t noalloc_spill(double** p);

namespace {

constexpr int kThreads = 1024;
constexpr int kMaxN = CFD_NOALLOC_MAX_N;
constexpr int kMaxBlocks = 2048;
constexpr int kMaxDevices = 64;
// layout of the scratch array (bytes)
constexpr size_t kVecBytes = (size_t)kMaxN * sizeof(double);
constexpr size_t kOffU = 0;  // u (or r); the other vectors live in shared memory
constexpr size_t kOffPart = kVecBytes;                                    // 6 x kMaxBlocks doubles
constexpr size_t kOffCtl = kOffPart + 6 * (size_t)kMaxBlocks * sizeof(double);  // barrier[2], err, pad
constexpr size_t kOffRes = kOffCtl + 256;                                       // 4 doubles
constexpr size_t kScratchBytes = kOffRes + 256;
constexpr size_t kMaxDynSmem = 200 * 1024;
constexpr unsigned long long kTimeoutNs = 2000000000ULL;

static __device__ __align__(256) unsigned char g_noalloc_scratch[kScratchBytes];

// Grid-wide wait number k (1, 2, ...) of the launch on a monotonic arrival
// counter (host-zeroed): every block has arrived k times.  Returns false in
// every thread of the block when the bounded wait gives up or another block
// has raised *err.  With NV > 0 also sums NV values over the grid: v in, the
// total out, every block adding the posted partials in the same order.
struct GridSync {
  unsigned* cnt;
  int* err;
  double* part;
  unsigned long long timeout_ns;
  unsigned extra[2];  // 0; a self-test's arrivals that never come [wait<0>, wait<3>]
  unsigned k;
  template <int NV>
  __device__ __forceinline__ bool wait(double (&v)[NV > 0 ? NV : 1]) {
    __shared__ double res[NV > 0 ? NV : 1];
    __shared__ int s_ok;
    const int G = gridDim.x;
    if (G == 1) {  // one block: no one to wait for
      if constexpr (NV > 0) {
        block_sum<NV>(v);
        if (threadIdx.x == 0)
          for (int i = 0; i < NV; i++) res[i] = v[i];
      }
      __syncthreads();
      if constexpr (NV > 0)
        for (int i = 0; i < NV; i++) v[i] = res[i];
      __syncthreads();
      return true;
    }
    k++;
    double* buf = part + (size_t)(k & 1) * 3 * G;
    if constexpr (NV > 0) {
      block_sum<NV>(v);
      if (threadIdx.x == 0)
        for (int i = 0; i < NV; i++) buf[(size_t)i * G + blockIdx.x] = v[i];
    } else {
      __syncthreads();
    }
    if (threadIdx.x < 32) {
      if (threadIdx.x == 0) {
        __threadfence();
        red_add_release_u32(cnt, 1u);
      }
      __syncwarp();
      const unsigned target = k * (unsigned)G + extra[NV > 0];
      int ok = 1;
      if (ld_acquire_u32(cnt) < target) {
        const unsigned long long t0 = global_ns();
        while (ld_acquire_u32(cnt) < target) {
          if (ld_volatile_i32(err) || global_ns() - t0 > timeout_ns) {
            ok = 0;
            break;
          }
        }
      }
      ok = __all_sync(0xffffffffu, ok);
      if (!ok && threadIdx.x == 0) atomicExch(err, 1);
      __threadfence();
      if constexpr (NV > 0) {
        for (int i = 0; i < NV; i++) {
          double s = 0;
          for (int b = threadIdx.x; b < G; b += 32) s += __ldcg(buf + (size_t)i * G + b);
          s = warp_sum(s);
          if (threadIdx.x == 0) res[i] = s;
        }
      }
      if (threadIdx.x == 0) s_ok = ok;
    }
    __syncthreads();
    if constexpr (NV > 0)
      for (int i = 0; i < NV; i++) v[i] = res[i];
    const bool r = s_ok != 0;
    __syncthreads();
    return r;
  }
};

// read-once loads that leave the L1 to the gathered vector
__device__ __forceinline__ int ldg_stream(const int* p) {
  int v;
  asm volatile("ld.global.nc.L1::no_allocate.s32 %0, [%1];" : "=r"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ double ldg_stream(const double* p) {
  double v;
  asm volatile("ld.global.nc.L1::no_allocate.f64 %0, [%1];" : "=d"(v) : "l"(p));
  return v;
}

// w = A u on the block's rows r0 .. r0 + nr, G lanes per row (w in shared
// memory, or global with SPILL); returns the thread's part of (w, u).  u, or with SPILL
// the r of u = D^-1 r, is read with plain loads: other blocks' parts of it are visible
// after the grid-wide wait before.
template <int G, bool SPILL>
__device__ __forceinline__ double spmv_rows(int r0, int nr, const int* __restrict__ rp, const int* __restrict__ col,
                                            const double* __restrict__ val, const double* __restrict__ dinv,
                                            const double* u, double* w) {
  auto at = [&](int i) { return SPILL ? u[i] * __ldg(dinv + i) : u[i]; };
  constexpr int R = 2, STEP = kThreads / G;  // rows per group at once, rows of a pass
  const int lane = threadIdx.x % G;
  double wu = 0;
  // the groups of a warp stay together (the sums below are warp-wide); the
  // next rows' extents are read ahead of this pass's entries
  const int base0 = (int)(threadIdx.x & ~31) / G, sub = (int)(threadIdx.x & 31) / G;
  int nb[R], ne[R];
#pragma unroll
  for (int k = 0; k < R; k++) {
    const int i = base0 + sub + k * STEP;
    nb[k] = i < nr ? __ldg(rp + r0 + i) : 0;
    ne[k] = i < nr ? __ldg(rp + r0 + i + 1) : 0;
  }
  for (int base = base0; base < nr; base += R * STEP) {
    int b[R], e[R], c[R][4];
    double v[R][4], s[R];
#pragma unroll
    for (int k = 0; k < R; k++) {
      b[k] = nb[k] + lane;
      e[k] = ne[k];
#pragma unroll
      for (int q = 0; q < 4; q++) {
        const int j = b[k] + q * G;
        c[k][q] = j < e[k] ? ldg_stream(col + j) : -1;
        v[k][q] = j < e[k] ? ldg_stream(val + j) : 0.0;
      }
    }
#pragma unroll
    for (int k = 0; k < R; k++) {
      const int i = base + sub + (R + k) * STEP;
      nb[k] = i < nr ? __ldg(rp + r0 + i) : 0;
      ne[k] = i < nr ? __ldg(rp + r0 + i + 1) : 0;
    }
#pragma unroll
    for (int k = 0; k < R; k++) {
      s[k] = 0;
#pragma unroll
      for (int q = 0; q < 4; q++)
        if (c[k][q] >= 0) s[k] += v[k][q] * at(c[k][q]);
      for (int j = b[k] + 4 * G; j < e[k]; j += G) s[k] += ldg_stream(val + j) * at(ldg_stream(col + j));
      s[k] = group_sum<G>(s[k]);
      const int i = base + sub + k * STEP;
      if (i < nr && lane == 0) {
        w[i] = s[k];
        wu += at(r0 + i) * s[k];
      }
    }
  }
  return wu;
}

template <bool SPILL>
__global__ void __launch_bounds__(kThreads, 1) k_pcg_noalloc(int n, const int* __restrict__ rp,
                                                              const int* __restrict__ col,
                                                              const double* __restrict__ val,
                                                              const double* __restrict__ dinv,
                                                              const double* __restrict__ b, double* xout, double rtol,
                                                              int maxit, unsigned char* scratch, double* spill,
                                                              unsigned long long timeout_ns, unsigned extra0,
                                                              unsigned extra1) {
  extern __shared__ double sv[];
  const int r0 = (int)((long long)n * blockIdx.x / gridDim.x);
  const int nr = (int)((long long)n * (blockIdx.x + 1) / gridDim.x) - r0;
  double* u = reinterpret_cast<double*>(scratch + kOffU);
  double* const r = SPILL ? u + r0 : sv;
  double* const p = SPILL ? spill + r0 : r + nr;
  double* const s = SPILL ? spill + kMaxN + r0 : p + nr;
  double* const w = SPILL ? spill + 2 * (size_t)kMaxN + r0 : s + nr;
  double* const x = SPILL ? xout + r0 : w + nr;
  double* result = reinterpret_cast<double*>(scratch + kOffRes);
  GridSync gs{reinterpret_cast<unsigned*>(scratch + kOffCtl), reinterpret_cast<int*>(scratch + kOffCtl + 8),
              reinterpret_cast<double*>(scratch + kOffPart), timeout_ns, {extra0, extra1}, 0u};
  // lanes per row: about four loads per lane for a row of the mean length
  const int mean = (int)(((long long)__ldg(rp + n) - __ldg(rp)) / n);
  double ru = 0, rr = 0, none[1];
  for (int i = threadIdx.x; i < nr; i += kThreads) {
    const double bi = b[r0 + i], ui = bi * dinv[r0 + i];
    r[i] = bi;
    p[i] = s[i] = x[i] = 0.0;
    if (!SPILL) u[r0 + i] = ui;
    ru += bi * ui;
    rr += bi * bi;
  }
  bool alive = gs.wait<0>(none);
  double bnorm = 0, tol = 0, rn = 0, gamma_old = 1, alpha_old = 1;
  int its = 0, status = 1;
  while (true) {
    if (!alive) { status = 3; break; }
    double v[3] = {ru, 0.0, rr};
    if (mean <= 8)
      v[1] = spmv_rows<2, SPILL>(r0, nr, rp, col, val, dinv, u, w);
    else if (mean <= 16)
      v[1] = spmv_rows<4, SPILL>(r0, nr, rp, col, val, dinv, u, w);
    else if (mean <= 32)
      v[1] = spmv_rows<8, SPILL>(r0, nr, rp, col, val, dinv, u, w);
    else if (mean <= 64)
      v[1] = spmv_rows<16, SPILL>(r0, nr, rp, col, val, dinv, u, w);
    else
      v[1] = spmv_rows<32, SPILL>(r0, nr, rp, col, val, dinv, u, w);
    if (!gs.wait<3>(v)) { status = 3; break; }
    const double gamma = v[0], delta = v[1];
    rn = sqrt(v[2]);
    if (its == 0) {
      bnorm = rn;
      tol = rtol * bnorm;
    }
    if (!isfinite(rn)) { status = 2; break; }
    if (rn <= tol) { status = 0; break; }
    if (its >= maxit) break;
    const double beta = its > 0 ? gamma / gamma_old : 0.0;
    const double alpha = its > 0 ? gamma / (delta - beta * gamma / alpha_old) : gamma / delta;
    gamma_old = gamma;
    alpha_old = alpha;
    ru = rr = 0;
    for (int i = threadIdx.x; i < nr; i += kThreads) {
      const double di = dinv[r0 + i];
      const double pi = (SPILL ? r[i] * di : u[r0 + i]) + beta * p[i], si = w[i] + beta * s[i];
      const double ri = r[i] - alpha * si, ui = ri * di;
      p[i] = pi;
      s[i] = si;
      x[i] += alpha * pi;
      r[i] = ri;
      if (!SPILL) u[r0 + i] = ui;
      ru += ri * ui;
      rr += ri * ri;
    }
    its++;
    alive = gs.wait<0>(none);
  }
  if (!SPILL)
    for (int i = threadIdx.x; i < nr; i += kThreads) xout[r0 + i] = x[i];
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    result[0] = its;
    result[1] = bnorm > 0 ? rn / bnorm : 0.0;
    result[2] = status;
    result[3] = bnorm;
  }
}

std::mutex g_setup_mutex;
void* g_scratch_addr[kMaxDevices] = {};
double* g_spill_addr[kMaxDevices] = {};

size_t block_smem(int n, long long grid) { return 5 * sizeof(double) * (size_t)((n + grid - 1) / grid); }

void put_err(char* buf, int len, const char* msg) {
  if (buf && len > 0) std::snprintf(buf, (size_t)len, "%s", msg);
}

}  // namespace

cudaError_t noalloc_selftest(int which, unsigned long long timeout_ns, const int* rp, const int* col, const double* val,
                             const double* dinv, const double* b, double* x, int n, double* status, cudaStream_t s) {
  void* p = nullptr;
  cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
  if (e != cudaSuccess) return e;
  unsigned char* base = static_cast<unsigned char*>(p);
  const int grid = 4;
  double rtol = 1e-10;
  int maxit = 200;
  double* spill = nullptr;
  unsigned extra[2] = {which == 0 ? 1u : 0u, which == 1 ? 1u : 0u};
  void* params[] = {&n, (void*)&rp, (void*)&col, (void*)&val, (void*)&dinv, (void*)&b, (void*)&x,
                    &rtol, &maxit, &base, &spill, &timeout_ns, &extra[0], &extra[1]};
  e = cudaFuncSetAttribute(k_pcg_noalloc<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxDynSmem);
  if (e == cudaSuccess) e = cudaMemsetAsync(base + kOffCtl, 0, 256, s);
  if (e == cudaSuccess)
    e = cudaLaunchCooperativeKernel((const void*)k_pcg_noalloc<false>, dim3(grid), dim3(kThreads), params,
                                    block_smem(n, grid), s);
  double res[4] = {0, 0, -1, 0};
  if (e == cudaSuccess) e = cudaMemcpyAsync(res, base + kOffRes, sizeof(res), cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  *status = res[2];
  return e;
}

}  // namespace cfd

extern "C" int cfd_pcg_solve_noalloc(const int* rowptr, const int* col, const double* val, const double* dinv,
                                     const double* b, double* x, int n, double rtol, int maxit, void* stream,
                                     double* info, char* errbuf, int errlen) {
  using namespace cfd;
  char msg[256];
  if (n <= 0 || n > kMaxN) {
    std::snprintf(msg, sizeof(msg), "cfd_pcg_solve_noalloc: n = %d is outside 1..%d (the size of its static work array)",
                  n, kMaxN);
    put_err(errbuf, errlen, msg);
    return CFD_E_BADARG;
  }
  if (!rowptr || !col || !val || !dinv || !b || !x || !(rtol > 0) || maxit <= 0) {
    put_err(errbuf, errlen, "cfd_pcg_solve_noalloc: null pointer, rtol <= 0 or maxit <= 0");
    return CFD_E_BADARG;
  }
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess || dev < 0 || dev >= kMaxDevices) {
    put_err(errbuf, errlen, "cfd_pcg_solve_noalloc: no current CUDA device");
    return CFD_E_CUDA;
  }
  int sms = 0;
  e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  // CFD_NOALLOC_SMS=<k>: as on a device of k SMs
  if (const char* lim = std::getenv("CFD_NOALLOC_SMS")) sms = std::max(1, std::min(sms, std::atoi(lim)));
  if (e != cudaSuccess || sms < 1) {
    put_err(errbuf, errlen, "cfd_pcg_solve_noalloc: no SM count");
    return CFD_E_CUDA;
  }
  sms = std::min(sms, kMaxBlocks);
  void* scratch = nullptr;
  double* spill = nullptr;
  {
    std::lock_guard<std::mutex> lock(g_setup_mutex);
    e = cudaSuccess;
    if (!g_scratch_addr[dev]) e = cudaGetSymbolAddress(&g_scratch_addr[dev], g_noalloc_scratch);
    if (e == cudaSuccess && !g_spill_addr[dev] && block_smem(kMaxN, sms) > kMaxDynSmem)
      e = noalloc_spill(&g_spill_addr[dev]);
    if (e != cudaSuccess) {
      std::snprintf(msg, sizeof(msg), "cfd_pcg_solve_noalloc: cudaGetSymbolAddress failed: %s", cudaGetErrorString(e));
      put_err(errbuf, errlen, msg);
      return CFD_E_CUDA;
    }
    scratch = g_scratch_addr[dev];
    spill = g_spill_addr[dev];
  }
  cudaStream_t s = (cudaStream_t)stream;
  // one block per SM, at least 256 rows each: a small system waits on fewer
  // arrivals, and one block on none, so up to 512 rows stay on one (512 rows
  // of 27: 6.8 us per iteration, two blocks 9.2; 8000 rows: 9.5 us on 32
  // blocks, 11.3 on 16)
  const long long grid = std::min<long long>(sms, n <= 512 ? 1 : (n + 255) / 256);
  size_t smem = block_smem(n, grid);
  const bool in_smem = smem <= kMaxDynSmem;
  const void* kernel = in_smem ? (const void*)k_pcg_noalloc<false> : (const void*)k_pcg_noalloc<true>;
  if (!in_smem) smem = 0;
  e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxDynSmem);
  if (e != cudaSuccess) {
    put_err(errbuf, errlen, "cfd_pcg_solve_noalloc: the device cannot hold the block vectors");
    return CFD_E_CUDA;
  }
  unsigned char* base = static_cast<unsigned char*>(scratch);
  e = cudaMemsetAsync(base + kOffCtl, 0, 256, s);  // barrier words and error flag start at zero
  if (e == cudaSuccess) {
    int nn = n, mi = maxit;
    double rt = rtol;
    unsigned char* sp = base;
    unsigned long long timeout_ns = kTimeoutNs;
    unsigned none = 0;
    void* params[] = {&nn, (void*)&rowptr, (void*)&col, (void*)&val, (void*)&dinv, (void*)&b, (void*)&x,
                      &rt, &mi, &sp, &spill, &timeout_ns, &none, &none};
    e = cudaLaunchCooperativeKernel(kernel, dim3((unsigned)grid), dim3(kThreads), params, smem, s);
  }
  double res[4] = {0, 0, 0, 0};
  if (e == cudaSuccess) e = cudaMemcpyAsync(res, base + kOffRes, sizeof(res), cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  if (e != cudaSuccess) {
    std::snprintf(msg, sizeof(msg), "cfd_pcg_solve_noalloc: %s", cudaGetErrorString(e));
    put_err(errbuf, errlen, msg);
    return CFD_E_CUDA;
  }
  if (info) {
    info[0] = res[0];
    info[1] = res[1];
    info[2] = res[2];
  }
  switch ((int)res[2]) {
    case 0: return CFD_OK;
    case 1: put_err(errbuf, errlen, "cfd_pcg_solve_noalloc: iteration limit reached"); return CFD_E_NOCONV;
    case 2: put_err(errbuf, errlen, "cfd_pcg_solve_noalloc: non-finite residual"); return CFD_E_NONFINITE;
    default: put_err(errbuf, errlen, "cfd_pcg_solve_noalloc: bounded grid barrier timed out"); return CFD_E_TIMEOUT;
  }
}
