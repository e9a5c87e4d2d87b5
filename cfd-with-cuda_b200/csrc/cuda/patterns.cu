// CSR patterns of the operators built on the device from the element map
// (the host build is build_patterns in host/mesh.cpp; both give sorted rows
// of distinct columns, so the patterns are identical):
//   K  (NN x NN):   row r = the 27 nodes of every element around node r;
//   G  (NN x NNp):  row r = the 8 corner (pressure) nodes of those elements;
//   G^T (NNp x NN): row p = K's row p (the 27 nodes of the elements around
//                   corner p), so it is K's first NNp rows;
//   Z  (NNp x NNp): row p = the corners of every element that shares a node
//                   with an element around p (Z = G^T diag G).
// A row's candidates are sorted (bitonic) and the first of each run is kept; a
// first pass counts, the host turns the counts into row pointers, a second pass
// writes the columns.  One warp per row sorts in registers, 512 candidates at
// most (K rows of a hexahedral mesh have 27 to 216, Z rows 216 and then 512); the
// rows with more go to a list that a kernel with one block per row works off in
// shared memory.  A row with more candidates than a block holds raises a flag,
// and the caller falls back to the host build.
#include <algorithm>
#include <climits>

#include "common.cuh"
#include "kernels.h"

namespace cfd {

namespace {

constexpr int kPatThreads = 256;
constexpr int kPatCap = 2048;  // candidates a block sorts (8 per thread)

__global__ void k_inc_count(long long nent, const int* __restrict__ ltog, int* __restrict__ cnt) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < nent; i += (long long)gridDim.x * blockDim.x)
    atomicAdd(cnt + ltog[i], 1);
}

__global__ void k_inc_fill(long long nent, const int* __restrict__ ltog, int* __restrict__ pos, int* __restrict__ inc_el) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < nent; i += (long long)gridDim.x * blockDim.x) {
    const int slot = atomicAdd(pos + ltog[i], 1);
    inc_el[slot] = (int)(i / 27);
  }
}

// In-place ascending bitonic sort of s[0, n), n a power of two <= kPatCap.
__device__ void block_sort(int* s, int n) {
  for (int k = 2; k <= n; k <<= 1)
    for (int j = k >> 1; j > 0; j >>= 1) {
      for (int i = threadIdx.x; i < n; i += blockDim.x) {
        const int l = i ^ j;
        if (l > i) {
          const int a = s[i], b = s[l];
          const bool up = (i & k) == 0;
          if ((a > b) == up) {
            s[i] = b;
            s[l] = a;
          }
        }
      }
      __syncthreads();
    }
}

// After block_sort: the number of distinct values below INT_MAX in s[0, n);
// with out, also writes them in order (out[0 .. count)).  Uses sflag (n ints)
// and swarp (kPatThreads / 32 ints) as scratch.
__device__ int block_unique(const int* s, int n, int* sflag, int* swarp, int* out) {
  // each thread owns a contiguous run of n / blockDim.x (at least 1) slots
  const int per = (n + blockDim.x - 1) / blockDim.x;
  const int b = threadIdx.x * per, e = min(n, b + per);
  int c = 0;
  for (int i = b; i < e; i++) {
    const int f = s[i] != INT_MAX && (i == 0 || s[i] != s[i - 1]);
    sflag[i] = f;
    c += f;
  }
  // exclusive prefix of c over the block
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int x = c;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) swarp[warp] = x;
  __syncthreads();
  if (warp == 0) {
    int w = lane < (int)(blockDim.x >> 5) ? swarp[lane] : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, w, o);
      if (lane >= o) w += y;
    }
    if (lane < (int)(blockDim.x >> 5)) swarp[lane] = w;  // inclusive per warp
  }
  __syncthreads();
  const int total = swarp[(blockDim.x >> 5) - 1];
  int pos = x - c + (warp > 0 ? swarp[warp - 1] : 0);
  if (out)
    for (int i = b; i < e; i++)
      if (sflag[i]) out[pos++] = s[i];
  __syncthreads();
  return total;
}

__device__ __forceinline__ int pow2_at_least(int n) {
  int p = 32;
  while (p < n) p <<= 1;
  return p;
}

// ---- one warp per row ----
// Bound by the issue of compare-exchanges (no barriers, no shared-memory
// round trips inside the sort).  Both passes of K, G and the element adjacency
// of 30^3 elements took 5.1 ms with a block of 256 threads per row, which sorts
// 27 to 216 values with up to 36 barriers, and Z's 1.9; with a warp per row 0.50 and
// 0.36.
constexpr int kWarpCap = 512;  // candidates of a warp: 16 registers per lane
constexpr int kWarpsPerBlock = kPatThreads / 32;

// Ascending bitonic sort of 32 R values, value i = 32 e + lane in v[e].
template <int R>
__device__ __forceinline__ void warp_sort(int (&v)[R], int lane) {
#pragma unroll
  for (int k = 2; k <= 32 * R; k <<= 1)
#pragma unroll
    for (int j = k >> 1; j > 0; j >>= 1) {
      if (j >= 32) {
#pragma unroll
        for (int e = 0; e < R; e++)
          if ((e & (j >> 5)) == 0) {
            const int a = v[e], b = v[e | (j >> 5)];
            const bool up = ((32 * e) & k) == 0;
            v[e] = up ? min(a, b) : max(a, b);
            v[e | (j >> 5)] = up ? max(a, b) : min(a, b);
          }
      } else {
#pragma unroll
        for (int e = 0; e < R; e++) {
          const int b = __shfl_xor_sync(0xffffffffu, v[e], j);
          const bool up = ((32 * e + lane) & k) == 0, low = (lane & j) == 0;
          v[e] = up == low ? min(v[e], b) : max(v[e], b);
        }
      }
    }
}

// Number of distinct values of buf[0, count), all >= 0; with out, also writes
// them in ascending order.  Called by a whole warp, count <= 32 R.
template <int R>
__device__ __forceinline__ int warp_unique(const int* buf, int count, int* out, int lane) {
  int v[R];
#pragma unroll
  for (int e = 0; e < R; e++) v[e] = 32 * e + lane < count ? buf[32 * e + lane] : INT_MAX;
  warp_sort<R>(v, lane);
  int total = 0, before = -1;
#pragma unroll
  for (int e = 0; e < R; e++) {
    int p = __shfl_up_sync(0xffffffffu, v[e], 1);
    if (lane == 0) p = before;
    before = __shfl_sync(0xffffffffu, v[e], 31);
    const bool first = v[e] != INT_MAX && v[e] != p;
    const unsigned m = __ballot_sync(0xffffffffu, first);
    if (first && out) out[total + __popc(m & ((1u << lane) - 1))] = v[e];
    total += __popc(m);
  }
  return total;
}
__device__ __forceinline__ int warp_unique_n(const int* buf, int count, int* out, int lane) {
  if (count <= 32) return warp_unique<1>(buf, count, out, lane);
  if (count <= 64) return warp_unique<2>(buf, count, out, lane);
  if (count <= 128) return warp_unique<4>(buf, count, out, lane);
  if (count <= 256) return warp_unique<8>(buf, count, out, lane);
  return warp_unique<16>(buf, count, out, lane);
}
// Exclusive prefix sum over the warp; total: the sum.
__device__ __forceinline__ int warp_scan(int d, int lane, int& total) {
  int x = d;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  total = __shfl_sync(0xffffffffu, x, 31);
  return x - d;
}

// The rows of a mode (0 to 2 as in k_rows, 3: Z as in k_zrows).  Rows that a
// warp cannot hold are left out; pass 0 puts them on the list.
template <int MODE>
__global__ void __launch_bounds__(kPatThreads) k_rows_warp(PatArgs a, int nrows, int pass) {
  __shared__ int sbuf[kWarpsPerBlock][kWarpCap];
  __shared__ int ssel[MODE == 3 ? kWarpsPerBlock : 1][MODE == 3 ? kWarpCap : 1];
  const int wib = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int* buf = sbuf[wib];
  for (int r = blockIdx.x * kWarpsPerBlock + wib; r < nrows; r += gridDim.x * kWarpsPerBlock) {
    __syncwarp();  // the last row's reads of buf
    int count = 0;
    bool fits = true;
    if constexpr (MODE < 2) {
      constexpr int nj = MODE == 0 ? 27 : 8;
      const int t0 = a.inc_rp[r], deg = a.inc_rp[r + 1] - t0;
      fits = deg <= kWarpCap / nj;
      count = fits ? deg * nj : 0;
      for (int i = lane; i < count; i += 32) buf[i] = a.ltog[(size_t)a.inc_el[t0 + i / nj] * 27 + i % nj];
    } else if constexpr (MODE == 2) {
      int t0 = 0, d = 0;
      if (lane < 27) {
        const int v = a.ltog[(size_t)r * 27 + lane];
        t0 = a.inc_rp[v];
        d = a.inc_rp[v + 1] - t0;
      }
      fits = __all_sync(0xffffffffu, d <= kWarpCap);  // so that the sum cannot overflow
      const int o = warp_scan(fits ? d : 0, lane, count);
      fits = fits && count <= kWarpCap;
      if (fits)
        for (int t = 0; t < d; t++) buf[o + t] = a.inc_el[t0 + t];
    } else {
      const int t0 = a.inc_rp[r], deg = a.inc_rp[r + 1] - t0;
      fits = deg <= 32;
      int b = 0, d = 0;
      if (fits && lane < deg) {
        const int e = a.inc_el[t0 + lane];
        b = a.adj_rp[e];
        d = a.adj_rp[e + 1] - b;
      }
      fits = fits && __all_sync(0xffffffffu, d <= kWarpCap);
      const int o = warp_scan(fits ? d : 0, lane, count);
      fits = fits && count <= kWarpCap;
      if (fits) {
        for (int q = 0; q < deg; q++) {
          const int bq = __shfl_sync(0xffffffffu, b, q), dq = __shfl_sync(0xffffffffu, d, q);
          const int oq = __shfl_sync(0xffffffffu, o, q);
          for (int t = lane; t < dq; t += 32) buf[oq + t] = a.adj_col[bq + t];
        }
        __syncwarp();
        int* sel = ssel[wib];
        const int ne = warp_unique_n(buf, count, sel, lane);  // the distinct elements
        __syncwarp();
        fits = ne <= kWarpCap / 8;
        count = fits ? 8 * ne : 0;
        for (int i = lane; i < count; i += 32) buf[i] = a.ltog[(size_t)sel[i >> 3] * 27 + (i & 7)];
      }
    }
    if (!fits) {
      if (pass == 0 && lane == 0) a.big[1 + atomicAdd(a.big, 1)] = r;
      continue;
    }
    __syncwarp();
    const int u = warp_unique_n(buf, count, pass == 1 ? a.col + a.rp[r] : nullptr, lane);
    if (pass == 0 && lane == 0) a.len[r] = u;
  }
}

// ---- one block per row, for the rows on the list ----
// mode 0: K rows (27 nodes of the elements around node r); 1: G rows (8
// corners); 2: element adjacency (elements around the 27 nodes of element r).
// pass 0 writes len[r]; pass 1 writes the columns at rp[r].
__global__ void __launch_bounds__(kPatThreads) k_rows(PatArgs a, int mode, int pass) {
  __shared__ int s[kPatCap];
  __shared__ int sflag[kPatCap];
  __shared__ int swarp[kPatThreads / 32];
  __shared__ int soff[28];
  const int nrows = a.big[0];
  for (int k = blockIdx.x; k < nrows; k += gridDim.x) {
    const int r = a.big[1 + k];
    int count;
    if (mode < 2) {
      const int nj = mode == 0 ? 27 : 8;
      const int t0 = a.inc_rp[r], deg = a.inc_rp[r + 1] - t0;
      count = deg * nj;
      if (count > kPatCap) {
        if (threadIdx.x == 0) {
          atomicExch(a.overflow, 1);
          if (pass == 0) a.len[r] = 0;
        }
        continue;
      }
      for (int i = threadIdx.x; i < count; i += blockDim.x) {
        const int e = a.inc_el[t0 + i / nj];
        s[i] = a.ltog[(size_t)e * 27 + i % nj];
      }
    } else {
      // offsets of the 27 incidence lists
      if (threadIdx.x == 0) {
        int o = 0;
        for (int j = 0; j < 27; j++) {
          soff[j] = o;
          const int v = a.ltog[(size_t)r * 27 + j];
          o += a.inc_rp[v + 1] - a.inc_rp[v];
        }
        soff[27] = o;
      }
      __syncthreads();
      count = soff[27];
      if (count > kPatCap) {
        if (threadIdx.x == 0) {
          atomicExch(a.overflow, 1);
          if (pass == 0) a.len[r] = 0;
        }
        __syncthreads();
        continue;
      }
      for (int i = threadIdx.x; i < count; i += blockDim.x) {
        int j = 0;
        while (soff[j + 1] <= i) j++;
        const int v = a.ltog[(size_t)r * 27 + j];
        s[i] = a.inc_el[a.inc_rp[v] + (i - soff[j])];
      }
    }
    const int n = pow2_at_least(count);
    for (int i = count + threadIdx.x; i < n; i += blockDim.x) s[i] = INT_MAX;
    __syncthreads();
    block_sort(s, n);
    const int u = block_unique(s, n, sflag, swarp, pass == 1 ? a.col + a.rp[r] : nullptr);
    if (pass == 0 && threadIdx.x == 0) a.len[r] = u;
  }
}

// Z rows p < NNp: the elements adjacent to the elements around p (sorted,
// distinct), then their corners (sorted, distinct).
__global__ void __launch_bounds__(kPatThreads) k_zrows(PatArgs a, int pass) {
  __shared__ int s[kPatCap];
  __shared__ int sflag[kPatCap];
  __shared__ int sel[kPatCap / 8];
  __shared__ int swarp[kPatThreads / 32];
  __shared__ int soff[65];
  __shared__ int sbad;
  const int nrows = a.big[0];
  for (int k = blockIdx.x; k < nrows; k += gridDim.x) {
    const int p = a.big[1 + k];
    const int t0 = a.inc_rp[p], deg = a.inc_rp[p + 1] - t0;
    if (threadIdx.x == 0) {
      sbad = deg > 64;
      int o = 0;
      for (int q = 0; q < deg && q < 64; q++) {
        soff[q] = o;
        const int e = a.inc_el[t0 + q];
        o += a.adj_rp[e + 1] - a.adj_rp[e];
      }
      soff[deg < 64 ? deg : 64] = o;
      if (o > kPatCap) sbad = 1;
    }
    __syncthreads();
    if (sbad) {
      if (threadIdx.x == 0) {
        atomicExch(a.overflow, 1);
        if (pass == 0) a.len[p] = 0;
      }
      __syncthreads();
      continue;
    }
    int count = soff[deg];
    for (int i = threadIdx.x; i < count; i += blockDim.x) {
      int q = 0;
      while (soff[q + 1] <= i) q++;
      const int e = a.inc_el[t0 + q];
      s[i] = a.adj_col[a.adj_rp[e] + (i - soff[q])];
    }
    int n = pow2_at_least(count);
    for (int i = count + threadIdx.x; i < n; i += blockDim.x) s[i] = INT_MAX;
    __syncthreads();
    block_sort(s, n);
    // the distinct elements (count first: the list must fit sel)
    const int ne = block_unique(s, n, sflag, swarp, nullptr);
    if (ne > kPatCap / 8) {
      if (threadIdx.x == 0) {
        atomicExch(a.overflow, 1);
        if (pass == 0) a.len[p] = 0;
      }
      __syncthreads();
      continue;
    }
    block_unique(s, n, sflag, swarp, sel);
    // their corners
    for (int i = threadIdx.x; i < ne; i += blockDim.x) {
      const int e = sel[i];
      for (int m = 0; m < 8; m++) s[8 * i + m] = a.ltog[(size_t)e * 27 + m];
    }
    count = ne * 8;
    n = pow2_at_least(count);
    for (int i = count + threadIdx.x; i < n; i += blockDim.x) s[i] = INT_MAX;
    __syncthreads();
    block_sort(s, n);
    const int u = block_unique(s, n, sflag, swarp, pass == 1 ? a.col + a.rp[p] : nullptr);
    if (pass == 0 && threadIdx.x == 0) a.len[p] = u;
  }
}

// gt_pos[t] = index in G's columns of (v, p) for the G^T entry t = (p, v).
__global__ void k_gt_pos(int nnp, const int* __restrict__ gt_rp, const int* __restrict__ gt_col,
                         const int* __restrict__ g_rp, const int* __restrict__ g_col, int* __restrict__ gt_pos,
                         int* __restrict__ bad) {
  for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < nnp; p += gridDim.x * blockDim.x)
    for (int t = gt_rp[p]; t < gt_rp[p + 1]; t++) {
      const int v = gt_col[t];
      int lo = g_rp[v], hi = g_rp[v + 1] - 1, at = -1;
      while (lo <= hi) {
        const int mid = (lo + hi) >> 1, c = g_col[mid];
        if (c == p) {
          at = mid;
          break;
        }
        if (c < p)
          lo = mid + 1;
        else
          hi = mid - 1;
      }
      if (at < 0) atomicExch(bad, 1);
      gt_pos[t] = at < 0 ? 0 : at;
    }
}

// first and last column of every row (rows sorted ascending; 0, -1 when empty)
__global__ void k_row_ends(int n, const int* __restrict__ rp, const int* __restrict__ col, int* __restrict__ first,
                           int* __restrict__ last) {
  for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < n; r += gridDim.x * blockDim.x) {
    const int b = rp[r], e = rp[r + 1];
    first[r] = b < e ? col[b] : 0;
    last[r] = b < e ? col[e - 1] : -1;
  }
}

int grid_for(long long n, int threads) {
  const long long g = (n + threads - 1) / threads;
  return (int)(g < 1 ? 1 : (g > 148 * 32 ? 148 * 32 : g));
}

}  // namespace

cudaError_t launch_incidence_count(long long nent, const int* ltog, int* cnt, cudaStream_t s) {
  k_inc_count<<<grid_for(nent, 256), 256, 0, s>>>(nent, ltog, cnt);
  return cudaGetLastError();
}
cudaError_t launch_incidence_fill(long long nent, const int* ltog, int* pos, int* inc_el, cudaStream_t s) {
  k_inc_fill<<<grid_for(nent, 256), 256, 0, s>>>(nent, ltog, pos, inc_el);
  return cudaGetLastError();
}
cudaError_t launch_pattern_rows(const PatArgs& a, int mode, int nrows, int pass, int num_sms, cudaStream_t s) {
  if (nrows <= 0) return cudaSuccess;
  if (pass == 0) {
    const cudaError_t e = cudaMemsetAsync(a.big, 0, sizeof(int), s);
    if (e != cudaSuccess) return e;
  }
  const int grid = (int)std::min<long long>((nrows + kWarpsPerBlock - 1LL) / kWarpsPerBlock, 8LL * num_sms);
  switch (mode) {
    case 0: k_rows_warp<0><<<grid, kPatThreads, 0, s>>>(a, nrows, pass); break;
    case 1: k_rows_warp<1><<<grid, kPatThreads, 0, s>>>(a, nrows, pass); break;
    case 2: k_rows_warp<2><<<grid, kPatThreads, 0, s>>>(a, nrows, pass); break;
    default: k_rows_warp<3><<<grid, kPatThreads, 0, s>>>(a, nrows, pass); break;
  }
  if (mode == 3)
    k_zrows<<<2 * num_sms, kPatThreads, 0, s>>>(a, pass);
  else
    k_rows<<<2 * num_sms, kPatThreads, 0, s>>>(a, mode, pass);
  return cudaGetLastError();
}
cudaError_t launch_gt_pos(int nnp, const int* gt_rp, const int* gt_col, const int* g_rp, const int* g_col, int* gt_pos,
                          int* bad, cudaStream_t s) {
  k_gt_pos<<<grid_for(nnp, 256), 256, 0, s>>>(nnp, gt_rp, gt_col, g_rp, g_col, gt_pos, bad);
  return cudaGetLastError();
}
cudaError_t launch_row_ends(int n, const int* rp, const int* col, int* first, int* last, cudaStream_t s) {
  k_row_ends<<<grid_for(n, 256), 256, 0, s>>>(n, rp, col, first, last);
  return cudaGetLastError();
}

}  // namespace cfd
