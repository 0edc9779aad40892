// Backward path: the point -> entry adjacency (CSR) and the first- and
// second-order adjoint kernels.
//
// Replaces csrc/backward.cu:5-121 (first order), csrc/backward.cu:124-328
// (second order, Eikonal) and their launchers csrc/backward.cu:331-455.  The
// reference scatters every point-side gradient with float atomicAdd; here
// each gradient is split into a query-side kernel (one query per half-warp,
// sums over its K neighbours) and a point-side kernel (one point per warp,
// sums over the sorted list of entries that selected it), so every sum has a
// fixed order and results are bit-reproducible.
//
// Notation for one entry e = (b, q, k) with point i = idxs[e]:
//   d = q - p_i, u_a = R_a . d, s = sum_a sigma_a u_a^2, w = exp(-s),
//   v = R^T diag(sigma) u  (so dw/dq = -2 w v),  c = gfo[q] . f[i].
// First order (gradient of <gfo, f_out>):
//   dq += -2 c w v,  dp += 2 c w v,  dsigma_a += -c w u_a^2,
//   dR_am += -2 c w sigma_a u_a d_m,  df[i] += w gfo[q].
// Second order (gradient of <g, dq> with g = grad_grad_q[q]):
//   A = g . v, r_a = R_a . g, Mg = sum_a sigma_a r_a R_a,
//   T = 2 c w (2 A v - Mg): dq += T, dp -= T,
//   dsigma_a += 2 c w u_a (u_a A - r_a),
//   dR_am += -2 c w sigma_a (-2 u_a d_m A + d_m r_a + u_a g_m),
//   df[i] += -2 w A gfo[q],  dgfo[q] += -2 w A f[i].
#include <math.h>

#include "knn_common.cuh"
#include "knn_internal.h"

namespace knnag {

// Rows up to which the fill scans the counts itself (64 KB of shared memory).
constexpr size_t kFillScanRows = 16384;

AdjLayout adj_layout(int B, int Q, int P, int K) {
  AdjLayout L{};
  const size_t n_rows = (size_t)B * P;
  const size_t n = (size_t)B * Q * K;
  size_t off = 0;
  L.rowptr = off;
  off += align256((n_rows + 1) * 4);
  L.cursor = off;
  off += align256(n_rows * 4);
  L.unsorted = off;
  off += align256(n * 4);
  L.entries = off;
  off += align256(n * 4);
  L.fill = off;
  if (n_rows <= kFillScanRows) off += align256(n_rows * 4);
  L.total = off;
  return L;
}

// ----------------------------------------------------------------- CSR

// Counts the entries of every row; also zeroes the fused fill's cursors
// (`rows` of them; none when cursor is null).
__global__ void adj_count_kernel(const int64_t* __restrict__ idxs, int n, int qk, int P, int* __restrict__ count,
                                 int* __restrict__ cursor, int rows) {
  if (cursor)
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < rows; r += gridDim.x * blockDim.x) cursor[r] = 0;
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < n; e += gridDim.x * blockDim.x) {
    const int64_t idx = idxs[e];
    if (idx < 0 || idx >= P) continue;  // not a point index: no row holds it
    atomicAdd(&count[(e / qk) * P + (int)idx], 1);
  }
}

// Exclusive scan of count[0..n) into rowptr[0..n] by one CTA of 1024
// threads (4 items per thread per pass); count is zeroed on the way so it
// can serve as the fill cursor.
__global__ void __launch_bounds__(1024) adj_scan_kernel(int* __restrict__ count, int64_t n, int* __restrict__ rowptr) {
  __shared__ int warp_sums[32];
  __shared__ int carry_s;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid == 0) carry_s = 0;
  __syncthreads();
  for (int64_t base = 0; base < n; base += 4096) {
    int v[4];
    int local = 0;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int64_t i = base + (int64_t)tid * 4 + u;
      v[u] = (i < n) ? count[i] : 0;
      if (i < n) count[i] = 0;
      local += v[u];
    }
    int incl = local;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += t;
    }
    if (lane == 31) warp_sums[warp] = incl;
    __syncthreads();
    if (warp == 0) {
      int ws = warp_sums[lane];
      int wi = ws;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, wi, o);
        if (lane >= o) wi += t;
      }
      warp_sums[lane] = wi - ws;  // exclusive prefix of warp totals
    }
    __syncthreads();
    int run = carry_s + warp_sums[warp] + incl - local;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int64_t i = base + (int64_t)tid * 4 + u;
      if (i < n) rowptr[i] = run;
      run += v[u];
    }
    __syncthreads();
    if (tid == 1023) carry_s = run;
    __syncthreads();
  }
  if (tid == 0) rowptr[n] = carry_s;
}

// Multi-CTA exclusive scan for long arrays, in three passes over chunks of
// kScanChunk elements (1024 threads x 8): (1) each CTA writes its chunk's
// sum to out[chunk start]; (2) one CTA replaces those sums by their
// exclusive prefix and writes the total to out[n]; (3) each CTA scans its
// chunk from that prefix into out and zeroes count.  The chunk sums live in
// out itself, so no scratch is needed.
constexpr int kScanChunk = 8192;

__device__ __forceinline__ int block_exclusive_scan_1024(int local, int* warp_sums, int& total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int incl = local;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int t = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += t;
  }
  if (lane == 31) warp_sums[warp] = incl;
  __syncthreads();
  if (warp == 0) {
    const int ws = warp_sums[lane];
    int wi = ws;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, wi, o);
      if (lane >= o) wi += t;
    }
    warp_sums[lane] = wi - ws;
    if (lane == 31) warp_sums[32] = wi;
  }
  __syncthreads();
  total = warp_sums[32];
  return warp_sums[warp] + incl - local;
}

// Eight consecutive ints from base (0 past n): two 128-bit loads where the
// address allows.
__device__ __forceinline__ void load8(const int* __restrict__ p, int64_t base, int64_t n, int (&v)[8]) {
  if (base + 8 <= n && (reinterpret_cast<uintptr_t>(p + base) & 15u) == 0) {
    const int4 a = *reinterpret_cast<const int4*>(p + base), b = *reinterpret_cast<const int4*>(p + base + 4);
    v[0] = a.x, v[1] = a.y, v[2] = a.z, v[3] = a.w;
    v[4] = b.x, v[5] = b.y, v[6] = b.z, v[7] = b.w;
  } else {
#pragma unroll
    for (int u = 0; u < 8; ++u) v[u] = base + u < n ? p[base + u] : 0;
  }
}
__device__ __forceinline__ void store8(int* __restrict__ p, int64_t base, int64_t n, const int (&v)[8]) {
  if (base + 8 <= n && (reinterpret_cast<uintptr_t>(p + base) & 15u) == 0) {
    *reinterpret_cast<int4*>(p + base) = make_int4(v[0], v[1], v[2], v[3]);
    *reinterpret_cast<int4*>(p + base + 4) = make_int4(v[4], v[5], v[6], v[7]);
  } else {
#pragma unroll
    for (int u = 0; u < 8; ++u)
      if (base + u < n) p[base + u] = v[u];
  }
}

__global__ void __launch_bounds__(1024) scan_chunk_sums_kernel(const int* __restrict__ count, int64_t n,
                                                               int* __restrict__ out) {
  __shared__ int warp_sums[33];
  const int64_t base = (int64_t)blockIdx.x * kScanChunk + (int64_t)threadIdx.x * 8;
  int v[8];
  load8(count, base, n, v);
  int local = 0;
#pragma unroll
  for (int u = 0; u < 8; ++u) local += v[u];
  int total;
  block_exclusive_scan_1024(local, warp_sums, total);
  if (threadIdx.x == 0) out[(int64_t)blockIdx.x * kScanChunk] = total;
}

__global__ void __launch_bounds__(1024) scan_chunk_prefix_kernel(int* __restrict__ out, int64_t n, int chunks) {
  __shared__ int warp_sums[33];
  __shared__ int carry_s;
  if (threadIdx.x == 0) carry_s = 0;
  __syncthreads();
  for (int c0 = 0; c0 < chunks; c0 += 1024) {
    const int c = c0 + threadIdx.x;
    const int v = c < chunks ? out[(int64_t)c * kScanChunk] : 0;
    int total;
    const int ex = block_exclusive_scan_1024(v, warp_sums, total);
    if (c < chunks) out[(int64_t)c * kScanChunk] = carry_s + ex;
    __syncthreads();
    if (threadIdx.x == 0) carry_s += total;
    __syncthreads();
  }
  if (threadIdx.x == 0) out[n] = carry_s;
}

__global__ void __launch_bounds__(1024) scan_chunk_apply_kernel(int* __restrict__ count, int64_t n,
                                                                int* __restrict__ out) {
  __shared__ int warp_sums[33];
  __shared__ int prefix_s;
  const int64_t chunk0 = (int64_t)blockIdx.x * kScanChunk;
  if (threadIdx.x == 0) prefix_s = out[chunk0];
  const int64_t base = chunk0 + (int64_t)threadIdx.x * 8;
  int v[8];
  load8(count, base, n, v);
  int local = 0;
#pragma unroll
  for (int u = 0; u < 8; ++u) local += v[u];
  int total;
  int run = block_exclusive_scan_1024(local, warp_sums, total) + prefix_s;  // barriers order the prefix read
  int zero[8];
#pragma unroll
  for (int u = 0; u < 8; ++u) {
    const int c = v[u];
    v[u] = run;
    run += c;
    zero[u] = 0;
  }
  store8(out, base, n, v);
  store8(count, base, n, zero);
}

__global__ void adj_fill_kernel(const int64_t* __restrict__ idxs, int n, int qk, int P, const int* __restrict__ rowptr,
                                int* __restrict__ cursor, int* __restrict__ unsorted) {
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < n; e += gridDim.x * blockDim.x) {
    const int64_t idx = idxs[e];
    if (idx < 0 || idx >= P) continue;
    const int row = (e / qk) * P + (int)idx;
    unsorted[rowptr[row] + atomicAdd(&cursor[row], 1)] = e;
  }
}

// The scan and the fill in one launch, for at most kFillScanRows rows: every
// CTA scans the counts into shared memory itself (read from L2) and fills its
// share; the first also writes rowptr.  `cursor` (zeroed beforehand) ranks a
// row's entries.  Two launches, the one-CTA scan first, took 18 us
// at 8192 rows and 393216 entries and 14 at 4096 rows and 196608; one takes 17
// and 10.  The sort sets the cursors back to
// zero, so that a graph's backward can run again on the same counts.
__global__ void __launch_bounds__(1024) adj_fill_scan_kernel(const int64_t* __restrict__ idxs, int n, int qk, int P,
                                                             const int* __restrict__ count, int rows,
                                                             int* __restrict__ cursor, int* __restrict__ rowptr,
                                                             int* __restrict__ unsorted) {
  extern __shared__ int start[];  // [rows]
  __shared__ int warp_sums[33];
  const int tid = threadIdx.x, per = (rows + 1023) / 1024;
  // coalesced in, then thread t takes rows [t per, (t + 1) per)
  for (int i = tid; i < rows; i += 1024) start[i] = count[i];
  __syncthreads();
  const int i0 = min(rows, tid * per), i1 = min(rows, i0 + per);
  int local = 0;
  for (int i = i0; i < i1; ++i) local += start[i];
  int total;
  int run = block_exclusive_scan_1024(local, warp_sums, total);
  for (int i = i0; i < i1; ++i) {
    const int c = start[i];
    start[i] = run;
    run += c;
  }
  __syncthreads();
  if (blockIdx.x == 0) {
    for (int i = tid; i < rows; i += 1024) rowptr[i] = start[i];
    if (tid == 0) rowptr[rows] = total;
  }
  constexpr int U = 4;  // entries in flight per thread
  for (int64_t e0 = blockIdx.x * 1024 + tid; e0 < n; e0 += (int64_t)gridDim.x * 1024 * U) {
    int row[U], rank[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int64_t e = e0 + (int64_t)u * gridDim.x * 1024;
      const int64_t idx = e < n ? idxs[e] : -1;
      row[u] = idx >= 0 && idx < P ? ((int)e / qk) * P + (int)idx : -1;
    }
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (row[u] >= 0) rank[u] = atomicAdd(&cursor[row[u]], 1);
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (row[u] >= 0) {
        const int end = row[u] + 1 < rows ? start[row[u] + 1] : total;
        if ((unsigned)rank[u] < (unsigned)(end - start[row[u]]))  // always: the row's count
          unsorted[start[row[u]] + rank[u]] = (int)(e0 + (int64_t)u * gridDim.x * 1024);
      }
  }
}

// Bitonic sort, ascending, of the 32*V ints of a warp: element lane + 32*h
// sits in x[h].  Stages with a partner distance below 32 exchange through
// shuffles, the others inside the lane.
template <int V>
__device__ __forceinline__ void warp_bitonic_sort(int (&x)[V], int lane) {
#pragma unroll
  for (int k = 2; k <= 32 * V; k <<= 1) {
#pragma unroll
    for (int j = k >> 1; j > 0; j >>= 1) {
      if (j >= 32) {
#pragma unroll
        for (int h = 0; h < V; ++h) {
          const int hp = h ^ (j >> 5);
          if (hp > h) {
            const bool up = ((32 * h) & k) == 0;  // lane < 32 <= j < k
            const int lo = min(x[h], x[hp]), hi = max(x[h], x[hp]);
            x[h] = up ? lo : hi;
            x[hp] = up ? hi : lo;
          }
        }
      } else {
#pragma unroll
        for (int h = 0; h < V; ++h) {
          const int e = lane + 32 * h;
          const int o = __shfl_xor_sync(0xffffffffu, x[h], j);
          const bool up = (e & k) == 0, lower = (e & j) == 0;
          x[h] = (lower == up) ? min(x[h], o) : max(x[h], o);
        }
      }
    }
  }
}

template <int V>
__device__ __forceinline__ void sort_row_regs(const int* src, int n, int* dst, int lane) {
  int x[V];
#pragma unroll
  for (int h = 0; h < V; ++h) x[h] = lane + 32 * h < n ? src[lane + 32 * h] : 0x7fffffff;
  warp_bitonic_sort<V>(x, lane);
#pragma unroll
  for (int h = 0; h < V; ++h)
    if (lane + 32 * h < n) dst[lane + 32 * h] = x[h];
}

constexpr int kAdjSortWarps = 8;      // warps per CTA of adj_sort_kernel
constexpr int kAdjLongRow = 256;      // rows beyond this are sorted by the whole CTA
constexpr int kAdjRun = 8192;         // in shared memory, runs of at most this many

// Ascending bitonic sort of n ints in shared memory by the CTA, padded to a
// power of two.
__device__ __forceinline__ void cta_bitonic_sort(int* sb, const int* src, int n) {
  int n2 = 512;
  while (n2 < n) n2 <<= 1;
  for (int i = threadIdx.x; i < n2; i += blockDim.x) sb[i] = i < n ? src[i] : 0x7fffffff;
  __syncthreads();
  for (int k = 2; k <= n2; k <<= 1)
    for (int j = k >> 1; j > 0; j >>= 1) {
      for (int t = threadIdx.x; t < n2 / 2; t += blockDim.x) {
        const int i = 2 * t - (t & (j - 1)), ixj = i + j;  // the t-th pair at distance j
        const int a = sb[i], b = sb[ixj];
        if ((a > b) == ((i & k) == 0)) {
          sb[i] = b;
          sb[ixj] = a;
        }
      }
      __syncthreads();
    }
}

// Sort every row by entry id (ids in a row are distinct: a query selects a
// point at most once).  Rows of up to 256 entries take one warp and its
// registers.  Longer ones (few points near many queries) take the whole CTA
// after its warps' rows: up to kAdjRun entries in shared memory, beyond that in
// sorted runs of kAdjRun, each id then placed at its rank, the sum of its ranks
// in all runs (written back over `unsorted`).  One warp per row whatever its
// length took 50 us where one has about 1000 entries (1000 rows in
// all; now 8 us), and time quadratic in the length beyond 1024.
__global__ void __launch_bounds__(kAdjSortWarps * 32) adj_sort_kernel(const int* __restrict__ rowptr, int* unsorted,
                                                                     int n_rows, int* __restrict__ entries,
                                                                     int* __restrict__ cursor) {
  __shared__ int sb[kAdjRun];
  __shared__ int more;
  const int lane = threadIdx.x & 31;
  const int gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int nw = (gridDim.x * blockDim.x) >> 5;
  if (threadIdx.x == 0) more = 0;
  __syncthreads();
  bool any = false;
  for (int r = gw; r < n_rows; r += nw) {
    const int start = rowptr[r];
    const int n = rowptr[r + 1] - start;
    const int* src = unsorted + start;
    int* dst = entries + start;
    if (cursor && lane == 0) cursor[r] = 0;
    if (n <= 32) {
      sort_row_regs<1>(src, n, dst, lane);
    } else if (n <= 64) {
      sort_row_regs<2>(src, n, dst, lane);
    } else if (n <= 128) {
      sort_row_regs<4>(src, n, dst, lane);
    } else if (n <= kAdjLongRow) {
      sort_row_regs<8>(src, n, dst, lane);
    } else {
      any = true;
    }
  }
  if (any && lane == 0) more = 1;
  __syncthreads();
  if (!more) return;
  // the CTA's long rows, in the same order (uniform control flow)
  for (int r0 = blockIdx.x * kAdjSortWarps; r0 < n_rows; r0 += nw)
    for (int r = r0; r < min(n_rows, r0 + kAdjSortWarps); ++r) {
      const int start = rowptr[r];
      const int n = rowptr[r + 1] - start;
      if (n <= kAdjLongRow) continue;
      int* src = unsorted + start;
      int* dst = entries + start;
      for (int run = 0; run < n; run += kAdjRun) {
        const int m = min(kAdjRun, n - run);
        cta_bitonic_sort(sb, src + run, m);
        int* out = n <= kAdjRun ? dst : src + run;
        for (int i = threadIdx.x; i < m; i += blockDim.x) out[i] = sb[i];
        __syncthreads();
      }
      if (n <= kAdjRun) continue;
      for (int i = threadIdx.x; i < n; i += blockDim.x) {
        const int x = src[i], own = i / kAdjRun;
        int rank = i - own * kAdjRun;
        for (int run = 0, t = 0; run < n; run += kAdjRun, ++t) {
          if (t == own) continue;
          int lo = 0, hi = min(kAdjRun, n - run);
          while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (src[run + mid] < x) lo = mid + 1;
            else hi = mid;
          }
          rank += lo;
        }
        dst[rank] = x;
      }
      __syncthreads();
    }
}

namespace {
int sm_count() {
  int dev = 0, v = 0;
  cudaGetDevice(&dev);
  if (cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || v <= 0) v = 148;
  return v;
}
inline unsigned blocks_for(int64_t n, int threads) {
  int64_t b = (n + threads - 1) / threads;
  const int64_t cap = (int64_t)sm_count() * 32;
  if (b > cap) b = cap;
  return (unsigned)(b < 1 ? 1 : b);
}
}  // namespace

// Exclusive scan of count[0..n) into out[0..n] (out[n] = total); count is
// zeroed so it can serve as a fill cursor.  One CTA for short arrays, the
// three-pass multi-CTA scan for long ones.
int launch_exclusive_scan(int* count, int n, int* out, cudaStream_t st) {
  if (n <= 4 * kScanChunk) {
    adj_scan_kernel<<<1, 1024, 0, st>>>(count, n, out);
    note_launches(1);
  } else {
    const int chunks = (int)(((int64_t)n + kScanChunk - 1) / kScanChunk);
    scan_chunk_sums_kernel<<<chunks, 1024, 0, st>>>(count, n, out);
    scan_chunk_prefix_kernel<<<1, 1024, 0, st>>>(out, n, chunks);
    scan_chunk_apply_kernel<<<chunks, 1024, 0, st>>>(count, n, out);
    note_launches(3);
  }
  return cudaGetLastError() == cudaSuccess ? KNNAG_OK : KNNAG_ERR_CUDA;
}

int launch_build_adjacency(const int64_t* idxs, int B, int Q, int P, int K, void* adjacency, cudaStream_t st,
                           bool counted) {
  NvtxRange range("knnag:adjacency");
  const AdjLayout L = adj_layout(B, Q, P, K);
  char* base = static_cast<char*>(adjacency);
  int* rowptr = reinterpret_cast<int*>(base + L.rowptr);
  int* cursor = reinterpret_cast<int*>(base + L.cursor);
  int* unsorted = reinterpret_cast<int*>(base + L.unsorted);
  int* entries = reinterpret_cast<int*>(base + L.entries);
  const int n = B * Q * K, rows = B * P, qk = Q * K;  // sizes checked < 2^31 by the caller
  const bool fused = (size_t)rows <= kFillScanRows;
  int* fill = fused ? reinterpret_cast<int*>(base + L.fill) : nullptr;
  if (!counted || n == 0) {  // else the forward counted the entries per row already (of no queries it counts nothing)
    if (cudaMemsetAsync(cursor, 0, (size_t)rows * 4, st) != cudaSuccess) return KNNAG_ERR_CUDA;
    adj_count_kernel<<<blocks_for(n, 256), 256, 0, st>>>(idxs, n, qk, P, cursor, fill, rows);
    note_launches(1);
  }
  if (fused) {
    const size_t smem = (size_t)rows * 4;
    if (smem > 47 * 1024 && cudaFuncSetAttribute(adj_fill_scan_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                 (int)(kFillScanRows * 4)) != cudaSuccess)
      return KNNAG_ERR_CUDA;
    int64_t blocks = ((int64_t)n + 2047) / 2048;  // two entries per thread or more: the scan is repeated by every CTA
    if (blocks > sm_count()) blocks = sm_count();
    if (blocks < 1) blocks = 1;
    adj_fill_scan_kernel<<<(unsigned)blocks, 1024, smem, st>>>(idxs, n, qk, P, cursor, rows,
                                                              fill, rowptr, unsorted);
    note_launches(1);
  } else {
    const int rc = launch_exclusive_scan(cursor, rows, rowptr, st);
    if (rc) return rc;
    adj_fill_kernel<<<blocks_for(n, 256), 256, 0, st>>>(idxs, n, qk, P, rowptr, cursor, unsorted);
    note_launches(1);
  }
  const int sort_threads = kAdjSortWarps * 32;
  adj_sort_kernel<<<blocks_for((int64_t)rows * 32, sort_threads), sort_threads, 0, st>>>(
      rowptr, unsorted, rows, entries, fill);
  note_launches(1);
  return cudaGetLastError() == cudaSuccess ? KNNAG_OK : KNNAG_ERR_CUDA;
}

// ------------------------------------------------------------ geometry

template <typename T>
struct Geo {
  T d[3], u[3], s, w;
};

// Offset, rotated offset, key and weight of query (qx,qy,qz) against a
// point record, with the forward's exact arithmetic (so w equals w_out).
template <typename T>
__device__ __forceinline__ void geometry(T qx, T qy, T qz, const T* rec, Geo<T>& g) {
  g.d[0] = add_rn(qx, rec[kNPX]);
  g.d[1] = add_rn(qy, rec[kNPY]);
  g.d[2] = add_rn(qz, rec[kNPZ]);
  const T* r = rec + kR00;
#pragma unroll
  for (int a = 0; a < 3; ++a) g.u[a] = row_dot(r[3 * a + 0], r[3 * a + 1], r[3 * a + 2], g.d[0], g.d[1], g.d[2]);
  g.s = quad_form(g.u[0], g.u[1], g.u[2], rec[kS0], rec[kS1], rec[kS2]);
  g.w = weight_of(g.s);
}

template <typename T>
struct QueryParams {
  const T* gfo;
  const T* ggq;
  const T* q;
  const T* rec;
  const T* f;
  const T* w_in;     // optional saved weights
  const int64_t* idxs;
  const T* coef_in;  // optional c = gfo . f (second order)
  int B, Q, P, F, K;
  T* dq;             // optional
  T* coef_out;       // optional (first order)
  T* dgfo;           // optional (second order)
  // ragged first order (FP32): sizes and offsets from the segment table,
  // records from the cloud set; gfo may be null (all ones).  Nothing is done
  // when *status is nonzero (a table that failed validation).
  const char* cs;
  const void* segs;
  const int* status;
  // broadcast grad_f_out: gfo points to one value s, and c = s * frowsum[i]
  // (frowsum = per-point sum over the columns of f)
  const T* frowsum;
  int* zero_status;  // optional (uniform calls): the backward's two status words, zeroed by the first CTA
};

template <typename T>
struct PointParams {
  const T* gfo;
  const T* ggq;
  const T* q;
  const T* rec;
  const T* w_in;
  const T* coef;
  const int* rowptr;
  const int* entries;
  int B, Q, P, F, K;
  int needs;
  T* dp;
  T* df;
  T* dsigma;
  T* dR;
  int* zero_status;  // as QueryParams
  bool gfo_scalar;  // gfo points to one value broadcast over [B,Q,F]
};

// The status words of a backward call: no kernel of it latches anything, so
// whichever runs first may clear them for a caller that reads them.
__device__ __forceinline__ void zero_status_words(int* status) {
  if (status && blockIdx.x == 0 && threadIdx.x < 2) status[threadIdx.x] = 0;
}

// v = R^T diag(sigma) u
template <typename T>
__device__ __forceinline__ void rot_back(const T* r, const T* sg, const T* u, T* v) {
#pragma unroll
  for (int m = 0; m < 3; ++m) v[m] = sg[0] * u[0] * r[m] + sg[1] * u[1] * r[3 + m] + sg[2] * u[2] * r[6 + m];
}

template <typename T>
__device__ __forceinline__ T warp_sum(T v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Per-point sum over the columns of f (one warp per row, fixed reduction
// order): with a broadcast grad_f_out s, c = gfo[q] . f[i] = s * rowsum[i].
// knnag_feature_row_sums exposes the same kernel, so row sums a caller
// keeps for resident features match the ones a backward call computes.
template <typename T>
__global__ void __launch_bounds__(256) row_sum_kernel(const T* __restrict__ f, int64_t rows, int F,
                                                      T* __restrict__ out) {
  const int lane = threadIdx.x & 31;
  const int64_t gw = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int64_t nw = (gridDim.x * (int64_t)blockDim.x) >> 5;
  for (int64_t r = gw; r < rows; r += nw) {
    T acc = T(0);
    for (int c = lane; c < F; c += 32) acc += f[r * F + c];
    acc = warp_sum(acc);
    if (lane == 0) out[r] = acc;
  }
}

// A query row's sizes, first entry, and its cloud's records, features and
// first point.
template <typename T>
struct QueryRow {
  int K, P;
  int64_t e0, pbase;
  const T* recb;
  const T* fb;
};
template <typename T>
__device__ __forceinline__ QueryRow<T> uniform_row(const QueryParams<T>& a, int64_t bq) {
  const int64_t b = bq / a.Q;
  return QueryRow<T>{a.K, a.P, bq * a.K, b * a.P, a.rec + b * a.P * kRecLen, a.f + b * a.P * a.F};
}
// Row bq of segment s of a ragged call.
template <typename T>
__device__ __forceinline__ QueryRow<T> segment_row(const QueryParams<T>& a, const SegDesc* sd, int s, int64_t bq) {
  const SegDesc g = sd[s];
  const CloudDesc c = cloud_descs(a.cs)[g.cloud];
  const T* rec = reinterpret_cast<const T*>(a.cs + reinterpret_cast<const CloudSetHeader*>(a.cs)->rec_off);
  return QueryRow<T>{g.K, c.P, g.e_off + (bq - g.q_off) * g.K, c.p_off, rec + c.p_off * kRecLen, a.f + c.p_off * a.F};
}

// Each lane's record `idx` (any valid one where the lane has none) of `recb`, for
// all lanes of a warp; the four lanes of a quad have the same recb.  FP32: the
// quad loads its four records together, 16 bytes a lane, so that a load
// instruction touches 8 lines instead of 32, and transposes.  At B = 1,
// Q = 524288, K = 16 the broadcast query side takes 153 us with it and 183
// without, the second order's launch 283 and 296.
__device__ __forceinline__ void load_rec_quad(const float* recb, int idx, float (&r)[kRecLen]) {
  const int t = threadIdx.x & 3;
  float4 d[4];
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    const int i = __shfl_sync(0xffffffffu, idx, u, 4);
    d[u] = __ldg(reinterpret_cast<const float4*>(recb + (int64_t)i * kRecLen) + t);
  }
  // d[u] holds part t of the quad's record u; exchanged to part u of record t
  auto swap = [](float4& x, float4& y, bool upper, int o) {  // y of the lower lane with x of the upper
    float4 v = upper ? x : y;
    v.x = __shfl_xor_sync(0xffffffffu, v.x, o);
    v.y = __shfl_xor_sync(0xffffffffu, v.y, o);
    v.z = __shfl_xor_sync(0xffffffffu, v.z, o);
    v.w = __shfl_xor_sync(0xffffffffu, v.w, o);
    if (upper) x = v;
    else y = v;
  };
  swap(d[0], d[1], t & 1, 1);
  swap(d[2], d[3], t & 1, 1);
  swap(d[0], d[2], t & 2, 2);
  swap(d[1], d[3], t & 2, 2);
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    r[4 * u + 0] = d[u].x;
    r[4 * u + 1] = d[u].y;
    r[4 * u + 2] = d[u].z;
    r[4 * u + 3] = d[u].w;
  }
}
__device__ __forceinline__ void load_rec_quad(const double* recb, int idx, double (&r)[kRecLen]) {
  load_rec(recb + (int64_t)idx * kRecLen, r);
}

// One neighbour's share of dq: -2 c w v.
template <typename T>
__device__ __forceinline__ void add_dq(const QueryParams<T>& a, const T (&rec)[kRecLen], T qx, T qy, T qz, int64_t e,
                                       T c, T (&acc)[3]) {
  Geo<T> geo;
  geometry(qx, qy, qz, rec, geo);
  const T w = a.w_in ? a.w_in[e] : geo.w;
  const T sg[3] = {rec[kS0], rec[kS1], rec[kS2]};
  T v[3];
  rot_back(rec + kR00, sg, geo.u, v);
  const T t = T(-2) * c * w;
#pragma unroll
  for (int m = 0; m < 3; ++m) acc[m] += t * v[m];
}

// First-order query side with a broadcast grad_f_out s: c_k = s *
// rowsum(f)[idx_k] needs no F-wide dot product, so each lane takes one
// neighbour, and a warp serves two queries when K <= 16.  A warp of a ragged
// call takes up to kRowBlock consecutive rows, so that the segment is looked up once
// for them and not by a chain of dependent loads per row; one row where there are
// no more than the warps that run at a time, which otherwise idle (50 rows, K =
// 40: 7 us, eight to a warp 23).
constexpr int kRowBlock = 8;
constexpr int kBroadcastWarps = 148 * 4 * 8;  // that run at a time

// Bound by the latency of a neighbour's index and record: a kernel of its own, at
// four CTAs per SM (5: 218 us where 4 take 153 at the sizes above, 6: 242; as a
// branch of query_order1_kernel at three: 207), table workload 13.0 -> 10.4 us,
// 24 ragged clouds 149 -> 129.
template <typename T>
__global__ void __launch_bounds__(256, sizeof(T) == 4 ? 4 : 2) query_order1_broadcast_kernel(QueryParams<T> a) {
  const SegHeader* sh = static_cast<const SegHeader*>(a.segs);
  if (sh && *a.status) return;
  zero_status_words(a.zero_status);
  const int64_t BQ = sh ? sh->grad_rows : (int64_t)a.B * a.Q;
  const int lane = threadIdx.x & 31;
  const int lpq = (!sh && a.K <= 16) ? 16 : 32;  // lanes per query
  const int qpw = 32 / lpq, sub = lane / lpq, kl = lane % lpq;
  const int64_t gw = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int64_t nw = (gridDim.x * (int64_t)blockDim.x) >> 5;
  const T sg0 = a.gfo ? a.gfo[0] : T(1);  // ragged calls: no grad_f_out means all ones
  const SegDesc* sd = sh ? seg_descs(a.segs) : nullptr;
  // of a warp's turn
  const int rows = sh ? (int)min((BQ + kBroadcastWarps - 1) / kBroadcastWarps, (int64_t)kRowBlock) : qpw;
  for (int64_t turn = gw * rows; turn < BQ; turn += nw * rows) {
    int s = sh ? seg_of_row(sd, sh->nseg, turn) : 0;
    for (int64_t base = turn; base < BQ && base < turn + rows; base += qpw) {
      const int64_t bq = base + sub;
      T acc[3] = {T(0), T(0), T(0)};
      if (sh)
        while (s + 1 < sh->nseg && sd[s + 1].q_off <= bq) ++s;
      const bool live = bq < BQ;
      const QueryRow<T> r = sh ? segment_row(a, sd, s, bq) : uniform_row(a, live ? bq : base);
      const T* qp = a.q + (live ? bq : base) * 3;
      const T qx = qp[0], qy = qp[1], qz = qp[2];
      for (int k0 = 0; k0 < r.K; k0 += lpq) {  // K is the same for the warp's queries
        const int k = k0 + kl;
        const int64_t e = r.e0 + k;
        const int64_t idx = live && k < r.K ? a.idxs[e] : -1;
        const bool ok = idx >= 0 && idx < r.P;
        T rec[kRecLen];
        if (!sh) load_rec_quad(r.recb, ok ? (int)idx : 0, rec);
        else if (ok) load_rec(r.recb + idx * kRecLen, rec);  // small K: idle lanes would load for nothing
        T c = T(0);
        if (ok) {
          c = sg0 * a.frowsum[r.pbase + idx];
          add_dq(a, rec, qx, qy, qz, e, c, acc);
        }
        if (a.coef_out && live && k < r.K) a.coef_out[e] = c;
      }
#pragma unroll
      for (int mm = 0; mm < 3; ++mm)
        for (int o = lpq >> 1; o >= 1; o >>= 1) acc[mm] += __shfl_xor_sync(0xffffffffu, acc[mm], o);
      if (bq < BQ && kl == 0 && a.dq) {
        a.dq[bq * 3 + 0] = acc[0];
        a.dq[bq * 3 + 1] = acc[1];
        a.dq[bq * 3 + 2] = acc[2];
      }
    }
  }
}

// 16-byte column groups of f and grad_f_out rows (C values), or single values.
template <typename T, bool VEC>
struct ColGroup {
  using type = typename Group16<T>::type;
  static constexpr int C = 16 / sizeof(T);
};
template <typename T>
struct ColGroup<T, false> {
  using type = T;
  static constexpr int C = 1;
};
__device__ __forceinline__ float dot_group(const float4& a, const float4& b, float s) {
  return __fmaf_rn(a.w, b.w, __fmaf_rn(a.z, b.z, __fmaf_rn(a.y, b.y, __fmaf_rn(a.x, b.x, s))));
}
__device__ __forceinline__ double dot_group(const double2& a, const double2& b, double s) {
  return __fma_rn(a.y, b.y, __fma_rn(a.x, b.x, s));
}
template <typename T>
__device__ __forceinline__ T dot_group(T a, T b, T s) {
  return fma_rn(a, b, s);
}
__device__ __forceinline__ void fill_group(float4& g, float v) { g = make_float4(v, v, v, v); }
__device__ __forceinline__ void fill_group(double2& g, double v) { g = make_double2(v, v); }
template <typename T>
__device__ __forceinline__ void fill_group(T& g, T v) {
  g = v;
}
template <typename T>
__device__ __forceinline__ void fma_group(T v, T w, T (&acc)[1]) {
  acc[0] = fma_rn(v, w, acc[0]);
}
template <typename V, typename T, int C>
__device__ __forceinline__ V to_group(const T (&a)[C]) {
  if constexpr (C == 1) return a[0];
  else return group_of(a);
}

// First-order query side: G lanes per query (16 for up to 64 column groups'
// worth of a half-warp, else 32), so a warp serves one or two.  For each 16
// neighbours the lanes sweep the feature columns, 16 bytes each where the rows
// allow, four rows in flight (eight of single columns); a reduce-scatter then leaves c_k = gfo[q] .
// f[idx_k] of neighbour k0 + l in lane l, which does that neighbour's geometry.
// dq = sum_k -2 c_k w_k v_k.
//
// Bound by the gathered feature rows (L2): one query per warp with 4-byte loads
// took 37 us at B = 2, Q = 12288, K = 16, F = 64 and now takes 20 (26 with eight
// rows in flight, which spills at three CTAs per SM).
template <typename T, int G, bool VEC>
__global__ void __launch_bounds__(256, sizeof(T) == 4 ? 3 : 2) query_order1_kernel(QueryParams<T> a) {
  using V = typename ColGroup<T, VEC>::type;
  constexpr int C = ColGroup<T, VEC>::C, NK = 16, RB = VEC ? 4 : 8;  // neighbours a turn, rows in flight
  const int lane = threadIdx.x & 31, gl = lane % G;
  const SegHeader* sh = static_cast<const SegHeader*>(a.segs);
  if (sh && *a.status) return;
  zero_status_words(a.zero_status);
  const int64_t BQ = sh ? sh->grad_rows : (int64_t)a.B * a.Q;
  constexpr int N = 32 / G;  // queries of the warp
  const int cols = a.F / C;
  const int64_t gw = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int64_t nw = (gridDim.x * (int64_t)blockDim.x) >> 5;
  for (int64_t base = gw * N; base < BQ; base += nw * N) {
    const bool live = base + lane / G < BQ;
    const int64_t bq = live ? base + lane / G : BQ - 1;
    const SegDesc* sd = sh ? seg_descs(a.segs) : nullptr;
    const QueryRow<T> r = sh ? segment_row(a, sd, seg_of_row(sd, sh->nseg, bq), bq) : uniform_row(a, bq);
    const T qx = a.q[bq * 3 + 0], qy = a.q[bq * 3 + 1], qz = a.q[bq * 3 + 2];
    const V* grow = a.gfo ? reinterpret_cast<const V*>(a.gfo + bq * a.F) : nullptr;
    const V* frow = reinterpret_cast<const V*>(r.fb);
    T acc[3] = {T(0), T(0), T(0)};
    // the two queries of a warp may differ in K (segments): both take every turn
    int most = r.K;
    if (N > 1) most = max(most, __shfl_xor_sync(0xffffffffu, most, 16));
    for (int k0 = 0; k0 < most; k0 += NK) {
      const int km = k0 + (gl & (NK - 1));  // this lane's neighbour
      const int64_t idx = km < r.K ? a.idxs[r.e0 + km] : -1;
      const int mine = (idx >= 0 && idx < r.P) ? (int)idx : -1;
      T part[NK];
#pragma unroll
      for (int kk = 0; kk < NK; ++kk) part[kk] = T(0);
      for (int cb = 0; cb < cols; cb += G) {  // warp-uniform: the shuffles need every lane
        const int c = cb + gl;
        const bool col = c < cols;
        V g{};
        if (col) {
          if (grow) g = grow[c];
          else fill_group(g, T(1));
        }
#pragma unroll
        for (int kb = 0; kb < NK; kb += RB) {
          if (k0 + kb < most) {
            V v[RB];
            int ik[RB];
#pragma unroll
            for (int u = 0; u < RB; ++u) {
              ik[u] = __shfl_sync(0xffffffffu, mine, kb + u, G);
              if (col && ik[u] >= 0) v[u] = __ldg(frow + (int64_t)ik[u] * cols + c);
            }
#pragma unroll
            for (int u = 0; u < RB; ++u)
              if (col && ik[u] >= 0) part[kb + u] = dot_group(g, v[u], part[kb + u]);
          }
        }
      }
      // reduce-scatter: 16 values over 16 lanes -> lane l holds value l
#pragma unroll
      for (int h = NK / 2; h >= 1; h >>= 1) {
        const bool upper = (lane & h) != 0;
#pragma unroll
        for (int i = 0; i < h; ++i) {
          const T send = upper ? part[i] : part[i + h];
          const T keep = upper ? part[i + h] : part[i];
          part[i] = keep + __shfl_xor_sync(0xffffffffu, send, h);
        }
      }
      if (G == 32) part[0] += __shfl_xor_sync(0xffffffffu, part[0], 16);
      if (live && gl < NK && km < r.K) {
        const int64_t e = r.e0 + km;
        if (a.coef_out) a.coef_out[e] = part[0];
        if (mine >= 0) {
          T rec[kRecLen];
          load_rec(r.recb + (int64_t)mine * kRecLen, rec);
          add_dq(a, rec, qx, qy, qz, e, part[0], acc);
        }
      }
    }
#pragma unroll
    for (int mm = 0; mm < 3; ++mm)
#pragma unroll
      for (int o = G / 2; o >= 1; o >>= 1) acc[mm] += __shfl_xor_sync(0xffffffffu, acc[mm], o);
    if (live && gl == 0 && a.dq) {
      a.dq[bq * 3 + 0] = acc[0];
      a.dq[bq * 3 + 1] = acc[1];
      a.dq[bq * 3 + 2] = acc[2];
    }
  }
}

// Second-order query side: one warp per query, lane = neighbour.  With
// g = grad_grad_q[q], A = g . v, r_a = R_a . g, Mg = sum_a sigma_a r_a R_a:
// dq += 2 c w (2 A v - Mg); optionally dgfo[q] = sum_k (-2 w_k A_k) f[idx_k]
// accumulated in k order, lanes spanning columns, 8 rows in flight.
// Second order without dgfo and with K <= 16 (the Eikonal step): half a
// warp per query, one neighbour per lane, so a warp serves two queries.
template <typename T>
__device__ __forceinline__ void query_order2_half(const QueryParams<T>& a, int64_t blk, int64_t nblk) {
  const int lane = threadIdx.x & 31;
  const int sub = lane >> 4, k = lane & 15;
  const int64_t BQ = (int64_t)a.B * a.Q;
  const int K = a.K, P = a.P;
  const int64_t gw = (blk * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int64_t nw = (nblk * (int64_t)blockDim.x) >> 5;
  for (int64_t base = gw * 2; base < BQ; base += nw * 2) {
    const int64_t bq = base + sub;
    T acc[3] = {T(0), T(0), T(0)};
    if (a.coef_in) {  // uniform
      const int64_t row = bq < BQ ? bq : base;
      const int64_t b = row / a.Q;
      const int64_t e = bq * K + k;
      const int64_t idx = bq < BQ && k < K ? a.idxs[e] : -1;
      const bool ok = idx >= 0 && idx < P;
      T rr[kRecLen];
      load_rec_quad(a.rec + b * P * kRecLen, ok ? (int)idx : 0, rr);
      if (ok) {
        const T qx = a.q[bq * 3 + 0], qy = a.q[bq * 3 + 1], qz = a.q[bq * 3 + 2];
        const T g[3] = {a.ggq[bq * 3 + 0], a.ggq[bq * 3 + 1], a.ggq[bq * 3 + 2]};
        const T* rec = rr;
        Geo<T> geo;
        geometry(qx, qy, qz, rec, geo);
        const T w = a.w_in ? a.w_in[e] : geo.w;
        const T* r = rec + kR00;
        const T sg[3] = {rec[kS0], rec[kS1], rec[kS2]};
        T v[3];
        rot_back(r, sg, geo.u, v);
        const T A = g[0] * v[0] + g[1] * v[1] + g[2] * v[2];
        T rg[3];
#pragma unroll
        for (int s2 = 0; s2 < 3; ++s2) rg[s2] = r[3 * s2] * g[0] + r[3 * s2 + 1] * g[1] + r[3 * s2 + 2] * g[2];
        const T cw2 = T(2) * a.coef_in[e] * w;
#pragma unroll
        for (int m = 0; m < 3; ++m) {
          const T mg = sg[0] * rg[0] * r[m] + sg[1] * rg[1] * r[3 + m] + sg[2] * rg[2] * r[6 + m];
          acc[m] += cw2 * (T(2) * A * v[m] - mg);
        }
      }
    }
#pragma unroll
    for (int m = 0; m < 3; ++m)
#pragma unroll
      for (int o = 8; o >= 1; o >>= 1) acc[m] += __shfl_xor_sync(0xffffffffu, acc[m], o);
    if (bq < BQ && k == 0 && a.dq) {
      a.dq[bq * 3 + 0] = acc[0];
      a.dq[bq * 3 + 1] = acc[1];
      a.dq[bq * 3 + 2] = acc[2];
    }
  }
}

template <typename T>
__device__ __forceinline__ void query_order2_body(const QueryParams<T>& a, int blk, int nblk) {
  if (!a.dgfo && a.K <= 16) {
    query_order2_half(a, blk, nblk);
    return;
  }
  const int lane = threadIdx.x & 31;
  const int BQ = a.B * a.Q, K = a.K, F = a.F, P = a.P;
  const int gw = (blk * blockDim.x + threadIdx.x) >> 5;
  const int nw = (nblk * blockDim.x) >> 5;
  for (int bq = gw; bq < BQ; bq += nw) {
    const int b = bq / a.Q;
    const T qx = a.q[(int64_t)bq * 3 + 0], qy = a.q[(int64_t)bq * 3 + 1], qz = a.q[(int64_t)bq * 3 + 2];
    const T g[3] = {a.ggq[(int64_t)bq * 3 + 0], a.ggq[(int64_t)bq * 3 + 1], a.ggq[(int64_t)bq * 3 + 2]};
    const T* fb = a.f + (int64_t)b * P * F;
    T acc[3] = {T(0), T(0), T(0)};
    for (int k0 = 0; k0 < K; k0 += 32) {
      const int k = k0 + lane;
      const int64_t e = (int64_t)bq * K + k;
      T a_own = T(0);
      int64_t row = -1;
      if (k < K) {
        const int64_t idx = a.idxs[e];
        if (idx >= 0 && idx < P) {
          row = idx * F;
          T rr[kRecLen];
          load_rec(a.rec + ((int64_t)b * P + idx) * kRecLen, rr);
          const T* rec = rr;
          Geo<T> geo;
          geometry(qx, qy, qz, rec, geo);
          const T w = a.w_in ? a.w_in[e] : geo.w;
          const T* r = rec + kR00;
          const T sg[3] = {rec[kS0], rec[kS1], rec[kS2]};
          T v[3];
          rot_back(r, sg, geo.u, v);
          const T A = g[0] * v[0] + g[1] * v[1] + g[2] * v[2];
          a_own = T(-2) * w * A;
          if (a.coef_in) {
            T rg[3];
#pragma unroll
            for (int s2 = 0; s2 < 3; ++s2) rg[s2] = r[3 * s2] * g[0] + r[3 * s2 + 1] * g[1] + r[3 * s2 + 2] * g[2];
            const T cw2 = T(2) * a.coef_in[e] * w;
#pragma unroll
            for (int m = 0; m < 3; ++m) {
              const T mg = sg[0] * rg[0] * r[m] + sg[1] * rg[1] * r[3 + m] + sg[2] * rg[2] * r[6 + m];
              acc[m] += cw2 * (T(2) * A * v[m] - mg);
            }
          }
        }
      }
      if (a.dgfo) {
        const int nk = min(32, K - k0);
        T* drow = a.dgfo + (int64_t)bq * F;
        for (int cb = 0; cb < F; cb += 32) {  // warp-uniform: the shuffles below need every lane
          const int c = cb + lane;
          const bool col = c < F;
          T s = (k0 == 0 || !col) ? T(0) : drow[c];
          for (int j0 = 0; j0 < nk; j0 += 8) {
            T val[8], ak[8];
#pragma unroll
            for (int jj = 0; jj < 8; ++jj) {
              const int src = min(j0 + jj, 31);
              const int64_t rj = __shfl_sync(0xffffffffu, row, src);
              ak[jj] = __shfl_sync(0xffffffffu, a_own, src);
              val[jj] = (col && j0 + jj < nk && rj >= 0) ? fb[rj + c] : T(0);
            }
#pragma unroll
            for (int jj = 0; jj < 8; ++jj)
              if (j0 + jj < nk) s = fma_rn(ak[jj], val[jj], s);
          }
          if (col) drow[c] = s;
        }
      }
    }
    if (a.dq) {
#pragma unroll
      for (int m = 0; m < 3; ++m) acc[m] = warp_sum(acc[m]);
      if (lane == 0) {
        a.dq[(int64_t)bq * 3 + 0] = acc[0];
        a.dq[(int64_t)bq * 3 + 1] = acc[1];
        a.dq[(int64_t)bq * 3 + 2] = acc[2];
      }
    }
  }
}

template <typename T>
__global__ void __launch_bounds__(256) query_order2_kernel(QueryParams<T> a) {
  zero_status_words(a.zero_status);
  query_order2_body(a, blockIdx.x, gridDim.x);
}

// One entry of a point row: the query's offset, rotated offset, weight and
// v = R^T diag(sigma) u, and for the second order its grad_grad_q.
template <typename T, int ORDER>
struct PointEntry {
  Geo<T> geo;
  T v[3], g[3], w;
};
template <typename T, int ORDER>
__device__ __forceinline__ void point_entry(const PointParams<T>& a, const T (&pr)[kRecLen], int e, int64_t bq,
                                            PointEntry<T, ORDER>& x) {
  const T qx = a.q[bq * 3 + 0], qy = a.q[bq * 3 + 1], qz = a.q[bq * 3 + 2];
  if (ORDER == 2)
#pragma unroll
    for (int m = 0; m < 3; ++m) x.g[m] = a.ggq[bq * 3 + m];
  const T sg[3] = {pr[kS0], pr[kS1], pr[kS2]};
  geometry(qx, qy, qz, pr, x.geo);
  x.w = a.w_in ? a.w_in[e] : x.geo.w;
  rot_back(pr + kR00, sg, x.geo.u, x.v);
}

// Point side, geometry: one warp per point row, lane j takes entry j of each
// 32-entry chunk of the row and sums the 15 point-side scalars, reduced over
// the warp at the end.  With a broadcast grad_f_out s this is the whole point
// side: c = s * rowsum(f)[row] in every entry of the row, and df[i][c] = s *
// sum_e wgt_e for every column.  The entry order of a row is fixed (sorted), so
// every sum has a fixed order.
template <typename T, int ORDER>
__device__ __forceinline__ void point_geometry_body(const PointParams<T>& a, int blk, int nblk) {
  const int lane = threadIdx.x & 31;
  const int gw = (blk * blockDim.x + threadIdx.x) >> 5;
  const int nw = (nblk * blockDim.x) >> 5;
  const int rows = a.B * a.P;
  const int F = a.F, K = a.K;
  const int n_entries = a.B * a.Q * K;
  const bool want_geo = (a.needs & (KNNAG_NEED_DP | KNNAG_NEED_DSIGMA | KNNAG_NEED_DR)) != 0;
  const bool scalar_df = (a.needs & KNNAG_NEED_DF) != 0 && a.gfo_scalar;
  for (int row = gw; row < rows; row += nw) {
    T pr[kRecLen];
    load_rec(a.rec + (int64_t)row * kRecLen, pr);
    const T* r = pr + kR00;
    const T sg[3] = {pr[kS0], pr[kS1], pr[kS2]};
    const int start = a.rowptr[row], end = a.rowptr[row + 1];
    T gp[3] = {T(0), T(0), T(0)}, gs[3] = {T(0), T(0), T(0)}, gR[9], wsum = T(0), c_row = T(0);
#pragma unroll
    for (int m = 0; m < 9; ++m) gR[m] = T(0);
    if (a.gfo_scalar && want_geo && start < end) {
      const int e = a.entries[start];
      if (e >= 0 && e < n_entries) c_row = a.coef[e];
    }
    for (int j = start + lane; j < end; j += 32) {
      const int e = a.entries[j];
      if (e < 0 || e >= n_entries) continue;
      PointEntry<T, ORDER> x;
      point_entry<T, ORDER>(a, pr, e, e / K, x);
      const T c = !want_geo ? T(0) : (a.gfo_scalar ? c_row : a.coef[e]);
      const T cw = c * x.w;
      if (ORDER == 1) {
        wsum += x.w;
#pragma unroll
        for (int m = 0; m < 3; ++m) gp[m] += T(2) * cw * x.v[m];
#pragma unroll
        for (int s2 = 0; s2 < 3; ++s2) {
          gs[s2] -= cw * x.geo.u[s2] * x.geo.u[s2];
          const T t = T(-2) * cw * sg[s2] * x.geo.u[s2];
#pragma unroll
          for (int m = 0; m < 3; ++m) gR[3 * s2 + m] += t * x.geo.d[m];
        }
      } else {
        const T A = x.g[0] * x.v[0] + x.g[1] * x.v[1] + x.g[2] * x.v[2];
        wsum += T(-2) * x.w * A;
        T rg[3];
#pragma unroll
        for (int s2 = 0; s2 < 3; ++s2) rg[s2] = r[3 * s2] * x.g[0] + r[3 * s2 + 1] * x.g[1] + r[3 * s2 + 2] * x.g[2];
#pragma unroll
        for (int m = 0; m < 3; ++m) {
          const T mg = sg[0] * rg[0] * r[m] + sg[1] * rg[1] * r[3 + m] + sg[2] * rg[2] * r[6 + m];
          gp[m] -= T(2) * cw * (T(2) * A * x.v[m] - mg);
        }
#pragma unroll
        for (int s2 = 0; s2 < 3; ++s2) {
          gs[s2] += T(2) * cw * x.geo.u[s2] * (x.geo.u[s2] * A - rg[s2]);
          const T t = T(-2) * cw * sg[s2];
#pragma unroll
          for (int m = 0; m < 3; ++m)
            gR[3 * s2 + m] += t * (T(-2) * x.geo.u[s2] * x.geo.d[m] * A + x.geo.d[m] * rg[s2] + x.geo.u[s2] * x.g[m]);
        }
      }
    }
    if (scalar_df) {
      const T val = a.gfo[0] * warp_sum(wsum);
      for (int cc = lane; cc < F; cc += 32) a.df[(int64_t)row * F + cc] = val;
    }
    if (want_geo) {
      T vals[15];
#pragma unroll
      for (int m = 0; m < 3; ++m) {
        vals[m] = gp[m];
        vals[3 + m] = gs[m];
      }
#pragma unroll
      for (int m = 0; m < 9; ++m) vals[6 + m] = gR[m];
#pragma unroll
      for (int m = 0; m < 15; ++m) vals[m] = warp_sum(vals[m]);
      if (lane == 0) {
        if (a.needs & KNNAG_NEED_DP)
          for (int m = 0; m < 3; ++m) a.dp[(int64_t)row * 3 + m] = vals[m];
        if (a.needs & KNNAG_NEED_DSIGMA)
          for (int m = 0; m < 3; ++m) a.dsigma[(int64_t)row * 3 + m] = vals[3 + m];
        if (a.needs & KNNAG_NEED_DR)
          for (int m = 0; m < 9; ++m) a.dR[(int64_t)row * 9 + m] = vals[6 + m];
      }
    }
  }
}

// Point side, features: df[row] = sum_e wgt_e gfo[query of e], one warp per
// point row.  Lane j computes entry j's weight of each 32-entry chunk; the warp
// then walks the chunk with lanes spanning feature columns: G lanes per entry
// (two entries side by side where 16 lanes hold the columns), 16 bytes each
// where the rows allow, NV groups per lane, four entries in flight per half.
template <typename T, int ORDER, int G, int NV, bool VEC>
__device__ __forceinline__ void point_features_body(const PointParams<T>& a, int blk, int nblk) {
  using V = typename ColGroup<T, VEC>::type;
  constexpr int C = ColGroup<T, VEC>::C, H = 32 / G, RB = 4;
  const int lane = threadIdx.x & 31, gl = lane % G, half = lane / G;
  const int gw = (blk * blockDim.x + threadIdx.x) >> 5;
  const int nw = (nblk * blockDim.x) >> 5;
  const int rows = a.B * a.P;
  const int F = a.F, K = a.K, cols = F / C;
  const int n_entries = a.B * a.Q * K;
  for (int row = gw; row < rows; row += nw) {
    T pr[kRecLen];
    load_rec(a.rec + (int64_t)row * kRecLen, pr);
    const int start = a.rowptr[row], end = a.rowptr[row + 1];
    for (int c0 = 0; c0 < cols; c0 += G * NV) {
      T acc[NV][C];
#pragma unroll
      for (int u = 0; u < NV; ++u)
#pragma unroll
        for (int v = 0; v < C; ++v) acc[u][v] = T(0);
      for (int base = start; base < end; base += 32) {
        int bq = 0;
        T wgt = T(0);
        if (base + lane < end) {
          const int e = a.entries[base + lane];
          if (e >= 0 && e < n_entries) {
            bq = e / K;
            PointEntry<T, ORDER> x;
            point_entry<T, ORDER>(a, pr, e, bq, x);
            wgt = ORDER == 1 ? x.w : T(-2) * x.w * (x.g[0] * x.v[0] + x.g[1] * x.v[1] + x.g[2] * x.v[2]);
          }
        }
        const int nvalid = min(32, end - base);
        for (int j0 = 0; j0 < nvalid; j0 += RB * H) {
          V val[RB][NV];
          T wj[RB];
#pragma unroll
          for (int jj = 0; jj < RB; ++jj) {
            const int src = j0 + jj * H + half;  // at most 31: 32 is a multiple of RB * H
            const int bqj = __shfl_sync(0xffffffffu, bq, src);
            wj[jj] = __shfl_sync(0xffffffffu, wgt, src);
            const V* grow = reinterpret_cast<const V*>(a.gfo + (int64_t)bqj * F);
#pragma unroll
            for (int u = 0; u < NV; ++u) {
              const int cc = c0 + gl + G * u;
              if (src < nvalid && cc < cols) val[jj][u] = __ldg(grow + cc);
            }
          }
#pragma unroll
          for (int jj = 0; jj < RB; ++jj)
#pragma unroll
            for (int u = 0; u < NV; ++u)
              if (j0 + jj * H + half < nvalid && c0 + gl + G * u < cols) fma_group(val[jj][u], wj[jj], acc[u]);
        }
      }
#pragma unroll
      for (int u = 0; u < NV; ++u) {
        if (H == 2)
#pragma unroll
          for (int v = 0; v < C; ++v) acc[u][v] += __shfl_xor_sync(0xffffffffu, acc[u][v], 16);
        const int cc = c0 + gl + G * u;
        if (half == 0 && cc < cols) reinterpret_cast<V*>(a.df + (int64_t)row * F)[cc] = to_group<V>(acc[u]);
      }
    }
  }
}

// The point side in one launch over two ranges of blocks: the first f_blocks
// walk the feature rows, the rest sum the geometry.  A row's features are a
// chain of dependent gathers (entries, queries, grad_f_out rows) and the
// geometry needs many registers; apart, twice as many warps are in flight, each
// with more rows of its own.  At B = 2, Q = 12288, P = 4096, K = 16, F = 64: 33
// us with one warp doing both, 28 apart (31 with eight entries in flight per
// half at four CTAs per SM, which spills).
template <typename T, int ORDER, int G, int NV, bool VEC>
__global__ void __launch_bounds__(256, sizeof(T) == 4 ? 3 : 2) point_side_kernel(PointParams<T> a, int f_blocks) {
  zero_status_words(a.zero_status);
  if ((int)blockIdx.x < f_blocks)
    point_features_body<T, ORDER, G, NV, VEC>(a, blockIdx.x, f_blocks);
  else
    point_geometry_body<T, ORDER>(a, blockIdx.x - f_blocks, gridDim.x - f_blocks);
}

// The second-order query side and point side in one launch: they read the
// same inputs (ggq, coef, records) and write disjoint outputs, so the first
// q_blocks CTAs run the query side, the next f_blocks the point features and
// the rest the point geometry, side by side instead of one after the other.
template <typename T, int G, int NV, bool VEC>
__global__ void __launch_bounds__(256, 4) order2_fused_kernel(QueryParams<T> qa, PointParams<T> pa, int q_blocks,
                                                              int f_blocks) {
  zero_status_words(qa.zero_status);
  const int blk = (int)blockIdx.x - q_blocks;
  if (blk < 0)
    query_order2_body(qa, blockIdx.x, q_blocks);
  else if (blk < f_blocks)
    point_features_body<T, 2, G, NV, VEC>(pa, blk, f_blocks);
  else
    point_geometry_body<T, 2>(pa, blk - f_blocks, gridDim.x - q_blocks - f_blocks);
}

// ------------------------------------------------------------------ host

BwdLayout bwd_layout(int B, int Q, int P, int F, int K, int dtype) {
  BwdLayout L{};
  const size_t esz = dtype == KNNAG_F64 ? 8 : 4;
  size_t off = 0;
  L.status = off;
  off += 256;
  L.rec = off;
  off += align256((size_t)B * P * kRecLen * esz);
  L.adj = off;
  off += adj_layout(B, Q, P, K).total;
  L.coef = off;
  off += align256((size_t)B * Q * K * esz);
  L.rowsum = off;
  off += align256((size_t)B * P * esz);
  L.total = off;
  return L;
}

namespace {

// First-order query side of `rows` queries: 16-byte loads where f and
// grad_f_out rows are multiples of 16 bytes at 16-byte addresses; two queries
// per warp where 16 lanes cover their columns in as few passes as 32 would (or
// with no columns to sweep), which halves the idle lanes of the geometry.
template <typename T>
int launch_order1(const QueryParams<T>& p, int64_t rows, cudaStream_t st) {
  if (p.frowsum) {
    const bool pairs = !p.segs && p.K <= 16;
    query_order1_broadcast_kernel<T><<<blocks_for((pairs ? (rows + 1) / 2 : rows) * 32, 256), 256, 0, st>>>(p);
    note_launches(1);
    return cudaGetLastError() == cudaSuccess ? KNNAG_OK : KNNAG_ERR_CUDA;
  }
  constexpr int C = 16 / sizeof(T);
  const bool vec = p.F % C == 0 && (uintptr_t)p.f % 16 == 0 && (uintptr_t)p.gfo % 16 == 0;
  const int cols = vec ? p.F / C : p.F;
  const bool half = (cols + 15) / 16 <= 2 * ((cols + 31) / 32) && cols <= 64;
  const unsigned grid = blocks_for((half ? (rows + 1) / 2 : rows) * 32, 256);
  if (vec && half) query_order1_kernel<T, 16, true><<<grid, 256, 0, st>>>(p);
  else if (vec) query_order1_kernel<T, 32, true><<<grid, 256, 0, st>>>(p);
  else if (half) query_order1_kernel<T, 16, false><<<grid, 256, 0, st>>>(p);
  else query_order1_kernel<T, 32, false><<<grid, 256, 0, st>>>(p);
  note_launches(1);
  return cudaGetLastError() == cudaSuccess ? KNNAG_OK : KNNAG_ERR_CUDA;
}

template <typename T>
int launch_query(const QueryParams<T>& p, int order, cudaStream_t st) {
  NvtxRange range("knnag:query_side");
  const int64_t warps = (int64_t)p.B * p.Q;
  const unsigned grid = blocks_for(warps * 32, 256);
  if (order == 1) return launch_order1<T>(p, warps, st);
  query_order2_kernel<T><<<grid, 256, 0, st>>>(p);
  note_launches(1);
  return cudaGetLastError() == cudaSuccess ? KNNAG_OK : KNNAG_ERR_CUDA;
}

}  // namespace

// d(<gfo, f_out>)/dq of a ragged call (gfo null: all ones), weights
// recomputed from idxs.  One warp per query row up to the table's total.
int ragged_grad_q_impl(const char* cs, const void* segs, const float* q, const float* f, int F, const float* gfo,
                       const float* f_row_sums, const int64_t* idxs, int64_t cap_q, float* dq, const int* status,
                       cudaStream_t st) {
  QueryParams<float> p{};
  p.status = status;
  if (!gfo) p.frowsum = f_row_sums;  // all-ones grad_f_out: c = rowsum(f)[idx]
  p.gfo = gfo;
  p.q = q;
  p.f = f;
  p.idxs = idxs;
  p.F = F;
  p.dq = dq;
  p.cs = cs;
  p.segs = segs;
  return launch_order1<float>(p, cap_q, st);
}

int launch_row_sums(const void* f, int64_t rows, int F, int dtype, void* out, cudaStream_t st) {
  if (dtype == KNNAG_F64)
    row_sum_kernel<double><<<blocks_for(rows * 32, 256), 256, 0, st>>>((const double*)f, rows, F, (double*)out);
  else
    row_sum_kernel<float><<<blocks_for(rows * 32, 256), 256, 0, st>>>((const float*)f, rows, F, (float*)out);
  note_launches(1);
  return cudaGetLastError() == cudaSuccess ? KNNAG_OK : KNNAG_ERR_CUDA;
}

namespace {

// How the feature rows are walked: 16-byte groups where grad_f_out and df rows
// allow, else single columns; 16 lanes per entry (two entries side by side)
// where they hold the row, else 32 with up to two groups (eight single columns)
// per lane and as many passes as the row takes.  (37 single columns, B = 3,
// Q = 5003: 17 us with 32 lanes, 24 with 16 lanes of up to four columns.)  0: no rows to walk.
template <typename T>
int point_columns(const PointParams<T>& p) {
  constexpr int C = 16 / sizeof(T);
  if (p.gfo_scalar || !(p.needs & KNNAG_NEED_DF) || p.F == 0) return 0;
  const bool vec = p.F % C == 0 && (uintptr_t)p.gfo % 16 == 0 && (uintptr_t)p.df % 16 == 0;
  const int cols = vec ? p.F / C : p.F;
  if (vec) return cols <= 16 ? 1 : cols <= 32 ? 2 : 3;
  return cols <= 16 ? 4 : cols <= 32 ? 5 : cols <= 64 ? 6 : 7;
}

// Launches KERNEL<..., G, NV, VEC> for a point_columns() code.
#define KNN_POINT_DISPATCH(code, LAUNCH)     \
  switch (code) {                            \
    case 2: LAUNCH(32, 1, true); break;      \
    case 3: LAUNCH(32, 2, true); break;      \
    case 4: LAUNCH(16, 1, false); break;     \
    case 5: LAUNCH(32, 1, false); break;     \
    case 6: LAUNCH(32, 2, false); break;     \
    case 7: LAUNCH(32, 8, false); break;     \
    default: LAUNCH(16, 1, true); break;     \
  }

template <typename T>
bool point_geometry_wanted(const PointParams<T>& p) {
  return (p.needs & (KNNAG_NEED_DP | KNNAG_NEED_DSIGMA | KNNAG_NEED_DR)) != 0 ||
         ((p.needs & KNNAG_NEED_DF) && p.gfo_scalar);
}

template <typename T, int ORDER>
int launch_point_o(const PointParams<T>& p, cudaStream_t st) {
  const unsigned blocks = blocks_for((int64_t)p.B * p.P * 32, 256);
  const int code = point_columns(p);
  const unsigned fb = code ? blocks : 0, grid = fb + (point_geometry_wanted(p) ? blocks : 0);
  if (!grid) return KNNAG_OK;
#define KNN_LAUNCH(G, NV, VEC) point_side_kernel<T, ORDER, G, NV, VEC><<<grid, 256, 0, st>>>(p, (int)fb)
  KNN_POINT_DISPATCH(code, KNN_LAUNCH)
#undef KNN_LAUNCH
  note_launches(1);
  return cudaGetLastError() == cudaSuccess ? KNNAG_OK : KNNAG_ERR_CUDA;
}

template <typename T>
int launch_order2_fused(const QueryParams<T>& qa, const PointParams<T>& pa, cudaStream_t st) {
  const unsigned qb = blocks_for((int64_t)qa.B * qa.Q * 32, 256);
  const unsigned blocks = blocks_for((int64_t)pa.B * pa.P * 32, 256);
  const int code = point_columns(pa);
  const unsigned fb = code ? blocks : 0, grid = qb + fb + (point_geometry_wanted(pa) ? blocks : 0);
#define KNN_LAUNCH(G, NV, VEC) order2_fused_kernel<T, G, NV, VEC><<<grid, 256, 0, st>>>(qa, pa, (int)qb, (int)fb)
  KNN_POINT_DISPATCH(code, KNN_LAUNCH)
#undef KNN_LAUNCH
  note_launches(1);
  return cudaGetLastError() == cudaSuccess ? KNNAG_OK : KNNAG_ERR_CUDA;
}

template <typename T>
int backward_t(const BwdArgs& x, cudaStream_t st) {
  NvtxRange range(x.order == 1 ? "knnag:backward" : "knnag:backward_2nd");
  const BwdLayout L = bwd_layout(x.B, x.Q, x.P, x.F, x.K, x.dtype);
  char* ws = static_cast<char*>(x.workspace);
  int rc = KNNAG_OK;
  int* status = reinterpret_cast<int*>(ws + L.status);
  const void* rec = x.points;
  if (!rec) {
    rc = launch_pack_points(x.p, x.sigma, x.R, x.B, x.P, x.dtype, ws + L.rec, st);
    if (rc) return rc;
    rec = ws + L.rec;
  }
  const int point_bits = KNNAG_NEED_DP | KNNAG_NEED_DF | KNNAG_NEED_DSIGMA | KNNAG_NEED_DR;
  const int geo_bits = KNNAG_NEED_DP | KNNAG_NEED_DSIGMA | KNNAG_NEED_DR;

  const T* coef = static_cast<const T*>(x.coef_in);
  const bool need_coef = (x.order == 1) ? (x.needs & geo_bits) != 0
                                         : (x.needs & (geo_bits | KNNAG_NEED_DQ)) != 0;
  T* coef_ws = reinterpret_cast<T*>(ws + L.coef);
  T* coef_out = static_cast<T*>(x.coef_out);

  const bool gfo_scalar = (x.needs & KNNAG_GFO_SCALAR) != 0;
  T* rowsum = reinterpret_cast<T*>(ws + L.rowsum);
  bool rowsum_ready = false;
  bool query2_pending = false;
  // per-point column sums of f, for the query side with a broadcast grad_f_out
  auto ensure_rowsum = [&]() -> int {
    if (rowsum_ready) return KNNAG_OK;
    row_sum_kernel<T><<<blocks_for((int64_t)x.B * x.P * 32, 256), 256, 0, st>>>((const T*)x.f, (int64_t)x.B * x.P,
                                                                                  x.F, rowsum);
    note_launches(1);
    rowsum_ready = true;
    return cudaGetLastError() == cudaSuccess ? KNNAG_OK : KNNAG_ERR_CUDA;
  };

  QueryParams<T> qp{};
  qp.gfo = (const T*)x.gfo;
  qp.ggq = (const T*)x.ggq;
  qp.q = (const T*)x.q;
  qp.rec = (const T*)rec;
  qp.f = (const T*)x.f;
  qp.w_in = (const T*)x.w_in;
  qp.idxs = x.idxs;
  qp.B = x.B;
  qp.Q = x.Q;
  qp.P = x.P;
  qp.F = x.F;
  qp.K = x.K;
  qp.zero_status = status;

  if (x.order == 1) {
    T* cdst = coef_out ? coef_out : (need_coef ? coef_ws : nullptr);
    if ((x.needs & KNNAG_NEED_DQ) || cdst) {
      qp.dq = (x.needs & KNNAG_NEED_DQ) ? (T*)x.dq : nullptr;
      qp.coef_out = cdst;
      if (gfo_scalar) {
        if ((rc = ensure_rowsum())) return rc;
        qp.frowsum = rowsum;
      }
      rc = launch_query<T>(qp, 1, st);
      if (rc) return rc;
    }
    coef = cdst;
  } else {
    if (!coef && need_coef) {
      QueryParams<T> cp = qp;
      cp.dq = nullptr;
      cp.coef_out = coef_ws;
      if (gfo_scalar) {
        if ((rc = ensure_rowsum())) return rc;
        cp.frowsum = rowsum;
      }
      rc = launch_query<T>(cp, 1, st);
      if (rc) return rc;
      coef = coef_ws;
    }
    if (x.needs & (KNNAG_NEED_DQ | KNNAG_NEED_DGFO)) {
      qp.coef_in = coef;
      qp.dq = (x.needs & KNNAG_NEED_DQ) ? (T*)x.dq : nullptr;
      qp.dgfo = (x.needs & KNNAG_NEED_DGFO) ? (T*)x.dgfo : nullptr;
      query2_pending = true;  // launched with the point side when that runs too
    }
  }

  if (x.needs & point_bits) {
    NvtxRange r("knnag:point_side");
    const void* adj = x.adjacency;
    if (!adj) {
      rc = launch_build_adjacency(x.idxs, x.B, x.Q, x.P, x.K, ws + L.adj, st);
      if (rc) return rc;
      adj = ws + L.adj;
    }
    const AdjLayout AL = adj_layout(x.B, x.Q, x.P, x.K);
    PointParams<T> pp{};
    pp.gfo = (const T*)x.gfo;
    pp.ggq = (const T*)x.ggq;
    pp.q = (const T*)x.q;
    pp.rec = (const T*)rec;
    pp.w_in = (const T*)x.w_in;
    pp.coef = coef;
    pp.rowptr = reinterpret_cast<const int*>(static_cast<const char*>(adj) + AL.rowptr);
    pp.entries = reinterpret_cast<const int*>(static_cast<const char*>(adj) + AL.entries);
    pp.B = x.B;
    pp.Q = x.Q;
    pp.P = x.P;
    pp.F = x.F;
    pp.K = x.K;
    pp.needs = x.needs;
    pp.dp = (T*)x.dp;
    pp.df = (T*)x.df;
    pp.dsigma = (T*)x.dsigma;
    pp.dR = (T*)x.dR;
    pp.gfo_scalar = gfo_scalar;
    pp.zero_status = status;
    if constexpr (sizeof(T) == 4) {  // FP64 keeps separate launches (the fused one spills)
      if (query2_pending) {
        NvtxRange r2("knnag:query_side");
        return launch_order2_fused<T>(qp, pp, st);
      }
    }
    if (query2_pending && (rc = launch_query<T>(qp, 2, st))) return rc;
    rc = (x.order == 1) ? launch_point_o<T, 1>(pp, st) : launch_point_o<T, 2>(pp, st);
    return rc;
  }
  if (query2_pending) rc = launch_query<T>(qp, 2, st);
  return rc;
}

}  // namespace

int backward_impl(const BwdArgs& x, cudaStream_t st) {
  return x.dtype == KNNAG_F64 ? backward_t<double>(x, st) : backward_t<float>(x, st);
}

}  // namespace knnag
