// The reference's other forward ops:
//   * aggregation at caller-given neighbour indices
//     (knn_precomputed_aggregate_aniso_forward, csrc/forward.cu:186-230);
//   * the lookup variant: Euclidean nearest point, then its row of a
//     neighbour table (knn_lookup_aggregate_aniso_forward,
//     csrc/forward.cu:113-183);
//   * the isotropic forward (knn_aggregate_forward, csrc/forward.cu:5-53),
//     served by the exact MinK kernel with Euclidean keys.
// Keys, weights and sums use the same arithmetic and order as the reference,
// so dists / w_out / f_out match it bit for bit.
#include <math.h>

#include "knn_common.cuh"
#include "knn_internal.h"

namespace knnag {

// A warp takes N queries (4, 2 or 1).  The K (query, neighbour) pairs of all of
// them first: key from the packed record, w = exp(-key) (-> dists, w_out); then
// f_out = sum_k w_k f[idx_k] in k order, 32 / N lanes per query side by side: 16
// bytes a lane and eight rows in flight (VEC, where the rows allow) or one column a
// lane.  The neighbour index comes from `idxs` [B,Q,K] or, for the lookup, from
// `table` [P,K] at row nearest[b*Q+q] (and is written to idxs_out).  An index
// outside [0, P) contributes nothing (w = 0, dist = +inf).
//
// Bound by the gathered rows, which L2 serves (K * F values per query).  With the
// packing of the points, at B = 2, Q = 12288, K = 16: F = 64 31 us with a query a
// warp and a column a lane, 25 with four queries; F = 256 82 and, with a query a warp
// and 16 bytes a lane, 47.  Three CTAs per SM for the rows in flight (two: 27 and 64).
template <typename T, int N, bool VEC>
__global__ void __launch_bounds__(256, VEC ? 3 : 5)
    gather_aggregate_kernel(const T* __restrict__ q, const T* __restrict__ f, const T* __restrict__ rec,
                            const int64_t* __restrict__ idxs, const int64_t* __restrict__ table,
                            const int* __restrict__ nearest, int tstride, int B, int Q, int P, int F, int K,
                            T* __restrict__ f_out, T* __restrict__ w_out, T* __restrict__ dists,
                            int64_t* __restrict__ idxs_out) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr int G = 32 / N;  // lanes per query
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, sub = lane / G, gl = lane % G;
  T* sw = reinterpret_cast<T*>(smem_raw) + (size_t)(warp * N + sub) * K;
  int* si = reinterpret_cast<int*>(reinterpret_cast<T*>(smem_raw) + (size_t)(blockDim.x >> 5) * N * K) +
            (size_t)(warp * N + sub) * K;
  const int64_t BQ = (int64_t)B * Q;
  const int64_t gw = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int64_t nw = (gridDim.x * (int64_t)blockDim.x) >> 5;
  for (int64_t base = gw * N; base < BQ; base += nw * N) {
    const int64_t bq = base + sub;
    const int64_t b = (unsigned)bq / (unsigned)Q;  // queries are counted in 32 bits
    if (bq < BQ) {
      const T qx = q[bq * 3 + 0], qy = q[bq * 3 + 1], qz = q[bq * 3 + 2];
      const int64_t row = table ? (int64_t)nearest[bq] : 0;
      for (int k = gl; k < K; k += G) {
        const int64_t e = bq * K + k;
        const int64_t idx = table ? table[row * tstride + k] : idxs[e];
        T key = T(INFINITY), w = T(0);
        if (idx >= 0 && idx < P) {
          key = key_rec<T>(qx, qy, qz, rec + (b * P + idx) * kRecLen);
          w = weight_of(key);
        }
        dists[e] = key;
        w_out[e] = w;
        if (idxs_out) idxs_out[e] = idx;
        sw[k] = w;
        si[k] = (idx >= 0 && idx < P) ? (int)idx : -1;
      }
    }
    __syncwarp();
    if (bq < BQ) {
      const T* fb = f + b * P * F;
      if constexpr (VEC) {
        using V = typename Group16<T>::type;
        constexpr int RB = 8, C = 16 / sizeof(T);
        const int cols = F / C;
        for (int c = gl; c < cols; c += G) {
          T acc[C];
#pragma unroll
          for (int u = 0; u < C; ++u) acc[u] = T(0);
          for (int k0 = 0; k0 < K; k0 += RB) {
            V v[RB];
#pragma unroll
            for (int u = 0; u < RB; ++u)
              if (k0 + u < K && si[k0 + u] >= 0) v[u] = __ldg(reinterpret_cast<const V*>(fb + (int64_t)si[k0 + u] * F) + c);
#pragma unroll
            for (int u = 0; u < RB; ++u)
              if (k0 + u < K && si[k0 + u] >= 0) fma_group(v[u], sw[k0 + u], acc);
          }
          reinterpret_cast<V*>(f_out + bq * F)[c] = group_of(acc);
        }
      } else {
        for (int c = gl; c < F; c += G) {
          T acc = T(0);
          for (int k = 0; k < K; ++k)
            if (si[k] >= 0) acc = fma_rn(__ldg(fb + (int64_t)si[k] * F + c), sw[k], acc);
          f_out[bq * F + c] = acc;
        }
      }
    }
    __syncwarp();
  }
}

// Euclidean nearest point of every query: the smallest
// d = fma(z,z, fma(x,x, y*y)) for x*x + y*y + z*z below 1e10, of equal ones the
// lowest index; 0 when there is none (the reference's strict '<' scan in index
// order from 1e10, csrc/forward.cu:141-160).
//
// A CTA serves 32 queries per lane slot (N slots); its 8 warps share the
// points, four consecutive ones a step, staged in shared memory and broadcast
// to the N queries of a lane.  A step keeps the least of its four distances
// and, when that is below the best so far, its place; which of the four it was
// is found out once at the end, from the same arithmetic.  The broadcasts bound
// it at N = 1, FP32 issue at N = 2 (5 instructions per pair).  One thread per
// query with the whole scan left the chip idle: 96 CTAs at B = 2, Q = 12288,
// P = 4096, 83 us; N = 1 takes 52 us, N = 2 43 us.
constexpr int kNearestChunk = 1024;  // points staged at a time
constexpr int kNearestWarps = 8;

// Squared distances to four points, staged negated: x[4], y[4], z[4].
__device__ __forceinline__ void dist4(float qx, float qy, float qz, const float* s, float (&d)[4]) {
  const float4 px = *reinterpret_cast<const float4*>(s), py = *reinterpret_cast<const float4*>(s + 4),
               pz = *reinterpret_cast<const float4*>(s + 8);
  const float2 X = make_float2(qx, qx), Y = make_float2(qy, qy), Z = make_float2(qz, qz);
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const float2 x = __fadd2_rn(X, h ? make_float2(px.z, px.w) : make_float2(px.x, px.y));
    const float2 y = __fadd2_rn(Y, h ? make_float2(py.z, py.w) : make_float2(py.x, py.y));
    const float2 z = __fadd2_rn(Z, h ? make_float2(pz.z, pz.w) : make_float2(pz.x, pz.y));
    const float2 r = __ffma2_rn(z, z, __ffma2_rn(x, x, __fmul2_rn(y, y)));
    d[2 * h] = r.x;
    d[2 * h + 1] = r.y;
  }
}
__device__ __forceinline__ void dist4(double qx, double qy, double qz, const double* s, double (&d)[4]) {
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    const double x = qx + s[u], y = qy + s[4 + u], z = qz + s[8 + u];
    d[u] = fma_rn(z, z, fma_rn(x, x, mul_rn(y, y)));
  }
}

template <typename T, int N>
__global__ void __launch_bounds__(32 * kNearestWarps) nearest_point_kernel(const T* __restrict__ q,
                                                                           const T* __restrict__ p, int Q, int P,
                                                                           int* __restrict__ nearest) {
  __shared__ __align__(16) T sp[kNearestChunk * 3];  // steps of four points: x[4] y[4] z[4], negated
  __shared__ T sbest[kNearestWarps][32 * N];
  __shared__ int sarg[kNearestWarps][32 * N];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t blocks = (Q + 32 * N - 1) / (32 * N), b = blockIdx.x / blocks;
  const int q0 = (int)(blockIdx.x - b * blocks) * 32 * N + lane;  // queries q0 + 32 u
  const T* pb = p + b * P * 3;
  T qx[N], qy[N], qz[N], best[N];
  int step[N];  // first point of the best step
#pragma unroll
  for (int u = 0; u < N; ++u) {
    const int64_t bq = b * Q + min(q0 + 32 * u, Q - 1);
    qx[u] = q[bq * 3 + 0];
    qy[u] = q[bq * 3 + 1];
    qz[u] = q[bq * 3 + 2];
    best[u] = T(1e10);
    step[u] = -1;
  }
  // four points of step s (of the whole cloud), NaN past the last point: never
  // the nearest
  auto load = [&](int s, T* dst) {
#pragma unroll
    for (int u = 0; u < 4; ++u)
#pragma unroll
      for (int a = 0; a < 3; ++a) dst[4 * a + u] = 4 * s + u < P ? -pb[(int64_t)(4 * s + u) * 3 + a] : T(NAN);
  };
  for (int c0 = 0; c0 < P; c0 += kNearestChunk) {
    const int steps = (min(kNearestChunk, P - c0) + 3) / 4;
    __syncthreads();
    for (int s = tid; s < steps; s += 32 * kNearestWarps) load(c0 / 4 + s, sp + 12 * s);
    __syncthreads();
#pragma unroll 2
    for (int s = warp; s < steps; s += kNearestWarps) {
#pragma unroll
      for (int u = 0; u < N; ++u) {
        T d[4];
        dist4(qx[u], qy[u], qz[u], sp + 12 * s, d);
        const T m = fmin(fmin(d[0], d[1]), fmin(d[2], d[3]));  // NaN only if all are
        if (m < best[u]) {
          best[u] = m;
          step[u] = c0 + 4 * s;
        }
      }
    }
  }
#pragma unroll
  for (int u = 0; u < N; ++u) {
    int arg = 0x7fffffff;
    if (step[u] >= 0) {
      __align__(16) T s[12];
      T d[4];
      load(step[u] / 4, s);
      dist4(qx[u], qy[u], qz[u], s, d);
#pragma unroll
      for (int v = 3; v >= 0; --v)
        if (d[v] == best[u]) arg = step[u] + v;
    }
    sbest[warp][lane + 32 * u] = best[u];
    sarg[warp][lane + 32 * u] = arg;
  }
  __syncthreads();
  if (tid < 32 * N && q0 - lane + tid < Q) {
    T d = sbest[0][tid];
    int arg = sarg[0][tid];
    for (int w = 1; w < kNearestWarps; ++w) {
      const T dw = sbest[w][tid];
      const int i = sarg[w][tid];
      if (dw < d || (dw == d && i < arg)) {
        d = dw;
        arg = i;
      }
    }
    nearest[b * Q + q0 - lane + tid] = arg == 0x7fffffff ? 0 : arg;
  }
}

namespace {
int variant_blocks(int64_t warps, int cta_warps) {
  int dev = 0;
  cudaGetDevice(&dev);
  int64_t b = (warps + cta_warps - 1) / cta_warps;
  const int64_t cap = (int64_t)num_sms(dev) * 16;
  if (b > cap) b = cap;
  return (int)(b < 1 ? 1 : b);
}

// Two queries per lane where that leaves a CTA of 64 queries for every SM.
template <typename T>
int launch_nearest(const T* q, const T* p, int B, int Q, int P, int* nearest, cudaStream_t st) {
  int dev = 0;
  cudaGetDevice(&dev);
  const bool two = (int64_t)B * Q >= (int64_t)num_sms(dev) * 64;
  const int per = two ? 64 : 32;
  const int64_t blocks = (int64_t)((Q + per - 1) / per) * B;
  if (blocks > 0x7fffffff) return KNNAG_ERR_TOO_LARGE;
  if (two)
    nearest_point_kernel<T, 2><<<(unsigned)blocks, 32 * kNearestWarps, 0, st>>>(q, p, Q, P, nearest);
  else
    nearest_point_kernel<T, 1><<<(unsigned)blocks, 32 * kNearestWarps, 0, st>>>(q, p, Q, P, nearest);
  note_launches(1);
  return cudaGetLastError() == cudaSuccess ? KNNAG_OK : KNNAG_ERR_CUDA;
}

template <typename T, int N, bool VEC>
int launch_gather_n(const T* q, const T* f, const T* rec, const int64_t* idxs, const int64_t* table, const int* nearest,
                    int tstride, int B, int Q, int P, int F, int K, T* f_out, T* w_out, T* dists, int64_t* idxs_out,
                    cudaStream_t st) {
  const size_t per_query = (size_t)K * (sizeof(T) + sizeof(int));
  int cta_warps = 8;  // fewer where the neighbours of 8 x N queries do not fit
  while (cta_warps > 1 && cta_warps * N * per_query > 100 * 1024) cta_warps /= 2;
  const size_t smem = cta_warps * N * per_query;
  if (smem > 48 * 1024 && cudaFuncSetAttribute(gather_aggregate_kernel<T, N, VEC>,
                                               cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
    return KNNAG_ERR_CUDA;
  const int64_t warps = ((int64_t)B * Q + N - 1) / N;
  gather_aggregate_kernel<T, N, VEC><<<variant_blocks(warps, cta_warps), 32 * cta_warps, smem, st>>>(
      q, f, rec, idxs, table, nearest, tstride, B, Q, P, F, K, f_out, w_out, dists, idxs_out);
  note_launches(1);
  return cudaGetLastError() == cudaSuccess ? KNNAG_OK : KNNAG_ERR_CUDA;
}

// Queries per warp, and 16 bytes or a column a lane.  Lanes for the columns of a
// row and no more, four queries also where a query is little work, but never so
// few warps that the chip waits for them (12 per SM): F = 700, K = 16 at 1000 queries
// 49, 27 and 19 us with four, two and one; F = 128, K = 64 at 12288 88, 68 and 51,
// K = 4 14 in all ways; F = 16, K = 16 14, 17 and 19.  A query a warp and a column
// a lane for FP64 rows of more than 128 bytes (F = 128, K = 16 at 100000 queries: 204
// us, 16-byte groups 246 to 258) unless a query is little work (F = 24, K = 4: 49, four
// queries 41), and for long lists of narrow rows (F = 16, K = 64: 203, 213).
template <typename T>
int launch_gather(const T* q, const T* f, const T* rec, const int64_t* idxs, const int64_t* table, const int* nearest,
                  int tstride, int B, int Q, int P, int F, int K, T* f_out, T* w_out, T* dists, int64_t* idxs_out,
                  cudaStream_t st) {
  if (8 * (size_t)K * (sizeof(T) + sizeof(int)) > 200 * 1024) return KNNAG_ERR_TOO_LARGE;
  constexpr int C = 16 / sizeof(T);
  const int64_t enough = (int64_t)B * Q / (12 * 148);  // queries per warp that leave 12 warps per SM
  const bool vec = F % C == 0 && (uintptr_t)f % 16 == 0 && (uintptr_t)f_out % 16 == 0;
  const int cols = vec ? F / C : F;
  const int64_t work = (int64_t)K * cols;
  auto go = launch_gather_n<T, 1, false>;
  if (cols <= 8 && !(vec && K > 32)) {
    if (enough >= 2) go = vec ? launch_gather_n<T, 4, true> : launch_gather_n<T, 4, false>;
  } else if constexpr (sizeof(T) == 8) {
    if (vec && work <= 128 && enough >= 8) go = launch_gather_n<T, 4, true>;
  } else if (vec && cols > 8) {
    if (work <= 256 && enough >= 4) go = launch_gather_n<T, 4, true>;
    else if ((work <= 256 || cols <= 16) && enough >= 2) go = launch_gather_n<T, 2, true>;
    else go = launch_gather_n<T, 1, true>;
  }
  return go(q, f, rec, idxs, table, nearest, tstride, B, Q, P, F, K, f_out, w_out, dists, idxs_out, st);
}
}  // namespace

int variants_precomputed(const void* q, const void* f, const void* rec, const int64_t* idxs, int B, int Q, int P,
                         int F, int K, int dtype, void* f_out, void* w_out, void* dists, cudaStream_t st) {
  if (dtype == KNNAG_F64)
    return launch_gather<double>((const double*)q, (const double*)f, (const double*)rec, idxs, nullptr, nullptr, K, B,
                                 Q, P, F, K, (double*)f_out, (double*)w_out, (double*)dists, nullptr, st);
  return launch_gather<float>((const float*)q, (const float*)f, (const float*)rec, idxs, nullptr, nullptr, K, B, Q, P,
                              F, K, (float*)f_out, (float*)w_out, (float*)dists, nullptr, st);
}

int variants_lookup(const void* q, const void* p, const void* f, const void* rec, const int64_t* table, int tstride, int B, int Q,
                    int P, int F, int K, int dtype, int* nearest, void* f_out, void* w_out, void* dists,
                    int64_t* idxs, cudaStream_t st) {
  const int rc = dtype == KNNAG_F64 ? launch_nearest<double>((const double*)q, (const double*)p, B, Q, P, nearest, st)
                                    : launch_nearest<float>((const float*)q, (const float*)p, B, Q, P, nearest, st);
  if (rc) return rc;
  if (dtype == KNNAG_F64)
    return launch_gather<double>((const double*)q, (const double*)f, (const double*)rec, nullptr, table, nearest,
                                 tstride, B, Q, P, F, K, (double*)f_out, (double*)w_out, (double*)dists, idxs, st);
  return launch_gather<float>((const float*)q, (const float*)f, (const float*)rec, nullptr, table, nearest, tstride, B, Q,
                              P, F, K, (float*)f_out, (float*)w_out, (float*)dists, idxs, st);
}

}  // namespace knnag
