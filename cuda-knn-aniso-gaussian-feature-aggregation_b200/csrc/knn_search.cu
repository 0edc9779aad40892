// Forward path: point packing, the plan of the tensor-core search, the exact
// MinK kernel that applies the reference's selection rules to every query (calls
// without an index), workspace layout and the call's order of kernels.  The
// searches are in knn_search_warp.cu and knn_search_tc.cu, the replay of flagged
// queries in knn_replay.cu.
//
// Replaces csrc/forward.cu:56-110 (kernel), csrc/forward.cu:286-338
// (launcher) and csrc/mink.cuh of the reference.
#include <math.h>

#include <algorithm>

#include "knn_common.cuh"
#include "knn_internal.h"
#include "knn_search_dev.cuh"

namespace knnag {

// ------------------------------------------------------------------ packing

// Packing of the search path, grid (bound_parts(B), B): CTA (c, b) packs
// chunk c of batch element b's points, writes the chunk's bounding box to
// parts (what the cell kernels reduce to the element's box), zeroes the
// chunk's adjacency counts (zero_rows, optional) and its share of the cell
// counts; CTA (0, 0) zeroes the call's status words.  FP64 calls also get
// their points and queries rounded to FP32 (pf, qf): the cells are taken
// from those, and so are the boxes of the cells' grid.
template <typename T>
__global__ void __launch_bounds__(256) pack_points_bounded_kernel(
    const T* __restrict__ p, const T* __restrict__ sigma, const T* __restrict__ R, const T* __restrict__ q, int Q,
    int P, T* __restrict__ rec, float* __restrict__ parts, float* __restrict__ pf, float* __restrict__ qf,
    int* __restrict__ zero_words, int n_zero, int* __restrict__ zero_rows, int64_t zero_rows2,
    int* __restrict__ zero_cells, int64_t n_cells) {
  __shared__ float red[6][8];
  const int c = blockIdx.x, b = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (c == 0 && b == 0 && tid < n_zero) zero_words[tid] = 0;
  const int64_t flat = ((int64_t)b * gridDim.x + c) * blockDim.x + tid;
  const int64_t nthreads = (int64_t)gridDim.x * gridDim.y * blockDim.x;
  for (int64_t i = flat; i < n_cells; i += nthreads) zero_cells[i] = 0;
  if constexpr (sizeof(T) == 8)
    for (int64_t i = flat; i < (int64_t)gridDim.y * Q * 3; i += nthreads) qf[i] = (float)q[i];
  const int chunk = (int)(((int64_t)P + gridDim.x - 1) / gridDim.x);
  const int i0 = min(P, c * chunk), i1 = min(P, i0 + chunk);
  float mn[3] = {INFINITY, INFINITY, INFINITY}, mx[3] = {-INFINITY, -INFINITY, -INFINITY};
  for (int k = i0 + tid; k < i1; k += blockDim.x) {
    const int64_t i = (int64_t)b * P + k;
    pack_one<T>(p, sigma, R, i, rec);
    if (zero_rows) zero_rows[i] = zero_rows[i + zero_rows2] = 0;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      const float v = (float)p[i * 3 + a];
      if constexpr (sizeof(T) == 8) pf[i * 3 + a] = v;
      mn[a] = fminf(mn[a], v);
      mx[a] = fmaxf(mx[a], v);
    }
  }
#pragma unroll
  for (int a = 0; a < 3; ++a)
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      mn[a] = fminf(mn[a], __shfl_xor_sync(0xffffffffu, mn[a], o));
      mx[a] = fmaxf(mx[a], __shfl_xor_sync(0xffffffffu, mx[a], o));
    }
  if (lane == 0)
    for (int a = 0; a < 3; ++a) {
      red[a][warp] = mn[a];
      red[3 + a][warp] = mx[a];
    }
  __syncthreads();
  if (tid < 6) {
    float v = tid < 3 ? INFINITY : -INFINITY;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) v = tid < 3 ? fminf(v, red[tid][w]) : fmaxf(v, red[tid][w]);
    parts[((int64_t)b * gridDim.x + c) * 8 + tid] = v;
  }
}

// rec[(b*P+i)*16 + field]: -p, R (row-major), sigma, pad.
// zero_rows (optional): one int per point zeroed too (the adjacency's
// per-point entry counts the forward accumulates), and the one zero_rows2
// further (its fill cursors; 0 where it has none).
template <typename T>
__global__ void pack_points_kernel(const T* __restrict__ p, const T* __restrict__ sigma,
                                   const T* __restrict__ R, int64_t n_points, T* __restrict__ rec,
                                   int* __restrict__ zero_words, int n_zero, int* __restrict__ zero_rows,
                                   int64_t zero_rows2) {
  if (blockIdx.x == 0 && (int)threadIdx.x < n_zero) zero_words[threadIdx.x] = 0;  // the call's status words
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n_points;
       i += (int64_t)gridDim.x * blockDim.x) {
    if (zero_rows) zero_rows[i] = zero_rows[i + zero_rows2] = 0;
    pack_one<T>(p, sigma, R, i, rec);
  }
}

// ------------------------------------------------------------ exact MinK
//
// One CTA per query.  All threads compute the query's keys (same arithmetic
// as everywhere else) into shared memory, chunk by chunk; warp 0 then runs
// the reference's MinK selection over them in index order
// (csrc/mink.cuh:60-81):
//   fill:  the first K points take slots 0..K-1; the tracked maximum moves
//          only for the very first key or a strictly larger one;
//   full:  a point is taken only if strictly below the tracked maximum; it
//          overwrites the maximum's slot; the maximum is re-found by a strict
//          '>' scan that starts from the new key, i.e. it becomes the first
//          slot holding the largest key strictly above the new key, and stays
//          on the written slot when there is none;
//   sort:  bubble sort with a strict '<' swap (csrc/mink.cuh:99-112), which
//          without NaN keys is the stable sort by key.
// For K <= 32 slot s lives in lane s, so the re-scan is a warp max plus a
// ballot and the sort a stable rank; for K > 32, or when a kept key is NaN,
// lane 0 runs the rules sequentially on shared-memory slots.  A ballot
// skips keys that are not below the current maximum (it only falls, so they
// would be rejected anyway).

constexpr int kReplayThreads = 256;

template <typename T>
__host__ __device__ constexpr int replay_chunk() { return sizeof(T) == 4 ? 8192 : 4096; }

template <typename T>
__device__ __forceinline__ T warp_max(T v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// Four CTAs per SM (64 registers): left to itself the compiler holds FP32 to 48,
// which spills (K = 129, B = 1, Q = 22075, P = 906: 28.6 ms against 27.3).
template <typename T>
__global__ void __launch_bounds__(kReplayThreads, sizeof(T) == 4 ? 4 : 0) mink_replay_kernel(ExactParams<T> a) {
  constexpr int NTH = kReplayThreads;
  constexpr int CH = replay_chunk<T>();
  constexpr int HC = CH / 2;  // keys per chunk: two chunk buffers
  constexpr unsigned FULL = 0xffffffffu;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* skey = reinterpret_cast<T*>(smem_raw);
  T* slot_k = skey + CH;
  int* slot_v = reinterpret_cast<int*>(slot_k + a.K);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int F = a.F;
  const SegHeader* sh = static_cast<const SegHeader*>(a.segs);
  if (sh && *a.status) return;
  const int64_t n_items = sh ? sh->bigk_q : (int64_t)a.B * a.Q;

  for (int64_t item = blockIdx.x; item < n_items; item += gridDim.x) {
    // bq: the query's global row; e0: its first entry; b: batch element
    // (uniform) -- records, features and sizes of its cloud
    int64_t bq, e0, b = 0;
    int K, P;
    const T* recb;
    const T* fb;
    if (sh) {
      const SegDesc* sd = seg_descs(a.segs);
      const int s = seg_of_bigk(sd, sh->nseg, item);
      bq = sd[s].q_off + (item - sd[s].bigk_off);
      const SegDesc g = sd[s];
      const CloudDesc c = cloud_descs(a.cs)[g.cloud];
      K = g.K;
      P = c.P;
      e0 = g.e_off + (bq - g.q_off) * K;
      recb = reinterpret_cast<const T*>(a.cs + reinterpret_cast<const CloudSetHeader*>(a.cs)->rec_off) +
             c.p_off * kRecLen;
      fb = a.f + c.p_off * F;
      if (K > a.K || K > P) continue;  // the host checked the table; never reached
    } else {
      bq = item;
      b = bq / a.Q;
      K = a.K;
      P = a.P;
      e0 = bq * K;
      recb = a.rec + b * (int64_t)P * kRecLen;
      fb = a.f + b * (int64_t)P * F;
    }
    const bool in_lanes = K <= 32;
    const T qx = a.q[bq * 3 + 0], qy = a.q[bq * 3 + 1], qz = a.q[bq * 3 + 2];

    int size = 0, max_idx = 0, my_v = -1;
    T max_key = T(0), my_k = T(0);
    // Keys of chunk [c0, c0 + HC) into buf by threads first .. first + nth - 1
    // (four keys in flight per thread).
    auto fill = [&](int c0, T* buf, int first, int nth) {
      const int n = min(HC, P - c0);
      if (a.iso_p) {
        // squared Euclidean distance, accumulated as d = 0; d += c*c (csrc/forward.cu:32-36)
        const T* pb = a.iso_p + b * (int64_t)P * 3;
#pragma unroll 4
        for (int i = tid - first; i < n; i += nth) {
          const T* pp = pb + (int64_t)(c0 + i) * 3;
          const T x = qx - pp[0], y = qy - pp[1], z = qz - pp[2];
          buf[i] = fma_rn(z, z, fma_rn(y, y, mul_rn(x, x)));
        }
      } else {
#pragma unroll 4
        for (int i = tid - first; i < n; i += nth) buf[i] = key_rec<T>(qx, qy, qz, recb + (int64_t)(c0 + i) * kRecLen);
      }
    };
    // Two chunk buffers: while warp 0 runs MinK over chunk c in index order,
    // the other warps compute the keys of chunk c + 1.
    fill(0, skey, 0, NTH);
    __syncthreads();
    for (int c0 = 0, ci = 0; c0 < P; c0 += HC, ++ci) {
      const int n = min(HC, P - c0);
      const T* cur = skey + (ci & 1) * HC;
      if (warp != 0) {
        if (c0 + HC < P) fill(c0 + HC, skey + ((ci + 1) & 1) * HC, 32, NTH - 32);
      } else {
        // An accepted key kl (strictly below the max) at point index idx
        // replaces the max slot; the max is found again.
        auto accept = [&](T kl, int idx) {
          if (in_lanes) {
            if (lane == max_idx) {
              my_k = kl;
              my_v = idx;
            }
            const T v = (lane < K && my_k > kl) ? my_k : T(-INFINITY);
            const T m = warp_max(v);
            if (m > kl) {
              max_key = m;
              max_idx = __ffs(__ballot_sync(FULL, lane < K && v == m)) - 1;
            } else {
              max_key = kl;
            }
          } else {
            if (lane == 0) {
              slot_k[max_idx] = kl;
              slot_v[max_idx] = idx;
            }
            __syncwarp();
            max_key = kl;
            for (int s2 = 0; s2 < K; ++s2) {
              const T c = slot_k[s2];
              if (c > max_key) {
                max_key = c;
                max_idx = s2;
              }
            }
            __syncwarp();
          }
        };
        for (int base = 0; base < n;) {
          if (size >= K && base + 128 <= n) {
            // full list: 128 keys per step, lane l holding keys 4l .. 4l+3;
            // candidates in index order (lanes ascending, then t), each
            // checked against the max at its turn
            T k4[4];
#pragma unroll
            for (int t = 0; t < 4; ++t) k4[t] = cur[base + 4 * lane + t];
            const bool any = k4[0] < max_key || k4[1] < max_key || k4[2] < max_key || k4[3] < max_key;
            unsigned cand = __ballot_sync(FULL, any);
            while (cand) {
              const int l = __ffs(cand) - 1;
              cand &= cand - 1;
#pragma unroll
              for (int t = 0; t < 4; ++t) {
                const T kl = __shfl_sync(FULL, k4[t], l);
                if (kl < max_key) accept(kl, c0 + base + 4 * l + t);
              }
            }
            base += 128;
            continue;
          }
          const int nvalid = min(32, n - base);
          const T key = lane < nvalid ? cur[base + lane] : T(0);
          int j = 0;
          while (j < nvalid && size < K) {  // fill phase (uniform across the warp)
            const T kj = __shfl_sync(FULL, key, j);
            if (in_lanes) {
              if (lane == size) {
                my_k = kj;
                my_v = c0 + base + j;
              }
            } else if (lane == 0) {
              slot_k[size] = kj;
              slot_v[size] = c0 + base + j;
            }
            if (size == 0 || kj > max_key) {
              max_key = kj;
              max_idx = size;
            }
            ++size;
            ++j;
          }
          __syncwarp();
          if (j < nvalid) {
            unsigned cand = __ballot_sync(FULL, lane >= j && lane < nvalid && key < max_key);
            while (cand) {
              const int l = __ffs(cand) - 1;
              cand &= cand - 1;
              const T kl = __shfl_sync(FULL, key, l);
              if (!(kl < max_key)) continue;
              accept(kl, c0 + base + l);
            }
          }
          base += 32;
        }
      }
      __syncthreads();
    }
    if (warp == 0) {
      if (in_lanes && !__any_sync(FULL, lane < K && my_k != my_k)) {
        int rank = 0;
        for (int t = 0; t < K; ++t) {
          const T kt = __shfl_sync(FULL, my_k, t);
          rank += (kt < my_k || (kt == my_k && t < lane)) ? 1 : 0;
        }
        if (lane < K) {
          slot_k[rank] = my_k;
          slot_v[rank] = my_v;
        }
      } else {
        if (in_lanes && lane < K) {
          slot_k[lane] = my_k;
          slot_v[lane] = my_v;
        }
        __syncwarp();
        if (lane == 0) bubble_sort_slots(slot_k, slot_v, size);
      }
    }
    __syncthreads();
    if (a.iso_p) {
      // isotropic weights w_k = exp(-(d_k * sigma[idx_k][0])) and their sum
      // in k order (csrc/forward.cu:43-52); keep w_k in slot_k
      const T* sg = a.iso_sigma + b * (int64_t)P * a.iso_stride;
      for (int k = tid; k < K; k += NTH) {
        const int64_t e = e0 + k;
        a.dists[e] = slot_k[k];
        a.idxs[e] = (int64_t)slot_v[k];
      }
      __syncthreads();
      for (int k = tid; k < K; k += NTH)
        slot_k[k] = weight_of(mul_rn(slot_k[k], sg[(int64_t)slot_v[k] * a.iso_stride]));
      __syncthreads();
      if (tid == 0) {
        T ws = T(0);
        for (int k = 0; k < K; ++k) ws = add_rn(ws, slot_k[k]);
        a.w_out[bq] = ws;
      }
    } else {
      for (int k = tid; k < K; k += NTH) {
        const int64_t e = e0 + k;
        a.dists[e] = slot_k[k];
        a.idxs[e] = (int64_t)slot_v[k];
        a.w_out[e] = weight_of(slot_k[k]);
        if (a.adj_count && (unsigned)slot_v[k] < (unsigned)P) atomicAdd(&a.adj_count[b * P + slot_v[k]], 1);
      }
      __syncthreads();
      for (int k = tid; k < K; k += NTH) slot_k[k] = weight_of(slot_k[k]);
      __syncthreads();
    }
    for (int c = tid; c < F; c += NTH) {
      T acc = T(0);
      for (int k = 0; k < K; ++k) acc = fma_rn(fb[(int64_t)slot_v[k] * F + c], slot_k[k], acc);
      a.f_out[bq * F + c] = acc;
    }
    __syncthreads();
  }
}

// ------------------------------------------------------------ search plan
//
// search_plan_kernel, one CTA per block of qpc sorted queries (grid (nb, B),
// 16 queries per warp): the seed thresholds of the block's queries
// (seed_warp) into tau0, and the block's estimate -- the number of tiles
// whose bound against the block's query box is at most its largest seed,
// the tiles its search may visit -- into plan_est.
// search_items_kernel, one CTA of 1024 threads, turns the estimates into the
// search's CTA items (batch element, query range): blocks ordered by
// estimate, heaviest first, in kPlanGroups groups of about equal population
// (block order inside a group), so the heaviest blocks start in the first
// waves and the light ones fill the last.  The plan runs only when the
// blocks take more than one wave: in one wave every block starts at once and
// the order changes nothing (splitting the heaviest blocks over the spare
// slots of a wave was measured, and gained less than the plan cost).
// Items only decide which CTA runs which queries: results do not change.
constexpr int kPlanBins = 1024;
constexpr int kPlanGroups = 8;
constexpr int kPlanQPW = 16;              // queries per warp of the plan kernel
constexpr int kPlanItemsThreads = 1024;
constexpr int kPlanMaxBlocks = 32768;     // estimates staged in shared memory (128 KB)

// Exclusive scan of one int per thread over the CTA; *total gets the sum.
// wsum: 33 ints of shared memory.  Every thread of the CTA must call it.
__device__ __forceinline__ int cta_scan_excl(int v, int* wsum, int* total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  int incl = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int t = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += t;
  }
  if (lane == 31) wsum[warp] = incl;
  __syncthreads();
  if (warp == 0) {
    const int w = lane < nw ? wsum[lane] : 0;
    int wi = w;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, wi, o);
      if (lane >= o) wi += t;
    }
    if (lane < nw) wsum[lane] = wi - w;
    if (lane == 31) wsum[32] = wi;
  }
  __syncthreads();
  const int r = wsum[warp] + incl - v;
  *total = wsum[32];
  __syncthreads();  // wsum is reused by the next call
  return r;
}

__device__ __forceinline__ int4 plan_item(int bt, int nb, int qpc, int Q) {
  const int b = bt / nb, blk = bt - b * nb;
  const int q0 = blk * qpc;
  return make_int4(b, q0, min(q0 + qpc, Q), 0);
}

template <int KMAX>
__global__ void __launch_bounds__(256) search_plan_kernel(SearchParams a, int qpc, int nb) {
  constexpr int NQ = kPlanQPW;
  __shared__ float4 tab[256 / 32 * NQ];
  __shared__ float red[8][8];
  __shared__ int wsum[33];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, nw = blockDim.x >> 5;
  const int b = blockIdx.y, blk = blockIdx.x;
  const int q0 = blk * qpc, q1 = min(q0 + qpc, a.Q);
  const int sp = q0 + warp * NQ + lane;
  const bool valid = lane < NQ && sp < q1;
  const int64_t qrow = (int64_t)b * a.Q;
  int qi = valid ? a.perm_q[qrow + sp] : 0;
  if ((unsigned)qi >= (unsigned)a.Q) qi = 0;  // the search flags a bad permutation
  const float* qb = a.q + qrow * 3;
  const float x = qb[(int64_t)qi * 3 + 0], y = qb[(int64_t)qi * 3 + 1], z = qb[(int64_t)qi * 3 + 2];
  if (lane < NQ) tab[warp * NQ + lane] = make_float4(x, y, z, INFINITY);
  const int my_seed = valid ? a.qseed[qrow + sp] : 0;
  __syncwarp();
  seed_warp<KMAX, NQ>(tab + warp * NQ, my_seed, valid, a.pairs + (int64_t)b * (a.P_pad / 2) * kPairFloats, a.P,
                      a.K, lane);
  __syncwarp();
  float t0 = -INFINITY;
  if (valid) {
    t0 = tab[warp * NQ + lane].w;
    a.tau0[qrow + sp] = t0;
  }
  // the block's query box and largest seed
  float v[7] = {valid ? x : INFINITY,  valid ? y : INFINITY,  valid ? z : INFINITY, valid ? x : -INFINITY,
                valid ? y : -INFINITY, valid ? z : -INFINITY, t0};
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
    for (int c = 0; c < 3; ++c) v[c] = fminf(v[c], __shfl_xor_sync(0xffffffffu, v[c], o));
#pragma unroll
    for (int c = 3; c < 7; ++c) v[c] = fmaxf(v[c], __shfl_xor_sync(0xffffffffu, v[c], o));
  }
  if (lane == 0)
#pragma unroll
    for (int c = 0; c < 7; ++c) red[warp][c] = v[c];
  __syncthreads();
  float bmin[3], bmax[3], tmax0 = -INFINITY;
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    bmin[c] = INFINITY;
    bmax[c] = -INFINITY;
  }
  for (int w = 0; w < nw; ++w) {
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      bmin[c] = fminf(bmin[c], red[w][c]);
      bmax[c] = fmaxf(bmax[c], red[w][3 + c]);
    }
    tmax0 = fmaxf(tmax0, red[w][6]);
  }
  // the tiles the block's search may visit
  const float* tinfo_b = a.tinfo + (int64_t)b * a.ntile * kTinfoFloats;
  int c = 0;
  for (int t = tid; t < a.ntile; t += blockDim.x)
    c += tile_lower_bound(tinfo_b + (int64_t)t * kTinfoFloats, bmin, bmax) > tmax0 ? 0 : 1;
  int est;
  cta_scan_excl(c, wsum, &est);
  if (tid == 0) a.plan_est[(int64_t)b * nb + blk] = est;
}

// The item table from the estimates of nbt = B * nb blocks (one CTA of
// kPlanItemsThreads threads; dynamic shared memory: nbt ints).
__global__ void __launch_bounds__(kPlanItemsThreads) search_items_kernel(SearchParams a, int nb, int qpc) {
  extern __shared__ int est[];  // [nbt]
  __shared__ int hist[kPlanBins];
  __shared__ int wsum[33];
  __shared__ int misc[2 * kPlanGroups];
  const int tid = threadIdx.x, nth = blockDim.x;
  const int nbt = a.B * nb;
  const int nbins = a.ntile + 1 < kPlanBins ? a.ntile + 1 : kPlanBins;  // estimates are in [0, ntile]
  for (int i = tid; i < nbt; i += nth) {
    const int e = a.plan_est[i];
    est[i] = e < nbins - 1 ? e : nbins - 1;  // the bin
  }
  for (int i = tid; i < kPlanBins; i += nth) hist[i] = 0;
  if (tid < 2 * kPlanGroups) misc[tid] = 0;
  __syncthreads();
  for (int i = tid; i < nbt; i += nth) atomicAdd(&hist[est[i]], 1);
  __syncthreads();
  // blocks in bins above bin t (heaviest first): one bin per thread
  const int t = nbins - 1 - tid;  // thread tid holds bin t (tid < nbins)
  const int h = tid < nbins ? hist[t] : 0;
  int tot;
  const int above = cta_scan_excl(h, wsum, &tot);
  const int chunk = (nbt + nth - 1) / nth;  // thread tid takes blocks [i0, i1) in order
  const int i0 = min(nbt, tid * chunk), i1 = min(nbt, i0 + chunk);
  // group of each bin (heaviest bins first), each group's size and first item
  __syncthreads();  // every thread read its bin's count
  if (tid < nbins) {
    const int g = min(kPlanGroups - 1, (int)((int64_t)above * kPlanGroups / nbt));
    hist[t] = g;
    atomicAdd(&misc[g], h);
  }
  __syncthreads();
  if (tid == 0) {
    int o = 0;
    for (int g = 0; g < kPlanGroups; ++g) {
      misc[kPlanGroups + g] = o;
      o += misc[g];
    }
  }
  __syncthreads();
  int cnt[kPlanGroups], base[kPlanGroups];
#pragma unroll
  for (int g = 0; g < kPlanGroups; ++g) cnt[g] = 0;
  for (int i = i0; i < i1; ++i) {
    const int g = hist[est[i]];
#pragma unroll
    for (int u = 0; u < kPlanGroups; ++u) cnt[u] += g == u ? 1 : 0;
  }
#pragma unroll
  for (int g = 0; g < kPlanGroups; ++g) base[g] = misc[kPlanGroups + g] + cta_scan_excl(cnt[g], wsum, &tot);
  for (int i = i0; i < i1; ++i) {
    const int g = hist[est[i]];
    int p = 0;
#pragma unroll
    for (int u = 0; u < kPlanGroups; ++u)
      if (g == u) p = base[u]++;
    a.items[p] = plan_item(i, nb, qpc, a.Q);
  }
}

// ------------------------------------------------------------------ host

int num_sms(int dev) {
  static int cache[64] = {0};
  if (dev < 0 || dev >= 64) return 148;
  if (!cache[dev]) {
    int v = 0;
    if (cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || v <= 0) v = 148;
    cache[dev] = v;
  }
  return cache[dev];
}

namespace {

// Launch shape of the one-warp-per-query search (see search_qpw): a unit of
// four queries per warp, fewer when that would leave the chip's 24 warps per
// SM without work.
int choose_warp_shape(int B, int Q, int dev) {
  const int64_t n = (int64_t)B * Q, slots = (int64_t)num_sms(dev) * 24;
  return n <= slots ? 64 : n <= 2 * slots ? 32 : 4;
}

// The process-wide setting when one is made, else by size.  While the test
// hook of the bounded waits is armed the tensor-core search runs: it is the
// one that waits (on its tile copies).
int choose_splits(int B, int Q, int dev, bool stalled) {
  const int forced = search_splits_setting();
  if (search_setting_ok(forced)) return forced;
  if (stalled) return kShapeTensorFilter;
  return choose_warp_shape(B, Q, dev);
}

inline unsigned grid_for(int64_t n, int threads, int dev) {
  int64_t b = (n + threads - 1) / threads;
  const int64_t cap = (int64_t)num_sms(dev) * 32;
  if (b > cap) b = cap;
  return (unsigned)(b < 1 ? 1 : b);
}

}  // namespace

int search_plan_max_blocks() { return kPlanMaxBlocks; }

int launch_search_plan(const SearchParams& a, int qpc, int nb, cudaStream_t st) {
  const int64_t nbt = (int64_t)nb * a.B;
  if (nbt > kPlanMaxBlocks || !a.items || !a.tau0 || !a.plan_est) return KNNAG_ERR_ARG;
  int dev = 0;
  cudaGetDevice(&dev);
  static int items_smem[64];
  if (dev >= 0 && dev < 64 && items_smem[dev] < kPlanMaxBlocks * 4) {
    if (cudaFuncSetAttribute(search_items_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kPlanMaxBlocks * 4) !=
        cudaSuccess)
      return KNNAG_ERR_CUDA;
    items_smem[dev] = kPlanMaxBlocks * 4;
  }
  const dim3 grid((unsigned)nb, (unsigned)a.B);
  const unsigned threads = 32 * ((qpc + kPlanQPW - 1) / kPlanQPW);
  if (a.K <= 8)
    search_plan_kernel<8><<<grid, threads, 0, st>>>(a, qpc, nb);
  else if (a.K <= 16)
    search_plan_kernel<16><<<grid, threads, 0, st>>>(a, qpc, nb);
  else
    search_plan_kernel<32><<<grid, threads, 0, st>>>(a, qpc, nb);
  search_items_kernel<<<1, kPlanItemsThreads, (size_t)nbt * 4, st>>>(a, nb, qpc);
  note_launches(2);
  return cudaGetLastError() == cudaSuccess ? KNNAG_OK : KNNAG_ERR_CUDA;
}

template <typename T>
int launch_exact(const ExactParams<T>& a, cudaStream_t st) {
  const size_t smem = (size_t)replay_chunk<T>() * sizeof(T) + (size_t)a.K * (sizeof(T) + sizeof(int));
  if (smem > 200 * 1024) return KNNAG_ERR_TOO_LARGE;
  auto kernel = mink_replay_kernel<T>;
  if (smem > 48 * 1024 && cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) !=
                              cudaSuccess)
    return KNNAG_ERR_CUDA;
  int dev = 0;
  cudaGetDevice(&dev);
  int64_t blocks = (int64_t)a.B * a.Q;
  const int64_t cap = (int64_t)num_sms(dev) * 8;
  if (blocks > cap) blocks = cap;
  if (blocks < 1) blocks = 1;
  profile_begin(st);
  kernel<<<(unsigned)blocks, kReplayThreads, smem, st>>>(a);
  profile_end(st);
  note_launches(1);
  return cudaGetLastError() == cudaSuccess ? KNNAG_OK : KNNAG_ERR_CUDA;
}

template int launch_exact<float>(const ExactParams<float>&, cudaStream_t);
template int launch_exact<double>(const ExactParams<double>&, cudaStream_t);

FwdLayout fwd_layout(int B, int Q, int P, int K, int dtype, bool own_rec, bool indexed) {
  FwdLayout L{};
  const size_t esz = dtype == KNNAG_F64 ? 8 : 4;
  size_t off = 0;
  L.status = off;
  off += 256;
  L.flag_list = off;
  off += align256((size_t)B * Q * 4);
  L.rec = off;
  if (own_rec) off += align256((size_t)B * P * kRecLen * esz);
  L.P_pad = (int)round_up(P, kTilePoints);
  L.pairs = L.bounds = L.cell_count = L.cell_offset = L.perm_p = L.perm_q = L.tinfo = L.qseed = L.tau0 =
      L.plan_est = L.items = L.tcops = L.tcinfo = L.tbox = L.sbox = L.gbox = L.pf = L.qf = off;
  L.bits = 0;
  if (indexed) {
    L.bits = point_bits(P);
    const size_t cells = (size_t)1 << (3 * L.bits);
    const size_t ntiles = (size_t)B * (L.P_pad / kTilePoints);
    L.pairs = off;
    off += align256((size_t)B * L.P_pad * kRecLen * esz);
    // what the sort alone uses, and in the same place what the tile-info kernel
    // writes after it: the tensor-core filter's B operands
    const size_t sort_at = off;
    L.bounds = off;  // per element bound_parts(B) partial boxes
    off += align256((size_t)B * bound_parts(B) * 8 * 4);
    // point and query cells of each batch element, sorted together
    L.cell_count = off;
    off += align256(2 * (size_t)B * cells * 4);
    L.cell_offset = off;
    off += align256((2 * (size_t)B * cells + 1) * 4);
    L.tcops = sort_at;
    if (dtype == KNNAG_F32 && K <= 32) off = std::max(off, sort_at + align256(ntiles * kTcOpsBytes));
    L.perm_p = off;  // perm_q follows perm_p without a gap (one scatter fills both)
    L.perm_q = off + (size_t)B * P * 4;
    off += align256((size_t)B * P * 4 + (size_t)B * Q * 4);
    L.tinfo = off;
    off += align256(ntiles * kTinfoBytes);
    L.tbox = off;
    off += align256(ntiles * 7 * 4);
    L.sbox = off;
    off += align256(ntiles * 8 * 16);
    L.gbox = off;
    off += align256((size_t)B * ((L.P_pad / kTilePoints + 31) / 32) * 7 * 4);
    L.qseed = off;
    off += align256((size_t)B * Q * 4);
    if (dtype == KNNAG_F64) {
      L.pf = off;
      off += align256((size_t)B * P * 3 * 4);
      L.qf = off;
      off += align256((size_t)B * Q * 3 * 4);
    } else if (K <= 32) {
      // search plan of the tensor-core search: seed thresholds, per-block
      // estimates, CTA items
      const size_t nb_max = (size_t)B * ((Q + 7) / 8);
      L.tau0 = off;
      off += align256((size_t)B * Q * 4);
      L.plan_est = off;
      off += align256(nb_max * 4);
      L.items = off;
      off += align256(nb_max * 16);
      // tensor-core filter: bound terms of every tile
      L.tcinfo = off;
      off += align256(ntiles * kTcInfoBytes);
    }
  }
  L.total = off;
  return L;
}

FwdLayout fwd_layout_in(int B, int Q, int P, int K, int dtype, bool own_rec, size_t bytes, bool* indexed) {
  *indexed = forward_indexed(B, Q, P, K, dtype);
  FwdLayout L = fwd_layout(B, Q, P, K, dtype, own_rec, *indexed);
  if (*indexed && L.total > bytes && (dtype == KNNAG_F64 || K > 32)) {
    *indexed = false;
    L = fwd_layout(B, Q, P, K, dtype, own_rec, false);
  }
  return L;
}

template <typename T>
int launch_pack_points_bounded(const T* p, const T* sigma, const T* R, const T* q, int B, int Q, int P, T* rec,
                               float* parts, float* pf, float* qf, cudaStream_t st, int* zero_words, int n_zero,
                               int* zero_rows, int64_t zero_rows2, int* zero_cells, int64_t n_cells) {
  pack_points_bounded_kernel<T><<<dim3(bound_parts(B), B), 256, 0, st>>>(p, sigma, R, q, Q, P, rec, parts, pf, qf,
                                                                      zero_words, n_zero, zero_rows, zero_rows2, zero_cells,
                                                                      n_cells);
  note_launches(1);
  return cudaGetLastError() == cudaSuccess ? KNNAG_OK : KNNAG_ERR_CUDA;
}

int launch_pack_points(const void* p, const void* sigma, const void* R, int B, int P, int dtype, void* rec,
                       cudaStream_t st, int* zero_words, int n_zero, int* zero_rows, int64_t zero_rows2) {
  int dev = 0;
  cudaGetDevice(&dev);
  const int64_t n = (int64_t)B * P;
  if (dtype == KNNAG_F64)
    pack_points_kernel<double><<<grid_for(n, 256, dev), 256, 0, st>>>(
        (const double*)p, (const double*)sigma, (const double*)R, n, (double*)rec, zero_words, n_zero, zero_rows,
        zero_rows2);
  else
    pack_points_kernel<float><<<grid_for(n, 256, dev), 256, 0, st>>>((const float*)p, (const float*)sigma,
                                                                     (const float*)R, n, (float*)rec, zero_words,
                                                                     n_zero, zero_rows, zero_rows2);
  note_launches(1);
  return cudaGetLastError() == cudaSuccess ? KNNAG_OK : KNNAG_ERR_CUDA;
}

template <typename T>
static int forward_exact_all(const T* q, const T* rec, const T* f, int B, int Q, int P, int F, int K, T* f_out,
                             T* w_out, T* dists, int64_t* idxs, int* adj_count, cudaStream_t st) {
  ExactParams<T> e{q, rec, f, nullptr, nullptr, 0, B, Q, P, F, K, nullptr, nullptr, f_out, w_out, dists, idxs};
  e.adj_count = adj_count;
  return launch_exact<T>(e, st);
}

// The forward through the spatial index: pack, sort, search, exact replay of
// the flagged queries.
template <typename T>
static int forward_indexed_t(const T* q, const T* p, const T* f, const T* sigma, const T* R, int B, int Q, int P, int F,
                             int K, T* f_out, T* w_out, T* dists, int64_t* idxs, T* rec, char* ws, const FwdLayout& L,
                             int* adj_count, cudaStream_t st) {
  int* status = reinterpret_cast<int*>(ws + L.status);
  int* flag_count = status + 1;
  int* flag_list = reinterpret_cast<int*>(ws + L.flag_list);
  float* pf = reinterpret_cast<float*>(ws + L.pf);
  float* qf = reinterpret_cast<float*>(ws + L.qf);
  const int ntile = L.P_pad / kTilePoints;
  const AdjLayout AL = adj_layout(B, Q, P, K);
  const int64_t fill_off = AL.fill < AL.total ? (int64_t)(AL.fill - AL.cursor) / 4 : 0;
  int rc;
  int dev = 0;
  cudaGetDevice(&dev);
  SearchParams sp{};
  apply_search_debug(sp);
  int G = choose_warp_shape(B, Q, dev);
  if (sizeof(T) == 4 && K <= 32) G = choose_splits(B, Q, dev, sp.stall_visit >= 0);
  if (G == kShapeTensorFilter && !search_tc_fits(ntile)) G = choose_warp_shape(B, Q, dev);
  if (ntile > kSearchMaxTiles) return KNNAG_ERR_TOO_LARGE;
  if (G != kShapeTensorFilter && index_in_one_launch(B, Q, P)) {
    NvtxRange r("knnag:spatial_index");
    rc = launch_index_cluster<T>(p, sigma, R, q, B, Q, P, rec, ws, L, st, status, 2, adj_count, fill_off);
    if (rc) return rc;
  } else {
    {
      NvtxRange r("knnag:pack_points");
      // also zeroes the status words and the adjacency's entry counts, and
      // bounds the points; cell counts and offsets (the offsets are the
      // scatter's cursors when the scan is folded into it) are zeroed, padding
      // between them included
      rc = launch_pack_points_bounded<T>(
          p, sigma, R, q, B, Q, P, rec, reinterpret_cast<float*>(ws + L.bounds), pf, qf, st, status, 2, adj_count,
          fill_off, reinterpret_cast<int*>(ws + L.cell_count),
          (int64_t)(L.cell_offset - L.cell_count) / 4 + (2 * (int64_t)B << (3 * L.bits)) + 1);
    }
    if (rc) return rc;
    NvtxRange r("knnag:spatial_index");
    rc = launch_spatial_index<T>(sizeof(T) == 4 ? reinterpret_cast<const float*>(q) : qf, pf, rec, B, Q, P, L.P_pad, ws,
                                 L, st, G == kShapeTensorFilter);
    if (rc) return rc;
  }
  const int vec = F < (1 << 28) && (F % (16 / (int)sizeof(T)) == 0) && ((uintptr_t)f % 16 == 0) && ((uintptr_t)f_out % 16 == 0);
  if (G == kShapeTensorFilter) {
    NvtxRange r("knnag:search_tc");
    sp.q = reinterpret_cast<const float*>(q);
    sp.perm_q = reinterpret_cast<const int*>(ws + L.perm_q);
    sp.tinfo = reinterpret_cast<const float*>(ws + L.tinfo);
    sp.ntile = ntile;
    sp.pairs = reinterpret_cast<const float*>(ws + L.pairs);
    sp.rec = reinterpret_cast<const float*>(rec);
    sp.f = reinterpret_cast<const float*>(f);
    sp.B = B;
    sp.Q = Q;
    sp.P = P;
    sp.P_pad = L.P_pad;
    sp.F = F;
    sp.K = K;
    sp.vec4 = vec;
    sp.f_out = reinterpret_cast<float*>(f_out);
    sp.w_out = reinterpret_cast<float*>(w_out);
    sp.dists = reinterpret_cast<float*>(dists);
    sp.idxs = idxs;
    sp.status = status;
    sp.flag_count = flag_count;
    sp.flag_list = flag_list;
    sp.adj_count = adj_count;
    sp.qseed = reinterpret_cast<const int*>(ws + L.qseed);
    sp.tau0 = reinterpret_cast<float*>(ws + L.tau0);
    sp.plan_est = reinterpret_cast<int*>(ws + L.plan_est);
    sp.items = reinterpret_cast<int4*>(ws + L.items);
    sp.tcops = reinterpret_cast<const float*>(ws + L.tcops);
    sp.tcinfo = reinterpret_cast<const float*>(ws + L.tcinfo);
    rc = launch_search_tc(sp, st);
  } else {
    NvtxRange r("knnag:search");
    WarpSearchParams<T> wp{};
    wp.q = q;
    wp.perm_q = reinterpret_cast<const int*>(ws + L.perm_q);
    wp.qseed = reinterpret_cast<const int*>(ws + L.qseed);
    wp.rec = rec;
    wp.pairs = reinterpret_cast<const T*>(ws + L.pairs);
    wp.tbox = reinterpret_cast<const float*>(ws + L.tbox);
    wp.sbox = reinterpret_cast<const float4*>(ws + L.sbox);
    wp.gbox = reinterpret_cast<const float*>(ws + L.gbox);
    wp.ngroup = (ntile + 31) / 32;
    wp.f = f;
    wp.B = B;
    wp.Q = Q;
    wp.P = P;
    wp.F = F;
    wp.K = K;
    wp.ntile = ntile;
    wp.vec = vec;
    wp.f_out = f_out;
    wp.w_out = w_out;
    wp.dists = dists;
    wp.idxs = idxs;
    wp.status = status;
    wp.flag_count = flag_count;
    wp.flag_list = flag_list;
    wp.adj_count = adj_count;
    rc = launch_search_warp<T>(wp, G, st);
  }
  if (rc) return rc;
  // Exact MinK replay of the flagged queries (count read on the device).
  NvtxRange r("knnag:replay_flagged");
  ExactParams<T> e{q, rec, f, nullptr, nullptr, 0, B, Q, P, F, K, flag_list, flag_count, f_out, w_out, dists, idxs};
  e.adj_count = adj_count;
  return launch_replay_list<T>(e, P, st);
}

template <typename T>
static int forward_t(const T* q, const T* p, const T* f, const T* sigma, const T* R, int B, int Q, int P, int F, int K,
                     int dtype, T* f_out, T* w_out, T* dists, int64_t* idxs, void* points, char* ws, size_t ws_bytes,
                     int* adj_count, cudaStream_t st) {
  bool indexed = false;
  const FwdLayout L = fwd_layout_in(B, Q, P, K, dtype, points == nullptr, ws_bytes, &indexed);
  if (L.total > ws_bytes) return KNNAG_ERR_WORKSPACE;
  T* rec = points ? static_cast<T*>(points) : reinterpret_cast<T*>(ws + L.rec);
  if (indexed)
    return forward_indexed_t<T>(q, p, f, sigma, R, B, Q, P, F, K, f_out, w_out, dists, idxs, rec, ws, L, adj_count, st);
  // the exact kernel serves every query; the packing zeroes the status words
  // and the adjacency's entry counts
  const AdjLayout AL = adj_layout(B, Q, P, K);
  const int64_t fill_off = AL.fill < AL.total ? (int64_t)(AL.fill - AL.cursor) / 4 : 0;
  int rc;
  {
    NvtxRange r("knnag:pack_points");
    rc = launch_pack_points(p, sigma, R, B, P, dtype, rec, st, reinterpret_cast<int*>(ws + L.status), 2, adj_count, fill_off);
  }
  if (rc) return rc;
  return forward_exact_all<T>(q, rec, f, B, Q, P, F, K, f_out, w_out, dists, idxs, adj_count, st);
}

int forward_impl(const void* q, const void* p, const void* f, const void* sigma, const void* R, int B, int Q,
                 int P, int F, int K, int dtype, void* f_out, void* w_out, void* dists, int64_t* idxs,
                 void* points, void* workspace, size_t workspace_bytes, cudaStream_t st, void* adjacency) {
  NvtxRange range("knnag:forward");
  int* adj_count = adjacency ? reinterpret_cast<int*>(static_cast<char*>(adjacency) + adj_layout(B, Q, P, K).cursor)
                             : nullptr;
  char* ws = static_cast<char*>(workspace);
  if (dtype == KNNAG_F64)
    return forward_t<double>((const double*)q, (const double*)p, (const double*)f, (const double*)sigma,
                             (const double*)R, B, Q, P, F, K, dtype, (double*)f_out, (double*)w_out, (double*)dists,
                             idxs, points, ws, workspace_bytes, adj_count, st);
  return forward_t<float>((const float*)q, (const float*)p, (const float*)f, (const float*)sigma, (const float*)R, B,
                          Q, P, F, K, dtype, (float*)f_out, (float*)w_out, (float*)dists, idxs, points, ws,
                          workspace_bytes, adj_count, st);
}

RaggedLayout ragged_layout(int cap_segs, int64_t cap_q) {
  RaggedLayout L{};
  L.cap_cells = cap_q + 8 * (int64_t)cap_segs;
  size_t off = 0;
  L.status = off;
  off += 256;
  L.flag_list = off;
  off += align256((size_t)cap_q * 4);
  L.perm_q = off;
  off += align256((size_t)cap_q * 4);
  L.cell_count = off;
  off += align256((size_t)L.cap_cells * 4);
  L.cell_offset = off;
  off += align256(((size_t)L.cap_cells + 1) * 4);
  L.total = off;
  return L;
}

// Ragged forward: validate the table, sort every segment's queries, one
// persistent search launch over all segments with K <= 32, exact replay of
// the flagged queries, and the exact kernel for segments with K > 32.
int ragged_forward_impl(const char* cs, const void* segs, const float* q, const float* f, int F, int cap_segs,
                        int64_t cap_q, int64_t cap_e, int max_k, int ntile_cap, int splits, float* f_out, float* w_out,
                        float* dists, int64_t* idxs, void* workspace, cudaStream_t st) {
  NvtxRange range("knnag:ragged_forward");
  const RaggedLayout L = ragged_layout(cap_segs, cap_q);
  char* ws = static_cast<char*>(workspace);
  int* status = reinterpret_cast<int*>(ws + L.status);
  int* flag_count = status + 1;
  int* item_counter = status + 2;
  int* flag_list = reinterpret_cast<int*>(ws + L.flag_list);
  int* perm_q = reinterpret_cast<int*>(ws + L.perm_q);
  const int G = splits;
  const int qpc = search_qpc(G);
  if (cudaMemsetAsync(status, 0, 4 * sizeof(int), st) != cudaSuccess) return KNNAG_ERR_CUDA;
  int rc = launch_validate_segments(cs, segs, cap_segs, cap_q, cap_e, max_k, ntile_cap, qpc, status, st);
  if (rc) return rc;
  rc = launch_query_order(q, cs, segs, cap_segs, cap_q, (int)L.cap_cells, reinterpret_cast<int*>(ws + L.cell_count),
                          reinterpret_cast<int*>(ws + L.cell_offset), perm_q, status, st);
  if (rc) return rc;
  const int ks = max_k < 32 ? max_k : 32;
  if (ntile_cap > kSearchMaxTiles) return KNNAG_ERR_TOO_LARGE;
  WarpSearchParams<float> wp{};
  wp.q = q;
  wp.perm_q = perm_q;
  wp.f = f;
  wp.F = F;
  wp.K = ks;
  wp.ntile = ntile_cap;
  wp.vec = F < (1 << 28) && (F % 4 == 0) && ((uintptr_t)f % 16 == 0) && ((uintptr_t)f_out % 16 == 0);
  wp.f_out = f_out;
  wp.w_out = w_out;
  wp.dists = dists;
  wp.idxs = idxs;
  wp.status = status;
  wp.flag_count = flag_count;
  wp.flag_list = flag_list;
  wp.cs = cs;
  wp.segs = segs;
  wp.item_counter = item_counter;
  const int64_t cap_items = cap_q / qpc + cap_segs;
  rc = launch_search_warp_ragged(wp, G, cap_items, st);
  if (rc) return rc;
  ExactParams<float> e{};
  e.q = q;
  e.f = f;
  e.B = 1;
  e.Q = (int)(cap_q < (1 << 30) ? cap_q : (1 << 30));
  e.F = F;
  e.K = ks;
  e.list = flag_list;
  e.list_count = flag_count;
  e.f_out = f_out;
  e.w_out = w_out;
  e.dists = dists;
  e.idxs = idxs;
  e.cs = cs;
  e.segs = segs;
  e.status = status;
  rc = launch_replay_list<float>(e, ntile_cap * kTilePoints, st);
  if (rc || max_k <= 32) return rc;
  e.K = max_k;
  return launch_exact<float>(e, st);
}

}  // namespace knnag
