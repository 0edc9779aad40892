// Exact replay of the reference's MinK selection (csrc/mink.cuh:60-112) for the
// queries a search flagged: tied keys, or a NaN among the first K points.
//
// MinK reads a query's keys in index order and its slots remember that order,
// so the scan itself is serial; but it only ever acts on a point whose key is
// below the K-th smallest of the points before it, about K (1 + ln(P / K)) of
// them.  A cluster of CTAs finds them in parallel: every warp takes a range of
// consecutive points and keeps those below MinK's maximum after the ranges
// already replayed (an upper bound of what it will be at any later point, so
// no point MinK would take is lost) and points 0..K-1, which MinK takes
// whatever their key is.  The kept points of all warps go, in index order, to
// the cluster's first CTA, whose first warp runs the exact rules over them.
// The first ranges, kept whole, are short (32 points per warp): after them the
// maximum is low and the long ranges keep about one point in a hundred.
//
// What bounds it: the serial part, 150 to 300 accepted points of a few dozen
// dependent instructions each.  One CTA per query with one warp scanning every
// key took 148 us at P = 65536, K = 32 and 217 us at P = 131072, K = 16 (a
// handful of flagged queries each, side by side); the clusters take 77 and
// 71 us, about 0.2 us per accepted point.
#include <cooperative_groups.h>
#include <math.h>

#include "knn_common.cuh"
#include "knn_internal.h"

namespace knnag {

namespace {

namespace cg = cooperative_groups;

constexpr unsigned kFullMask = 0xffffffffu;
constexpr int kReplayWarps = 16;
constexpr int kReplayMaxRanks = 8;  // CTAs per cluster
constexpr int kReplayFirst = 32;    // points per warp of the first ranges
template <typename T>
constexpr int kReplayRange = sizeof(T) == 4 ? 512 : 256;  // of the others
constexpr int kReplayMerged = 8192; // kept points merged at a time (8 CTAs' first ranges fit)

// Points per lane whose records are loaded together.
constexpr int kInFlight = 4;

template <typename T>
struct Kept {
  T key;
  int idx;
};

// Largest value over the warp (no NaN), by integer reductions of
// order-preserving bits.
__device__ __forceinline__ float warp_largest(float v) {
  const int b = __float_as_int(v);
  const int m = __reduce_max_sync(kFullMask, b ^ ((b >> 31) & 0x7fffffff));
  return __int_as_float(m ^ ((m >> 31) & 0x7fffffff));
}
__device__ __forceinline__ double warp_largest(double v) {
  const long long b = __double_as_longlong(v);
  const long long o = b ^ ((b >> 63) & 0x7fffffffffffffffLL);
  const int hi = (int)(o >> 32);
  const int mh = __reduce_max_sync(kFullMask, hi);
  const unsigned lo = hi == mh ? (unsigned)o : 0u;
  const unsigned ml = __reduce_max_sync(kFullMask, lo);
  const long long m = ((long long)mh << 32) | ml;
  return __longlong_as_double(m ^ ((m >> 63) & 0x7fffffffffffffffLL));
}

// MinK's state: slot s = lane + 32 h in lane's register h.
template <typename T, int V>
struct MinK {
  T key[V];
  int idx[V];
  T max_key;
  int max_slot, size;

  __device__ __forceinline__ void put(int s, T k, int i, int lane) {
#pragma unroll
    for (int h = 0; h < V; ++h)
      if (s == lane + 32 * h) {
        key[h] = k;
        idx[h] = i;
      }
  }
  // One point (uniform arguments), the rules of csrc/mink.cuh:60-81.
  __device__ __forceinline__ void add(T k, int i, int K, int lane) {
    if (size < K) {
      put(size, k, i, lane);
      if (size == 0 || k > max_key) {
        max_key = k;
        max_slot = size;
      }
      ++size;
    } else if (k < max_key) {
      put(max_slot, k, i, lane);
      // the first slot with the largest key strictly above k; the written one
      // stays the maximum when there is none
      T v = T(-INFINITY);
#pragma unroll
      for (int h = 0; h < V; ++h)
        if (lane + 32 * h < K && key[h] > k) v = fmax(v, key[h]);
      const T m = warp_largest(v);
      max_key = k;
      if (m > k) {
        max_key = m;
#pragma unroll
        for (int h = V - 1; h >= 0; --h) {
          const unsigned b = __ballot_sync(kFullMask, lane + 32 * h < K && key[h] == m);
          if (b) max_slot = 32 * h + __ffs(b) - 1;
        }
      }
    }
  }
};

// Shared memory: the warps' kept points, the merged list, slots for the sort
// and the epilogue.
template <typename T, int V>
struct ReplayShared {
  Kept<T> kept[kReplayWarps][kReplayRange<T>];
  Kept<T> merged[kReplayMerged];
  T slot_key[32 * V];
  int slot_idx[32 * V];
  int count[kReplayMaxRanks * kReplayWarps];  // kept points of all the cluster's warps
  T limit;                       // MinK's maximum once it is full, else +inf
};

template <typename T, int V>
__global__ void __launch_bounds__(32 * kReplayWarps) replay_list_kernel(ExactParams<T> a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  ReplayShared<T, V>& sm = *reinterpret_cast<ReplayShared<T, V>*>(smem_raw);
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = (int)cluster.block_rank(), ranks = (int)cluster.num_blocks();
  ReplayShared<T, V>& sm0 = *cluster.map_shared_rank(&sm, 0);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const SegHeader* sh = static_cast<const SegHeader*>(a.segs);
  if (sh && *a.status) return;  // nothing writes it while this kernel runs
  const int64_t n_items = *a.list_count;
  const int64_t rows = sh ? sh->total_q : (int64_t)a.B * a.Q;
  for (int64_t item = blockIdx.x / ranks; item < n_items; item += gridDim.x / ranks) {
    const int64_t bq = a.list[item];
    if (bq < 0 || bq >= rows) continue;  // the search lists its own rows: never taken
    // the query's sizes, first entry, records and features
    int K, P;
    int64_t e0, b = 0;
    const T* recb;
    const T* fb;
    if (sh) {
      const SegDesc* sd = seg_descs(a.segs);
      const SegDesc g = sd[seg_of_row(sd, sh->nseg, bq)];
      const CloudDesc c = cloud_descs(a.cs)[g.cloud];
      K = g.K;
      P = c.P;
      e0 = g.e_off + (bq - g.q_off) * K;
      recb = reinterpret_cast<const T*>(a.cs + reinterpret_cast<const CloudSetHeader*>(a.cs)->rec_off) +
             c.p_off * kRecLen;
      fb = a.f + c.p_off * a.F;
      if (K > a.K || K > P) continue;  // the host checked the table; never reached
    } else {
      b = bq / a.Q;
      K = a.K;
      P = a.P;
      e0 = bq * K;
      recb = a.rec + b * (int64_t)P * kRecLen;
      fb = a.f + b * (int64_t)P * a.F;
    }
    const T qx = a.q[bq * 3 + 0], qy = a.q[bq * 3 + 1], qz = a.q[bq * 3 + 2];
    MinK<T, V> mk;
    mk.size = 0;
    mk.max_slot = 0;
    mk.max_key = T(0);
#pragma unroll
    for (int h = 0; h < V; ++h) {
      mk.key[h] = T(0);
      mk.idx[h] = -1;
    }
    T limit = T(INFINITY);
    for (int c0 = 0, len = kReplayFirst; c0 < P; c0 += ranks * kReplayWarps * len, len = kReplayRange<T>) {
      // ---- this warp's range
      const int r0 = c0 + (rank * kReplayWarps + warp) * len;
      const int r1 = min(P, r0 + len);
      Kept<T>* kept = sm.kept[warp];
      int n = 0;
      for (int i0 = r0; i0 < r1; i0 += 32 * kInFlight) {
        // several points per lane, their records in flight together
        T key[kInFlight];
        bool keep[kInFlight];
#pragma unroll
        for (int u = 0; u < kInFlight; ++u) {
          const int i = i0 + 32 * u + lane;
          keep[u] = i < r1;
          key[u] = key_rec<T>(qx, qy, qz, recb + (int64_t)min(i, P - 1) * kRecLen);
          keep[u] = keep[u] && (i < K || key[u] < limit);
        }
#pragma unroll
        for (int u = 0; u < kInFlight; ++u) {
          const unsigned m = __ballot_sync(kFullMask, keep[u]);
          if (keep[u]) kept[n + __popc(m & ((1u << lane) - 1u))] = Kept<T>{key[u], i0 + 32 * u + lane};
          n += __popc(m);
        }
      }
      if (lane < ranks) cluster.map_shared_rank(&sm, lane)->count[rank * kReplayWarps + warp] = n;
      cluster.sync();
      // ---- kept points to the first CTA, in index order
      int before = 0, total = 0;  // kept points of the warps before this one, of all
      for (int s0 = 0; s0 < ranks * kReplayWarps; s0 += 32) {
        const int s = s0 + lane, c = s < ranks * kReplayWarps ? sm.count[s] : 0;
        total += __reduce_add_sync(kFullMask, c);
        before += __reduce_add_sync(kFullMask, s < rank * kReplayWarps + warp ? c : 0);
      }
      const bool merge = total <= kReplayMerged;
      if (merge)
        for (int i = lane; i < n; i += 32) sm0.merged[before + i] = kept[i];
      cluster.sync();
      // ---- the exact rules over them
      if (rank == 0 && warp == 0) {
        auto run = [&](const Kept<T>* list, int m) {
          Kept<T> next = lane < m ? list[lane] : Kept<T>{T(0), 0};
          for (int i0 = 0; i0 < m; i0 += 32) {
            const Kept<T> x = next;
            if (i0 + 32 + lane < m) next = list[i0 + 32 + lane];
            unsigned todo = i0 + 32 <= m ? kFullMask : (1u << (m - i0)) - 1u;
            while (todo) {
              if (mk.size >= K) {  // only keys below the maximum act, and it only falls
                todo &= __ballot_sync(kFullMask, x.key < mk.max_key);
                if (!todo) break;
              }
              const int l = __ffs(todo) - 1;
              todo &= todo - 1;
              mk.add(__shfl_sync(kFullMask, x.key, l), __shfl_sync(kFullMask, x.idx, l), K, lane);
            }
          }
        };
        if (merge) {
          run(sm.merged, total);
        } else {
          for (int s = 0; s < ranks * kReplayWarps; ++s) {
            const ReplayShared<T, V>* from = cluster.map_shared_rank(&sm, s / kReplayWarps);
            run(from->kept[s % kReplayWarps], sm.count[s]);
          }
        }
        // a NaN maximum lets nothing in, ever
        if (lane == 0) sm.limit = mk.size < K ? T(INFINITY) : (mk.max_key == mk.max_key ? mk.max_key : T(-INFINITY));
      }
      cluster.sync();
      limit = sm0.limit;
    }
    // ---- sort (csrc/mink.cuh:99-112: a bubble sort with a strict '<' swap,
    // without NaN the stable order by key) and outputs
    if (rank == 0) {
      if (warp == 0) {
        bool nan = false;
#pragma unroll
        for (int h = 0; h < V; ++h) {
          const int s = lane + 32 * h;
          if (s < K) {
            sm.slot_key[s] = mk.key[h];
            sm.slot_idx[s] = mk.idx[h];
            nan = nan || mk.key[h] != mk.key[h];
          }
        }
        __syncwarp();
        if (!__any_sync(kFullMask, nan)) {
          int place[V];
#pragma unroll
          for (int h = 0; h < V; ++h) {
            place[h] = 0;
            for (int t = 0; t < K; ++t) {
              const T kt = sm.slot_key[t];
              place[h] += kt < mk.key[h] || (kt == mk.key[h] && t < lane + 32 * h);
            }
          }
          __syncwarp();
#pragma unroll
          for (int h = 0; h < V; ++h)
            if (lane + 32 * h < K) {
              sm.slot_key[place[h]] = mk.key[h];
              sm.slot_idx[place[h]] = mk.idx[h];
            }
        } else if (lane == 0) {
          bubble_sort_slots(sm.slot_key, sm.slot_idx, K);
        }
      }
      __syncthreads();
      T w = T(0);
      if (tid < K) {
        w = weight_of(sm.slot_key[tid]);
        const int idx = sm.slot_idx[tid];
        a.dists[e0 + tid] = sm.slot_key[tid];
        a.idxs[e0 + tid] = (int64_t)idx;
        a.w_out[e0 + tid] = w;
        if (a.adj_count && (unsigned)idx < (unsigned)P) atomicAdd(&a.adj_count[b * P + idx], 1);
      }
      __syncthreads();
      if (tid < K) sm.slot_key[tid] = w;
      __syncthreads();
      for (int c = tid; c < a.F; c += 32 * kReplayWarps) {
        T acc = T(0);
#pragma unroll 8
        for (int k = 0; k < K; ++k) acc = fma_rn(fb[(int64_t)sm.slot_idx[k] * a.F + c], sm.slot_key[k], acc);
        a.f_out[bq * a.F + c] = acc;
      }
      __syncthreads();
    }
    // the next query's ranges touch only this CTA's own memory until its
    // first cluster barrier
  }
  cluster.sync();  // no CTA leaves while another may still read its memory
}

template <typename T, int V>
int launch_v(const ExactParams<T>& a, int max_points, cudaStream_t st) {
  // CTAs per query: as many as have a full second range, up to 8
  int ranks = 1;
  while (ranks < kReplayMaxRanks && ranks * kReplayWarps * kReplayRange<T> < max_points) ranks *= 2;
  const size_t smem = sizeof(ReplayShared<T, V>);
  static_assert(sizeof(ReplayShared<T, V>) <= 227 * 1024, "shared memory");
  int dev = 0;
  cudaGetDevice(&dev);
  if (cudaFuncSetAttribute(replay_list_kernel<T, V>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) !=
      cudaSuccess)
    return KNNAG_ERR_CUDA;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)(num_sms(dev) / ranks * ranks));  // flagged queries are few; clusters loop over them
  cfg.blockDim = dim3(32 * kReplayWarps);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = ranks;
  attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  if (cudaLaunchKernelEx(&cfg, replay_list_kernel<T, V>, a) != cudaSuccess) return KNNAG_ERR_CUDA;
  note_launches(1);
  return cudaGetLastError() == cudaSuccess ? KNNAG_OK : KNNAG_ERR_CUDA;
}

}  // namespace

template <typename T>
int launch_replay_list(const ExactParams<T>& a, int max_points, cudaStream_t st) {
  if (a.K <= 32) return launch_v<T, 1>(a, max_points, st);
  if (a.K <= 64) return launch_v<T, 2>(a, max_points, st);
  if (a.K <= kWarpSearchMaxK) return launch_v<T, 4>(a, max_points, st);
  return KNNAG_ERR_ARG;
}
template int launch_replay_list<float>(const ExactParams<float>&, int, cudaStream_t);
template int launch_replay_list<double>(const ExactParams<double>&, int, cudaStream_t);

}  // namespace knnag
