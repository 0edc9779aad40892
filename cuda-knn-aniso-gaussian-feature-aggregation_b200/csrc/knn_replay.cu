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
// the cluster's first CTA, whose first warp runs the exact rules over them, 32
// at a time where no keys are equal (add_batch), else one by one (add).
// The first ranges, kept whole, are 512 points in all; the next are 16 times
// as long, then as long as the kept lists hold: after each the maximum is lower.
//
// What bounds it: the first warp's serial work (about 12 batches of 3000
// cycles and 20 single points of 400 at P = 65536, K = 32: half the time) and
// three or four rounds of dependent loads and cluster barriers.  One CTA per
// query with one warp scanning every key took 148 us there and 217 us at
// P = 131072, K = 16 (a handful of flagged queries each, side by side);
// clusters with every point taken singly 77 and 71; in batches 60 and 62; with
// the first ranges 512 points instead of 4096 and growing 16 times 52 and 55
// (8 times: 58 and 62, 4 times: 60 and 66).  The loops over batches are not
// unrolled further: a lone warp waits for instructions (unrolled four times
// as far, the same batches take 66 and 69 us).
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
// Points of the first ranges per warp of one CTA, kept whole (at least
// kWarpSearchMaxK in all); the next ranges are this much longer each, up to:
constexpr int kReplayFirst = 32, kReplayGrowth = 16;
static_assert(kReplayFirst * kReplayWarps >= kWarpSearchMaxK, "the first ranges fill MinK's slots");
template <typename T>
constexpr int kReplayRange = sizeof(T) == 4 ? 512 : 256;
constexpr int kReplayMerged = 2048; // kept points merged at a time (the first ranges fit)

// Points per lane whose records are loaded together.
constexpr int kInFlight = 4;

template <typename T>
struct Kept {
  T key;
  int idx;
};

// MinK's full list (csrc/mink.cuh:60-81) in eviction order: position m = lane +
// 32 h in lane's register h holds a slot's key, ascending, of equal keys the
// higher slot first, so the last position is the slot that MinK's next point
// replaces (the first one with the largest key).  One exception keeps that
// order: a point that no other key exceeds stays the one to be replaced, also
// beside equal keys in lower slots; it is put last.  NaN slots are never
// replaced and take no position; a NaN in slot 0 is MinK's maximum for good and
// lets nothing in.  Which point a slot holds is in shared memory.
template <typename T, int V>
struct MinK {
  T key[V];
  int slot[V];
  int last;         // last position
  T max_key, next;  // keys of it and of the position before
  int max_slot;

  __device__ __forceinline__ T key_at(int m) const {
    T v = key[0];
    if constexpr (V > 1) {
#pragma unroll
      for (int h = 1; h < V; ++h)
        if (m >> 5 == h) v = key[h];
    }
    return __shfl_sync(kFullMask, v, m & 31);
  }
  __device__ __forceinline__ int slot_at(int m) const {
    int v = slot[0];
    if constexpr (V > 1) {
#pragma unroll
      for (int h = 1; h < V; ++h)
        if (m >> 5 == h) v = slot[h];
    }
    return __shfl_sync(kFullMask, v, m & 31);
  }

  // From points 0..K-1 in slots 0..K-1; pos_key and pos_slot are scratch.
  __device__ __forceinline__ void start(const T* slot_key, T* pos_key, int* pos_slot, int K, int lane) {
    int n = 0;
#pragma unroll
    for (int h = 0; h < V; ++h) {
      const int s = lane + 32 * h;
      const T ks = s < K ? slot_key[s] : T(0);
      const bool number = s < K && ks == ks;
      if (number) {
        int m = 0;
        for (int t = 0; t < K; ++t) {
          const T kt = slot_key[t];
          m += kt < ks || (kt == ks && t > s);
        }
        pos_key[m] = ks;
        pos_slot[m] = s;
      }
      n += __popc(__ballot_sync(kFullMask, number));
    }
    __syncwarp();
    last = n - 1;
#pragma unroll
    for (int h = 0; h < V; ++h) {
      const int m = lane + 32 * h;
      key[h] = m < n ? pos_key[m] : T(0);
      slot[h] = m < n ? pos_slot[m] : -1;
    }
    const T first = slot_key[0];
    if (first != first) {
      max_key = first;  // nothing is below it
      next = first;
      max_slot = 0;
      return;
    }
    top();
  }

  // max_key, next and max_slot of the positions.
  __device__ __forceinline__ void top() {
    max_key = key_at(last);
    max_slot = slot_at(last);
    next = last > 0 ? key_at(last - 1) : T(-INFINITY);
  }

  // Candidates 0..m-1 (a lane each, in index order; no NaN) at once, the same
  // as add() for each in turn that is below max_key by then; false, and
  // nothing done, if a candidate's key equals another's or a position's: only
  // then do the slots decide what is replaced.  Without such ties MinK keeps the
  // last + 1 smallest keys of positions and candidates, so a candidate's rank
  // among the positions and the candidates up to some point says whether MinK
  // holds it then.  The candidate that lifts a rank past the last position
  // replaces the one with that rank; the others that are taken replace
  // positions from the last one down.
  __device__ __forceinline__ bool add_batch(T c, int i, int m, T* pos_key, int* pos_slot, int* slot_idx, int lane) {
    const int n = last + 1;
#pragma unroll
    for (int h = 0; h < V; ++h)
      if (lane + 32 * h < n) {
        pos_key[lane + 32 * h] = key[h];
        pos_slot[lane + 32 * h] = slot[h];
      }
    __syncwarp();
    const bool live = lane < m;
    if (!live) c = T(INFINITY);  // above every candidate and position: changes nothing
    int rank = 0;
    bool tie = false;
#pragma unroll 8
    for (int t = 0; t < n; ++t) {
      const T v = pos_key[t];
      rank += v < c;
      tie = tie || v == c;
    }
    bool taken = false;
    int by = -1;       // the candidate this one replaces
    int up[V] = {};    // candidates below each position
#pragma unroll 4
    for (int u = 0; u < 32; ++u) {
      const T cu = __shfl_sync(kFullMask, c, u);
      if (lane == u) taken = rank < n;
      tie = tie || (cu == c && lane != u);
      const bool less = cu < c;
      rank += less;
      const unsigned out = __ballot_sync(kFullMask, less && rank == n && lane < u);
      if (lane == u) by = __ffs(out) - 1;
#pragma unroll
      for (int h = 0; h < V; ++h) up[h] += cu < key[h];
    }
    if (__any_sync(kFullMask, live && tie)) return false;
    // the slots: of the position replaced, or of the candidate replaced
    const unsigned of_list = __ballot_sync(kFullMask, live && taken && by < 0);
    int s = -1, root = by < 0 ? lane : by;
    if (live && taken && by < 0) s = pos_slot[last - __popc(of_list & ((1u << lane) - 1u))];
#pragma unroll 1
    for (int r = 0; r < 5; ++r) root = __shfl_sync(kFullMask, root, root);
    s = __shfl_sync(kFullMask, s, root);
    __syncwarp();
    if (live && rank < n) {
      pos_key[rank] = c;
      pos_slot[rank] = s;
      slot_idx[s] = i;
    }
#pragma unroll
    for (int h = 0; h < V; ++h) {
      const int t = lane + 32 * h;
      if (t < n && t + up[h] < n) {
        pos_key[t + up[h]] = key[h];
        pos_slot[t + up[h]] = slot[h];
      }
    }
    __syncwarp();
#pragma unroll
    for (int h = 0; h < V; ++h) {
      const int t = lane + 32 * h;
      if (t < n) {
        key[h] = pos_key[t];
        slot[h] = pos_slot[t];
      }
    }
    __syncwarp();
    top();
    return true;
  }

  // One point below max_key (uniform arguments).  On the way from one point to
  // the next are only max_key's update and the caller's search for that point.
  __device__ __forceinline__ void add(T k, int i, int* slot_idx, int lane) {
    const int s = max_slot;
    if (lane == 0) slot_idx[s] = i;
    if (!(k < next)) {  // none above it: it takes the last position
#pragma unroll
      for (int h = 0; h < V; ++h)
        if (lane + 32 * h == last) key[h] = k;
      max_key = k;
      return;
    }
    max_key = next;
    // those above it move up a position, over the last one
    T uk[V];
    int us[V];
#pragma unroll
    for (int h = 0; h < V; ++h) {
      uk[h] = __shfl_up_sync(kFullMask, key[h], 1);
      us[h] = __shfl_up_sync(kFullMask, slot[h], 1);
      if (h > 0) {
        const T k31 = __shfl_sync(kFullMask, key[h > 0 ? h - 1 : 0], 31);
        const int s31 = __shfl_sync(kFullMask, slot[h > 0 ? h - 1 : 0], 31);
        if (lane == 0) {
          uk[h] = k31;
          us[h] = s31;
        }
      }
    }
#pragma unroll
    for (int h = 0; h < V; ++h) {
      const int m = lane + 32 * h;
      const bool below = key[h] < k || (key[h] == k && slot[h] > s);
      const bool left_below = m == 0 || uk[h] < k || (uk[h] == k && us[h] > s);
      if (m <= last && !below) {
        key[h] = left_below ? k : uk[h];
        slot[h] = left_below ? s : us[h];
      }
    }
    max_slot = slot_at(last);
    next = key_at(last - 1);  // last > 0: next was a key
  }
};

// Shared memory: the warps' kept points, the merged list, slots for the sort
// and the epilogue.
template <typename T, int V>
struct ReplayShared {
  Kept<T> kept[kReplayWarps][kReplayRange<T>];
  Kept<T> merged[kReplayMerged];
  T slot_key[32 * V], pos_key[32 * V];
  int slot_idx[32 * V], pos_slot[32 * V];
  Kept<T> pending[64];           // kept points below MinK's maximum, not acted on yet
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
    MinK<T, V> mk;  // the first CTA's first warp's
    T limit = T(INFINITY);
    for (int c0 = 0, len = kReplayFirst / ranks; c0 < P;
         c0 += ranks * kReplayWarps * len, len = min(len * kReplayGrowth, kReplayRange<T>)) {
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
          key[u] = key_rec<T>(qx, qy, qz, recb + (int64_t)min(i, r1 - 1) * kRecLen);
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
        int i0 = 0;  // of the first ranges' points
        if (c0 == 0) {  // points 0..K-1 fill the slots (the first ranges hold them, and are merged)
          for (int t = lane; t < K; t += 32) {
            sm.slot_key[t] = sm.merged[t].key;
            sm.slot_idx[t] = sm.merged[t].idx;
          }
          __syncwarp();
          mk.start(sm.slot_key, sm.pos_key, sm.pos_slot, K, lane);
          i0 = K;
        }
        int waiting = 0;
        auto act = [&](int m) {  // on the first m of the pending
          const Kept<T> x = sm.pending[lane];
          if (mk.add_batch(x.key, x.idx, m, sm.pos_key, sm.pos_slot, sm.slot_idx, lane)) return;
          unsigned todo = m < 32 ? (1u << m) - 1u : kFullMask;
          while (true) {
            todo &= __ballot_sync(kFullMask, x.key < mk.max_key);  // only those act, and it only falls
            if (!todo) break;
            const int l = __ffs(todo) - 1;
            todo &= todo - 1;
            mk.add(__shfl_sync(kFullMask, x.key, l), __shfl_sync(kFullMask, x.idx, l), sm.slot_idx, lane);
          }
        };
        auto run = [&](const Kept<T>* list, int i0, int m) {
          Kept<T> next = i0 + lane < m ? list[i0 + lane] : Kept<T>{T(0), 0};
#pragma unroll 1
          for (; i0 < m; i0 += 32) {
            const Kept<T> x = next;
            const bool below = i0 + lane < m && x.key < mk.max_key;
            if (i0 + 32 + lane < m) next = list[i0 + 32 + lane];
            const unsigned b = __ballot_sync(kFullMask, below);
            if (!b) continue;
            if (below) sm.pending[waiting + __popc(b & ((1u << lane) - 1u))] = x;
            waiting += __popc(b);
            __syncwarp();
            if (waiting >= 32) {
              act(32);
              waiting -= 32;
              __syncwarp();
              if (lane < waiting) sm.pending[lane] = sm.pending[32 + lane];
              __syncwarp();
            }
          }
        };
        if (merge) {
          run(sm.merged, i0, total);
        } else {
          for (int s = 0; s < ranks * kReplayWarps; ++s) {
            const ReplayShared<T, V>* from = cluster.map_shared_rank(&sm, s / kReplayWarps);
            run(from->kept[s % kReplayWarps], 0, sm.count[s]);
          }
        }
        if (waiting) act(waiting);
        // a NaN maximum lets nothing in, ever
        if (lane == 0) sm.limit = mk.max_key == mk.max_key ? mk.max_key : T(-INFINITY);
      }
      cluster.sync();
      limit = sm0.limit;
    }
    // ---- sort (csrc/mink.cuh:99-112: a bubble sort with a strict '<' swap,
    // without NaN the stable order by key) and outputs
    if (rank == 0) {
      if (warp == 0) {
        bool nan = false;
        T key[V];
        int idx[V];
#pragma unroll
        for (int h = 0; h < V; ++h)
          if (lane + 32 * h <= mk.last) sm.slot_key[mk.slot[h]] = mk.key[h];
        __syncwarp();
#pragma unroll
        for (int h = 0; h < V; ++h) {
          const int s = lane + 32 * h;
          key[h] = s < K ? sm.slot_key[s] : T(0);
          idx[h] = s < K ? sm.slot_idx[s] : 0;
          nan = nan || key[h] != key[h];
        }
        if (!__any_sync(kFullMask, nan)) {
          int place[V];
#pragma unroll
          for (int h = 0; h < V; ++h) {
            place[h] = 0;
            for (int t = 0; t < K; ++t) {
              const T kt = sm.slot_key[t];
              place[h] += kt < key[h] || (kt == key[h] && t < lane + 32 * h);
            }
          }
          __syncwarp();
#pragma unroll
          for (int h = 0; h < V; ++h)
            if (lane + 32 * h < K) {
              sm.slot_key[place[h]] = key[h];
              sm.slot_idx[place[h]] = idx[h];
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
