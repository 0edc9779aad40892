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
// P = 131072, K = 16 (a handful of flagged queries each, side by side; many are
// served by replay_passes);
// clusters with every point taken singly 77 and 71; in batches 60 and 62; with
// the first ranges 512 points instead of 4096 and growing 16 times 52 and 55
// (8 times: 58 and 62, 4 times: 60 and 66).  The loops over batches are not
// unrolled further: a lone warp waits for instructions (unrolled four times
// as far, the same batches take 66 and 69 us).
#include <cooperative_groups.h>
#include <math.h>

#include <algorithm>
#include <atomic>

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

// A query's slots, the positions' scratch and the points below MinK's maximum
// that it has not acted on yet.
template <typename T, int V>
struct Scratch {
  T slot_key[32 * V], pos_key[32 * V];
  int slot_idx[32 * V], pos_slot[32 * V];
  Kept<T> pending[64];
};

// The exact rules over the first m pending points; whether they went as a batch.
template <typename T, int V>
__device__ __forceinline__ bool act(MinK<T, V>& mk, Scratch<T, V>& s, int m, bool batch, int lane) {
  const Kept<T> x = s.pending[lane];
  if (batch && mk.add_batch(x.key, x.idx, m, s.pos_key, s.pos_slot, s.slot_idx, lane)) return true;
  unsigned todo = m < 32 ? (1u << m) - 1u : kFullMask;
  while (true) {
    todo &= __ballot_sync(kFullMask, lane < m && x.key < mk.max_key);  // only those act, and it only falls
    if (!todo) break;
    const int l = __ffs(todo) - 1;
    todo &= todo - 1;
    mk.add(__shfl_sync(kFullMask, x.key, l), __shfl_sync(kFullMask, x.idx, l), s.slot_idx, lane);
  }
  return false;
}

// MinK's final sort (csrc/mink.cuh:99-112: a bubble sort with a strict '<' swap,
// without NaN the stable order by key) of a warp's query into slot_key, slot_idx.
template <typename T, int V>
__device__ __forceinline__ void sort_slots(const MinK<T, V>& mk, Scratch<T, V>& s, int K, int lane) {
  bool nan = false;
  T key[V];
  int idx[V];
#pragma unroll
  for (int h = 0; h < V; ++h)
    if (lane + 32 * h <= mk.last) s.slot_key[mk.slot[h]] = mk.key[h];
  __syncwarp();
#pragma unroll
  for (int h = 0; h < V; ++h) {
    const int t = lane + 32 * h;
    key[h] = t < K ? s.slot_key[t] : T(0);
    idx[h] = t < K ? s.slot_idx[t] : 0;
    nan = nan || key[h] != key[h];
  }
  if (!__any_sync(kFullMask, nan)) {
    int place[V];
#pragma unroll
    for (int h = 0; h < V; ++h) {
      place[h] = 0;
      for (int t = 0; t < K; ++t) {
        const T kt = s.slot_key[t];
        place[h] += kt < key[h] || (kt == key[h] && t < lane + 32 * h);
      }
    }
    __syncwarp();
#pragma unroll
    for (int h = 0; h < V; ++h)
      if (lane + 32 * h < K) {
        s.slot_key[place[h]] = key[h];
        s.slot_idx[place[h]] = idx[h];
      }
  } else if (lane == 0) {
    bubble_sort_slots(s.slot_key, s.slot_idx, K);
  }
  __syncwarp();
}

// A flagged query: its row, sizes, first entry, records and features.
template <typename T>
struct FlaggedQuery {
  int64_t bq, e0, row0;  // row0: first point row of its batch element (uniform calls)
  int K, P, cloud;
  const T* rec;
  const T* f;
};
template <typename T>
__device__ __forceinline__ bool flagged_query(const ExactParams<T>& a, int row, FlaggedQuery<T>& x) {
  const SegHeader* sh = static_cast<const SegHeader*>(a.segs);
  x.bq = row;
  if (x.bq < 0 || x.bq >= (sh ? sh->total_q : (int64_t)a.B * a.Q)) return false;  // the search lists its own rows: never taken
  if (sh) {
    const SegDesc* sd = seg_descs(a.segs);
    const SegDesc g = sd[seg_of_row(sd, sh->nseg, x.bq)];
    const CloudDesc c = cloud_descs(a.cs)[g.cloud];
    x.cloud = g.cloud;
    x.K = g.K;
    x.P = c.P;
    x.e0 = g.e_off + (x.bq - g.q_off) * x.K;
    x.row0 = 0;
    x.rec = reinterpret_cast<const T*>(a.cs + reinterpret_cast<const CloudSetHeader*>(a.cs)->rec_off) +
            c.p_off * kRecLen;
    x.f = a.f + c.p_off * a.F;
    return x.K <= a.K && x.K <= x.P;  // the host checked the table; always
  }
  x.cloud = (int)(x.bq / a.Q);
  x.K = a.K;
  x.P = a.P;
  x.e0 = x.bq * x.K;
  x.row0 = (int64_t)x.cloud * a.P;
  x.rec = a.rec + x.row0 * kRecLen;
  x.f = a.f + x.row0 * a.F;
  return true;
}

// Shared memory: the warps' kept points, the merged list, the query's scratch.
template <typename T, int V>
struct ReplayShared {
  Kept<T> kept[kReplayWarps][kReplayRange<T>];
  Kept<T> merged[kReplayMerged];
  Scratch<T, V> s;
  int count[kReplayMaxRanks * kReplayWarps];  // kept points of all the cluster's warps
  T limit;                       // MinK's maximum once it is full, else +inf
};

// ------------------------------------------------------------ many queries
//
// With more flagged queries than clusters (lattices, repeated points: often every
// query of a call), a cluster per query wastes the chip: its warps wait while one
// of them acts.  Then every warp takes a query of its own, and the sixteen of a
// CTA go through their cloud together: chunks of records, staged in shared memory
// two deep, a point per lane, MinK's rules in place.  Queries of other clouds
// among the sixteen wait for a pass of their own.
// What bounds it: instruction latency at 16 warps per SM (24 instructions per 32
// keys), and the barrier per chunk, at which fifteen warps wait for one that acts.
// A forward with every query flagged, by the kernel before the clusters (a CTA
// per query), by clusters and by passes: B = 2, Q = 12288, P = 4096, K = 16 3.2,
// 6.0 and 0.9 ms; Q = 32768, P = 131072, K = 16 33, 141 and 15 ms; Q = 16384, P =
// 65536, K = 32 10.8, 79 and 4.9 ms; FP64, Q = 4096, P = 30000, K = 16 3.6, 24 and
// 1.2 ms; 24 ragged clouds of 1000 to 20000 points, Q = 1000 each 4.0, 26 and 1.7 ms.
// Two CTAs per SM at 64 registers: 0.8, 16.5, 5.7, 1.3 and 1.6 ms, but the clusters'
// registers spill (51 -> 58 us for a handful of queries).
template <typename T, int V>
constexpr int kPassPoints = (V == 1 ? 1024 : V == 2 ? 768 : 512) * 4 / sizeof(T);
// A staged record: 16 bytes more than its length, so that eight lanes' 16-byte
// loads of consecutive records meet all banks.
template <typename T>
constexpr int kPassStride = kRecLen + 16 / sizeof(T);
constexpr int kPassBuckets = 2048;  // of rows, where the list is ordered
constexpr int kPassRows = 2048;     // most rows of a bucket, and of a CTA at a time
struct PassOrder {
  int count[kPassBuckets], start[kPassBuckets];
  long long cost[kPassBuckets];
};
template <typename T, int V>
struct PassShared {
  union {
    T rec[2][kPassPoints<T, V> * kPassStride<T>];
    PassOrder order;  // before the passes
  };
  Scratch<T, V> s[kReplayWarps];
  int cloud[kReplayWarps];
  int rows[kPassRows];  // the CTA's queries in row order, where the call has several clouds
  int wsum[kReplayWarps];
  long long wcost[kReplayWarps], total;
};

// 16 bytes from global to shared memory, completed by copy_wait (the thread's own).
__device__ __forceinline__ void copy16_async(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void copy_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// The list is in the order the search met the queries, many clouds side by side.
// To put the queries of a cloud together every CTA counts the list by buckets
// of 2^shift consecutive rows; a bucket costs its count times its cloud's points
// (and what a query takes besides).  Leaves every bucket's first place and cost
// before it, its end in `count`, and the total cost.
template <typename T, int V>
__device__ __forceinline__ void order_rows(const ExactParams<T>& a, int64_t n_items, int shift, PassShared<T, V>& sm) {
  PassOrder& o = sm.order;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  constexpr int NT = 32 * kReplayWarps, PER = kPassBuckets / NT;
  for (int b = tid; b < kPassBuckets; b += NT) o.count[b] = 0;
  __syncthreads();
  for (int64_t i = tid; i < n_items; i += NT) {
    const unsigned b = (unsigned)a.list[i] >> shift;
    if (b < kPassBuckets) atomicAdd(&o.count[b], 1);
  }
  __syncthreads();
  int n[PER], sum = 0;
  long long cost[PER], csum = 0;
#pragma unroll
  for (int u = 0; u < PER; ++u) {
    const int b = tid * PER + u;
    n[u] = o.count[b];
    int P = a.P;
    if (a.segs && n[u]) {
      const SegHeader* sh = static_cast<const SegHeader*>(a.segs);
      const SegDesc* sd = seg_descs(a.segs);
      P = cloud_descs(a.cs)[sd[seg_of_row(sd, sh->nseg, (int64_t)b << shift)].cloud].P;
    }
    cost[u] = (long long)n[u] * (P + kPassRows);
    sum += n[u];
    csum += cost[u];
  }
  int incl = sum;
  long long cincl = csum;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const int t = __shfl_up_sync(kFullMask, incl, d);
    const long long ct = __shfl_up_sync(kFullMask, cincl, d);
    if (lane >= d) {
      incl += t;
      cincl += ct;
    }
  }
  if (lane == 31) {
    sm.wsum[warp] = incl;
    sm.wcost[warp] = cincl;
  }
  __syncthreads();
  int at = incl - sum;
  long long cat = cincl - csum;
  for (int w = 0; w < warp; ++w) {
    at += sm.wsum[w];
    cat += sm.wcost[w];
  }
#pragma unroll
  for (int u = 0; u < PER; ++u) {
    const int b = tid * PER + u;
    o.start[b] = at;
    o.cost[b] = cat;
    at += n[u];
    cat += cost[u];
    o.count[b] = at;
  }
  if (tid == NT - 1) sm.total = cat;
  __syncthreads();
}

template <typename T>
__device__ __forceinline__ T staged_key(T qx, T qy, T qz, const T* rec) {
  using V16 = typename Group16<T>::type;
  T r[kRecLen];
#pragma unroll
  for (int m = 0; m < kRecLen; m += 16 / sizeof(T)) {
    const V16 v = *reinterpret_cast<const V16*>(rec + m);
    r[m] = v.x;
    r[m + 1] = v.y;
    if constexpr (sizeof(T) == 4) {
      r[m + 2] = v.z;
      r[m + 3] = v.w;
    }
  }
  return key_from_offset<T>(add_rn(qx, r[kNPX]), add_rn(qy, r[kNPY]), add_rn(qz, r[kNPZ]), r + kR00, r[kS0], r[kS1],
                            r[kS2]);
}

template <typename T, int V>
__device__ __noinline__ void replay_passes(const ExactParams<T>& a, int64_t n_items) {
  extern __shared__ __align__(16) unsigned char smem_raw[];  // not an argument: a generic pointer's loads are slower
  PassShared<T, V>& sm = *reinterpret_cast<PassShared<T, V>*>(smem_raw);
  constexpr int CH = kPassPoints<T, V>, N = 16 / sizeof(T), PARTS = kRecLen / N;  // 16-byte pieces of a record
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  Scratch<T, V>& s = sm.s[warp];
  const int64_t rows = a.segs ? static_cast<const SegHeader*>(a.segs)->total_q : (int64_t)a.B * a.Q;
  const int64_t share = (n_items + gridDim.x - 1) / gridDim.x;
  // the CTA's part of the list: [first, end) of it, or of its rows in order
  const bool ordered = (a.segs || a.B > 1) && rows < (int64_t)kPassBuckets * kPassRows;
  int64_t first = ordered ? 0 : blockIdx.x * share, end = ordered ? 0 : min(n_items, first + share);
  int shift = 0, bucket = -1, bucket_end = 0;
  while (rows >> shift >= kPassBuckets) ++shift;
  while (true) {
    if (first >= end) {
      if (!ordered || bucket >= bucket_end) break;
      order_rows(a, n_items, shift, sm);
      if (bucket < 0) {  // the CTA's buckets: those that start in its share of the cost
        const long long c0 = sm.total * blockIdx.x / gridDim.x, c1 = sm.total * (blockIdx.x + 1) / gridDim.x;
        bucket = 0;
        for (int step = kPassBuckets / 2; step > 0; step >>= 1) {
          if (sm.order.cost[bucket + step - 1] < c0) bucket += step;
          if (sm.order.cost[bucket_end + step - 1] < c1) bucket_end += step;
        }
        bucket += sm.order.cost[bucket] < c0;
        bucket_end += sm.order.cost[bucket_end] < c1;
        if (bucket >= bucket_end) break;
      }
      // the next buckets that fit, their rows in order of bucket
      const int from = bucket, start = sm.order.start[from];
      do ++bucket;
      while (bucket < bucket_end && sm.order.count[bucket] - start <= kPassRows);
      first = 0;
      end = min(sm.order.count[bucket - 1] - start, kPassRows);
      __syncthreads();  // every thread has read the starts
      for (int64_t i = tid; i < n_items; i += 32 * kReplayWarps) {
        const int row = a.list[i], b = (int)((unsigned)row >> shift);
        if (b >= from && b < bucket) {
          const int at = atomicAdd(&sm.order.start[b], 1) - start;
          if (at < kPassRows) sm.rows[at] = row;  // a row is listed once: always
        }
      }
      __syncthreads();
      continue;
    }
    const int per = (int)min((int64_t)kReplayWarps, end - first);
    FlaggedQuery<T> x{};
    const bool mine = warp < per && flagged_query(a, ordered ? sm.rows[first + warp] : a.list[first + warp], x);
    first += per;
    if (lane == 0) sm.cloud[warp] = mine ? x.cloud : -1;
    __syncthreads();
    const T qx = mine ? a.q[x.bq * 3 + 0] : T(0), qy = mine ? a.q[x.bq * 3 + 1] : T(0),
            qz = mine ? a.q[x.bq * 3 + 2] : T(0);
    for (int w0 = 0; w0 < kReplayWarps; ++w0) {  // a pass per cloud
      const int cloud = sm.cloud[w0];
      bool again = cloud < 0;
      for (int w = 0; w < w0; ++w) again = again || sm.cloud[w] == cloud;
      if (again) continue;
      int P = a.P;
      const T* rec = a.rec + (int64_t)cloud * P * kRecLen;
      if (a.segs) {
        const CloudDesc c = cloud_descs(a.cs)[cloud];
        P = c.P;
        rec = reinterpret_cast<const T*>(a.cs + reinterpret_cast<const CloudSetHeader*>(a.cs)->rec_off) +
              c.p_off * kRecLen;
      }
      const bool takes = mine && x.cloud == cloud;
      MinK<T, V> mk;
      int waiting = 0, failed = 0;
      auto load = [&](int c0, int buf) {  // points [c0, c0 + CH), asynchronously
        const int n = min(CH, P - c0) * PARTS;
        for (int j = tid; j < n; j += 32 * kReplayWarps)
          copy16_async(&sm.rec[buf][j / PARTS * kPassStride<T> + j % PARTS * N], rec + ((int64_t)c0 * PARTS + j) * N);
      };
      load(0, 0);
      copy_wait();
      __syncthreads();
      for (int c0 = 0, buf = 0; c0 < P; c0 += CH, buf ^= 1) {
        if (c0 + CH < P) load(c0 + CH, buf ^ 1);
        if (takes) {
          const T* staged = sm.rec[buf];
          const int n = min(CH, P - c0);
          int i0 = 0, from = 0;  // points before `from` fill the slots
          if (c0 == 0) {
            from = i0 = x.K;
            for (int t = lane; t < x.K; t += 32) {
              s.slot_key[t] = staged_key<T>(qx, qy, qz, staged + t * kPassStride<T>);
              s.slot_idx[t] = t;
            }
            __syncwarp();
            mk.start(s.slot_key, s.pos_key, s.pos_slot, x.K, lane);
          }
          constexpr int U = sizeof(T) == 4 ? 4 : 2;  // keys in flight
          static_assert(CH % (32 * U) == 0, "whole turns");
          i0 &= ~(32 * U - 1);
          for (; i0 < n; i0 += 32 * U) {
            T key[U];
            bool any = false;  // points before `from` and past n are left out below
#pragma unroll
            for (int u = 0; u < U; ++u) {
              key[u] = staged_key<T>(qx, qy, qz, staged + (i0 + 32 * u + lane) * kPassStride<T>);
              any = any || key[u] < mk.max_key;
            }
            if (!__any_sync(kFullMask, any)) continue;
#pragma unroll 1
            for (int u = 0; u < U; ++u) {
              T ku = key[0];
#pragma unroll
              for (int v = 1; v < U; ++v)
                if (u == v) ku = key[v];
              const int i = i0 + 32 * u + lane;
              const bool below = i >= from && i < n && ku < mk.max_key;
              const unsigned b = __ballot_sync(kFullMask, below);
              if (!b) continue;
              if (below) s.pending[waiting + __popc(b & ((1u << lane) - 1u))] = Kept<T>{ku, c0 + i};
              waiting += __popc(b);
              __syncwarp();
              if (waiting >= 32) {
                failed = act(mk, s, 32, failed < 2, lane) ? 0 : failed + 1;
                waiting -= 32;
                __syncwarp();
                if (lane < waiting) s.pending[lane] = s.pending[32 + lane];
                __syncwarp();
              }
            }
          }
        }
        copy_wait();
        __syncthreads();
      }
      if (takes) {
        if (waiting) act(mk, s, waiting, failed < 2, lane);
        __syncwarp();
        sort_slots(mk, s, x.K, lane);
        for (int e = lane; e < x.K; e += 32) {
          const T key = s.slot_key[e], w = weight_of(key);
          const int idx = s.slot_idx[e];
          a.dists[x.e0 + e] = key;
          a.idxs[x.e0 + e] = (int64_t)idx;
          a.w_out[x.e0 + e] = w;
          if (a.adj_count && (unsigned)idx < (unsigned)P) atomicAdd(&a.adj_count[x.row0 + idx], 1);
          s.slot_key[e] = w;
        }
        __syncwarp();
        for (int c = lane; c < a.F; c += 32) {
          T acc = T(0);
#pragma unroll 8
          for (int k = 0; k < x.K; ++k) acc = fma_rn(x.f[(int64_t)s.slot_idx[k] * a.F + c], s.slot_key[k], acc);
          a.f_out[x.bq * a.F + c] = acc;
        }
        __syncwarp();
      }
    }
    __syncthreads();  // the next queries' clouds
  }
}

template <typename T, int V>
__global__ void __launch_bounds__(32 * kReplayWarps) replay_list_kernel(
    const __grid_constant__ ExactParams<T> a, int64_t pass_from) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  ReplayShared<T, V>& sm = *reinterpret_cast<ReplayShared<T, V>*>(smem_raw);
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = (int)cluster.block_rank(), ranks = (int)cluster.num_blocks();
  ReplayShared<T, V>& sm0 = *cluster.map_shared_rank(&sm, 0);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const SegHeader* sh = static_cast<const SegHeader*>(a.segs);
  if (sh && *a.status) return;  // nothing writes it while this kernel runs
  const int64_t n_items = *a.list_count;
  if (n_items > pass_from) {  // the same for all CTAs
    replay_passes<T, V>(a, n_items);
    return;
  }
  for (int64_t item = blockIdx.x / ranks; item < n_items; item += gridDim.x / ranks) {
    FlaggedQuery<T> x;
    if (!flagged_query(a, a.list[item], x)) continue;
    const int64_t bq = x.bq, e0 = x.e0;
    const int K = x.K, P = x.P;
    const T* recb = x.rec;
    const T* fb = x.f;
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
            sm.s.slot_key[t] = sm.merged[t].key;
            sm.s.slot_idx[t] = sm.merged[t].idx;
          }
          __syncwarp();
          mk.start(sm.s.slot_key, sm.s.pos_key, sm.s.pos_slot, K, lane);
          i0 = K;
        }
        int waiting = 0;
        auto run = [&](const Kept<T>* list, int i0, int m) {
          Kept<T> next = i0 + lane < m ? list[i0 + lane] : Kept<T>{T(0), 0};
#pragma unroll 1
          for (; i0 < m; i0 += 32) {
            const Kept<T> x = next;
            const bool below = i0 + lane < m && x.key < mk.max_key;
            if (i0 + 32 + lane < m) next = list[i0 + 32 + lane];
            const unsigned b = __ballot_sync(kFullMask, below);
            if (!b) continue;
            if (below) sm.s.pending[waiting + __popc(b & ((1u << lane) - 1u))] = x;
            waiting += __popc(b);
            __syncwarp();
            if (waiting >= 32) {
              act(mk, sm.s, 32, true, lane);
              waiting -= 32;
              __syncwarp();
              if (lane < waiting) sm.s.pending[lane] = sm.s.pending[32 + lane];
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
        if (waiting) act(mk, sm.s, waiting, true, lane);
        // a NaN maximum lets nothing in, ever
        if (lane == 0) sm.limit = mk.max_key == mk.max_key ? mk.max_key : T(-INFINITY);
      }
      cluster.sync();
      limit = sm0.limit;
    }
    // ---- sort and outputs
    if (rank == 0) {
      if (warp == 0) sort_slots(mk, sm.s, K, lane);
      __syncthreads();
      T w = T(0);
      if (tid < K) {
        w = weight_of(sm.s.slot_key[tid]);
        const int idx = sm.s.slot_idx[tid];
        a.dists[e0 + tid] = sm.s.slot_key[tid];
        a.idxs[e0 + tid] = (int64_t)idx;
        a.w_out[e0 + tid] = w;
        if (a.adj_count && (unsigned)idx < (unsigned)P) atomicAdd(&a.adj_count[x.row0 + idx], 1);
      }
      __syncthreads();
      if (tid < K) sm.s.slot_key[tid] = w;
      __syncthreads();
      for (int c = tid; c < a.F; c += 32 * kReplayWarps) {
        T acc = T(0);
#pragma unroll 8
        for (int k = 0; k < K; ++k) acc = fma_rn(fb[(int64_t)sm.s.slot_idx[k] * a.F + c], sm.s.slot_key[k], acc);
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
  constexpr size_t smem = std::max(sizeof(ReplayShared<T, V>), sizeof(PassShared<T, V>));
  static_assert(smem <= 227 * 1024, "shared memory");
  int dev = 0;
  cudaGetDevice(&dev);
  if (cudaFuncSetAttribute(replay_list_kernel<T, V>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) !=
      cudaSuccess)
    return KNNAG_ERR_CUDA;
  cudaLaunchConfig_t cfg{};
  cfg.blockDim = dim3(32 * kReplayWarps);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = ranks;
  attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  // as many clusters as run at a time (eight CTAs find room 15 times, not 18),
  // which loop over the queries
  static std::atomic<int> resident[64][kReplayMaxRanks + 1];  // by device; threads that meet find the same value
  int clusters = dev >= 0 && dev < 64 ? resident[dev][ranks].load(std::memory_order_relaxed) : 0;
  if (!clusters) {
    cfg.gridDim = dim3((unsigned)(num_sms(dev) / ranks * ranks));
    if (cudaOccupancyMaxActiveClusters(&clusters, replay_list_kernel<T, V>, &cfg) != cudaSuccess || clusters < 1) {
      cudaGetLastError();
      clusters = num_sms(dev) / ranks;
    }
    clusters = std::max(1, std::min(clusters, num_sms(dev) / ranks));
    if (dev >= 0 && dev < 64) resident[dev][ranks].store(clusters, std::memory_order_relaxed);
  }
  cfg.gridDim = dim3((unsigned)(clusters * ranks));
  // A pass takes about as long as one round of clusters over up to 24576 points
  // and as long as one more for every 24576 after that (the launch's own time with
  // 74, 148 and 300 flagged queries, clusters against passes: P = 4096 30, 30 and
  // 90 us against 40, 40 and 45; P = 30000 150, 260 and 520 against 115, 130 and 140;
  // P = 131072 345, 680 and 1360 against 365, 390 and 415).
  const int64_t pass_from = (int64_t)clusters * std::max(1, max_points / 24576);
  if (cudaLaunchKernelEx(&cfg, replay_list_kernel<T, V>, a, pass_from) != cudaSuccess) return KNNAG_ERR_CUDA;
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
