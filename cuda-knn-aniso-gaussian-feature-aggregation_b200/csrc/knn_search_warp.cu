// kNN search + aggregation, one warp per query (FP32 and FP64, K <= 128,
// uniform and ragged calls).
//
// Replaces csrc/forward.cu:56-110 of the reference (one thread per query that
// scans every point and keeps its top K in global memory) and the launcher
// csrc/forward.cu:286-338.
//
// A warp owns a unit of up to QU consecutive queries of the Hilbert order (4
// in FP32 with K <= 32) and shares nothing with the other warps of its CTA
// but the L1 cache.  For the unit's queries:
//   1. window: the keys of the 64 V points around the query's cell in the
//      sorted order.  A bitonic network sorts all the unit's windows at once
//      (32 / QU lanes per query); the smallest 32 V keys are the query's
//      list, entry e in lane e % 32, register e / 32.  The K-th entry is the
//      threshold tau: any K points bound the K-th smallest key from above.
//   2. tiles: lanes test the bound of every 128-point tile (in groups of 32
//      tiles, whose own bound is tested first) against the box of the unit's
//      queries and the largest tau, then the 32-point sub-boxes of the listed
//      tiles against each query and its tau.
//   3. keys: two sub-boxes some query needs at a time, one per half-warp, a
//      point pair per lane: 15 coalesced loads of the field-major tile, then
//      18 packed FP32 operations per query give it 64 keys.  Keys below tau
//      are inserted one by one: an entry moves up a lane where the new key is
//      smaller than its left neighbour, two shuffles and a few selects.
// The window costs one step and leaves little to insert: at B = 2, Q = 12288,
// P = 4096, K = 16 a query visits 11 sub-boxes (9 % of the points) and
// inserts 9 points.  The unit's queries are neighbours and need much the same
// sub-boxes, so a point is loaded once for up to QU queries.
//
// Exactness.  The result equals the reference's MinK selection whenever the
// K smallest keys are pairwise distinct, the (K+1)-th is larger, and no NaN
// key falls in MinK's fill phase (points 0..K-1).  A point is dropped only if
// its key is above a threshold that is >= the K-th smallest key, or equal to
// the threshold; the smallest key dropped on equality is tracked (tie), as is
// one that leaves a full list equal to its new last entry.  A query is
// flagged for the exact replay when adjacent entries of its first K + 1 are
// equal, an entry is empty (NaN and infinite keys never fill one), tie <= the
// K-th key, or a fill-phase key is NaN.
#include <math.h>

#include "knn_common.cuh"
#include "knn_internal.h"

namespace knnag {

namespace {

constexpr unsigned kFull = 0xffffffffu;
// Tiles listed at a time per warp (a longer list is processed in batches,
// the tiles nearest to the unit in the sorted order first).
constexpr int kTileList = 96;
// Queries of a unit: what the registers hold lists of.
template <typename T, int V>
constexpr int kUnit = sizeof(T) == 4 ? (V == 1 ? 4 : V == 2 ? 2 : 1) : (V == 1 ? 2 : 1);

template <typename T>
struct Pair;
template <>
struct Pair<float> {
  using type = float2;
};
template <>
struct Pair<double> {
  using type = double2;
};

// Keys of one query against a point pair (fields 0..14 of the record).
__device__ __forceinline__ float2 pair_keys(float x, float y, float z, const float2* pr) {
  return key_pair(make_float2(x, x), make_float2(y, y), make_float2(z, z), pr);
}
__device__ __forceinline__ double2 pair_keys(double x, double y, double z, const double2* pr) {
  double ra[9], rb[9];
#pragma unroll
  for (int m = 0; m < 9; ++m) {
    ra[m] = pr[kR00 + m].x;
    rb[m] = pr[kR00 + m].y;
  }
  return make_double2(key_from_offset<double>(add_rn(x, pr[kNPX].x), add_rn(y, pr[kNPY].x), add_rn(z, pr[kNPZ].x), ra,
                                              pr[kS0].x, pr[kS1].x, pr[kS2].x),
                      key_from_offset<double>(add_rn(x, pr[kNPX].y), add_rn(y, pr[kNPY].y), add_rn(z, pr[kNPZ].y), rb,
                                              pr[kS0].y, pr[kS1].y, pr[kS2].y));
}

// Original point index of a record, kept in its pad field.
__device__ __forceinline__ int rec_index(float pad) { return __float_as_int(pad); }
__device__ __forceinline__ int rec_index(double pad) { return (int)pad; }

// Float interval holding a coordinate (the bounds are FP32).
__device__ __forceinline__ float lo_of(float v) { return v; }
__device__ __forceinline__ float hi_of(float v) { return v; }
__device__ __forceinline__ float lo_of(double v) { return __double2float_rd(v); }
__device__ __forceinline__ float hi_of(double v) { return __double2float_ru(v); }

template <typename T>
__device__ __forceinline__ T inf_of() {
  return T(INFINITY);
}

// Ascending bitonic sort of the N = GL * R distinct ints of each group of GL
// lanes (element lane_in_group * R + h in register h).  Blocks that a phase
// sorts downwards are complemented for it, so that every exchange in a lane is
// a plain min / max.
template <int GL, int R>
__device__ __forceinline__ void sort_group(int (&v)[R], int r) {
  constexpr int N = GL * R;
  int flip = 0;  // complement of this lane's registers in the current phase (phases of at least R)
#pragma unroll
  for (int kk = 2; kk <= N; kk <<= 1) {
    if (kk >= R) {
      const int f = kk < N && (r & (kk / R)) ? -1 : 0;
      if (f != flip || kk > R) {
#pragma unroll
        for (int h = 0; h < R; ++h) v[h] ^= flip ^ f;
      }
      flip = f;
    }
#pragma unroll
    for (int j = kk >> 1; j > 0; j >>= 1) {
      if (j >= R) {
        const bool upper = (r & (j / R)) != 0;
#pragma unroll
        for (int h = 0; h < R; ++h) {
          const int o = __shfl_xor_sync(kFull, v[h], j / R);
          v[h] = (o < v[h]) != upper ? o : v[h];
        }
      } else {
#pragma unroll
        for (int h = 0; h < R; ++h) {
          if ((h & j) == 0) {
            const int lo = min(v[h], v[h + j]), hi = max(v[h], v[h + j]);
            const bool up = kk >= R || (h & kk) == 0;  // compile-time
            v[h] = up ? lo : hi;
            v[h + j] = up ? hi : lo;
          }
        }
      }
    }
  }
}

// Sortable int of a key's leading bits with the window slot in its low bits.
// The sum makes -0 the +0 it equals.
template <int BITS>
__device__ __forceinline__ int tagged(float key, int slot) {
  const int b = __float_as_int(__fadd_rn(key, 0.f));
  return ((b ^ ((b >> 31) & 0x7fffffff)) & ~((1 << BITS) - 1)) | slot;
}
template <int BITS>
__device__ __forceinline__ int tagged(double key, int slot) {
  const int b = __double2hiint(__dadd_rn(key, 0.0));
  return ((b ^ ((b >> 31) & 0x7fffffff)) & ~((1 << BITS) - 1)) | slot;
}

// A list entry: key and position in the sorted points (-1: empty).
template <typename T>
struct __align__(2 * sizeof(T)) Entry {
  T key;
  int pos;
};

// Key of list entry e (uniform) in every lane.
template <typename T, int V>
__device__ __forceinline__ T list_key(const T (&k)[V], int e) {
  T v = k[0];
#pragma unroll
  for (int h = 1; h < V; ++h)
    if ((e >> 5) == h) v = k[h];
  return __shfl_sync(kFull, v, e & 31);
}

// Insert (nk, np), nk below the K-th key: entries above nk move one up; the
// last one leaves.
template <typename T, int V>
__device__ __forceinline__ void list_push(T (&k)[V], int (&p)[V], T nk, int np, int lane) {
  T rk[V];
  int rp[V];
#pragma unroll
  for (int h = 0; h < V; ++h) {  // the left neighbour's entry (lane 0: lane 31's)
    rk[h] = V == 1 ? __shfl_up_sync(kFull, k[h], 1) : __shfl_sync(kFull, k[h], (lane + 31) & 31);
    rp[h] = V == 1 ? __shfl_up_sync(kFull, p[h], 1) : __shfl_sync(kFull, p[h], (lane + 31) & 31);
  }
#pragma unroll
  for (int h = V - 1; h >= 0; --h) {
    const T lk = (h == 0 || lane) ? rk[h] : rk[h ? h - 1 : 0];
    const int lp = (h == 0 || lane) ? rp[h] : rp[h ? h - 1 : 0];
    const bool left = (h > 0 || lane > 0) && lk > nk, here = k[h] > nk;
    k[h] = left ? lk : (here ? nk : k[h]);
    p[h] = left ? lp : (here ? np : p[h]);
  }
}

// Lower bound of the keys of a query box [lo, hi] against a box of points
// (min xyz, mu), (max xyz): see key_bound.
template <typename T>
__device__ __forceinline__ float box_bound(const float (&mn)[3], const float (&mx)[3], float mu, const float (&lo)[3],
                                           const float (&hi)[3]) {
  float d2 = 0.f;
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const float g = fmaxf(fmaxf(mn[c] - hi[c], lo[c] - mx[c]), 0.f);
    d2 = __fmaf_rn(g, g, d2);
  }
  return key_bound<T>(mu, d2);
}

// What a unit of queries is searched against, and where its results go.
// Pointers are offset to the unit's batch element or segment and cloud.
template <typename T>
struct Item {
  const T* q;
  const int* perm_q;     // sorted position -> query index
  const T* rec;
  const typename Pair<T>::type* pairs;
  const float* tbox;     // tile boxes, plane m at tbox + m * tplane
  int64_t tplane;
  const float* gbox;     // boxes of groups of 32 tiles, plane m at gbox + m * gplane
  int64_t gplane;
  const float4* sbox;    // sub-boxes: 4 x (min xyz, mu), 4 x (max xyz, 0) per tile
  const T* f;
  T* f_out;
  T* w_out;
  T* dists;
  int64_t* idxs;
  int64_t row0;
  int* adj_count;
  const int* qseed;      // window centres per sorted query, or from the cell:
  const int* cell_start;
  const float* cbox;
  int cbits;
  int Q, P, K, ntile;
};

// Per-warp shared memory: a query of the unit, its window start and the
// smallest key it dropped on equality; its list (the window's keys before
// that); the tile list.
template <typename T>
struct __align__(16) UnitQuery {
  T x, y, z;
  int win;
  T tie;
};
template <typename T, int V>
struct __align__(16) WarpShared {
  static constexpr int NL = 32 * V, W = 64 * V, U = kUnit<T, V>;
  UnitQuery<T> q[U];
  union {
    struct {
      T key[U][W];    // the windows' keys
      int tag[U][NL]; // the smallest NL of each, sorted, as tagged()
    } win;
    Entry<T> list[U][NL];  // the results
  };
  int tiles[kTileList];
};

// Box planes of tile or group t.
template <typename T>
__device__ __forceinline__ float plane_bound(const float* box, int64_t plane, int t, const float (&lo)[3],
                                             const float (&hi)[3]) {
  float mn[3], mx[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    mn[c] = __ldg(box + c * plane + t);
    mx[c] = __ldg(box + (3 + c) * plane + t);
  }
  return box_bound<T>(mn, mx, __ldg(box + 6 * plane + t), lo, hi);
}

// The unit's queries: sorted positions [s0, s0 + n), n <= kUnit.
template <typename T, int V>
__device__ __forceinline__ void search_unit(const WarpSearchParams<T>& a, const Item<T>& it, int s0, int n,
                                            WarpShared<T, V>& sm) {
  using P2 = typename Pair<T>::type;
  constexpr int NL = 32 * V;            // list entries
  constexpr int W = 64 * V;             // window points
  constexpr int U = kUnit<T, V>;
  const int lane = threadIdx.x & 31;
  const int K = it.K, P = it.P;
  const int npos = it.ntile * kTilePoints;

  // lane j < U holds query min(j, n - 1)
  bool valid = lane < n;
  const int sp = s0 + min(lane, n - 1);
  int qi = it.perm_q[sp];
  if ((unsigned)qi >= (unsigned)it.Q) {  // the query order is a permutation: never taken
    if (valid) atomicOr(a.status, kStatusBadIndex);
    qi = 0;
    valid = false;
  }
  const T qx = it.q[(int64_t)qi * 3 + 0], qy = it.q[(int64_t)qi * 3 + 1], qz = it.q[(int64_t)qi * 3 + 2];
  int win = 0;
  if (lane < U) {
    if (it.qseed) {
      win = it.qseed[sp];
    } else {
      const int c = (int)cell_of((float)qx, (float)qy, (float)qz, it.cbox, it.cbits);
      win = ((it.cell_start[c] + it.cell_start[c + 1]) >> 1) - it.cell_start[0];
    }
  }
  int home = __shfl_sync(kFull, win, 0) / (kTilePoints * 32);  // group of tiles visited first
  // whole sub-boxes (those of the window are not visited again), at most 31 of
  // the last window's positions past the points
  win = max(0, min(win - W / 2 + 16, (P - W + 31) & ~31)) & ~31;
  if (lane < U) {
    UnitQuery<T>& uq = sm.q[lane];
    uq.x = qx;
    uq.y = qy;
    uq.z = qz;
    uq.win = win;
    uq.tie = inf_of<T>();
  }

  // A NaN key among points 0..K-1 changes MinK's result in ways only the
  // replay reproduces.  With those records and the query at most 1e6 in
  // magnitude no key overflows or is NaN; otherwise the keys are evaluated.
  bool nan_fill = false;
  {
    bool ok = fabs(qx) <= T(1e6) && fabs(qy) <= T(1e6) && fabs(qz) <= T(1e6);
    for (int i = lane; i < K; i += 32) {
      T r[kRecLen];
      load_rec(it.rec + (int64_t)i * kRecLen, r);
#pragma unroll
      for (int m = 0; m < kRecLen - 1; ++m) ok = ok && fabs(r[m]) <= T(1e6);  // NaN fails
    }
    if (!__all_sync(kFull, ok))
      for (int i = 0; i < K; ++i) {
        const T s = key_rec<T>(qx, qy, qz, it.rec + (int64_t)i * kRecLen);
        nan_fill = nan_fill || s != s;
      }
  }
  __syncwarp();

  // ---- windows: keys to shared memory (NaN and padding as +inf)
#pragma unroll
  for (int j = 0; j < U; ++j) {
    if (j && j >= n) continue;  // warp-uniform; unused keys below are never read as a live query's
    const UnitQuery<T> uq = sm.q[j];
#pragma unroll
    for (int v = 0; v < V; ++v) {
      const int pos = uq.win + 2 * (lane + 32 * v);  // even
      T k0 = inf_of<T>(), k1 = inf_of<T>();
      if (V <= 2 || pos < npos) {  // a window of V <= 2 fits one tile
        const P2* tp = it.pairs + (int64_t)(pos >> 7) * (64 * kRecLen) + ((pos & 127) >> 1);
        P2 pr[kRecLen];
#pragma unroll
        for (int m = 0; m < kRecLen - 1; ++m) pr[m] = __ldg(tp + m * 64);
        const P2 s = pair_keys(uq.x, uq.y, uq.z, pr);
        if (s.x < inf_of<T>()) k0 = s.x;
        if (s.y < inf_of<T>()) k1 = s.y;
      }
      P2 out;
      out.x = k0;
      out.y = k1;
      *reinterpret_cast<P2*>(&sm.win.key[j][2 * (lane + 32 * v)]) = out;
    }
  }
  __syncwarp();
  // all windows sorted at once by their keys' leading bits, the slot as a tag
  unsigned redo;  // groups whose order the leading bits leave open
  constexpr int GL = 32 / U;  // lanes per query
  {
    constexpr int R = W / GL;
    constexpr int BITS = V == 1 ? 6 : V == 2 ? 7 : 8;
    const int qj = min(lane / GL, n - 1), r = lane % GL;
    int v[R];
#pragma unroll
    for (int h = 0; h < R; ++h) v[h] = tagged<BITS>(sm.win.key[qj][r * R + h], r * R + h);
    sort_group<GL, R>(v, r);
    const int after = __shfl_down_sync(kFull, v[0], 1);
    bool open = false;
#pragma unroll
    for (int h = 0; h < R; ++h) {
      const int next = h + 1 < R ? v[h + 1 < R ? h + 1 : h] : after;
      open = open || ((v[h] ^ next) >> BITS) == 0 && v[h] < tagged<BITS>(inf_of<T>(), 0);
    }
    redo = __ballot_sync(kFull, open && r * R < NL);  // the last lane of a group has r * R >= NL
    if (r * R < NL) {
#pragma unroll
      for (int h = 0; h < R; ++h) sm.win.tag[lane / GL][r * R + h] = v[h] & (W - 1);
    }
  }
  __syncwarp();
  if (redo) {
    // leading bits in common: rank the window's exact keys (equal ones by slot).  Of
    // windows of uniform points 0.3, 2 and 11 % in FP32 (V = 1, 2, 4), 2, 12 and 63 % in FP64
    for (int j = 0; j < n; ++j) {
      if (!((redo >> (j * GL)) & (GL == 32 ? kFull : (1u << (GL & 31)) - 1u))) continue;
      for (int s = lane; s < W; s += 32) {
        const T ks = sm.win.key[j][s];
        int rank = 0;
        bool twin = false;
        for (int u = 0; u < W; ++u) {
          const T ku = sm.win.key[j][u];
          rank += ku < ks || (ku == ks && u < s);
          twin = twin || (ku == ks && u > s);
        }
        if (rank < NL) sm.win.tag[j][rank] = s;
        // the last entry of a full list equals a key left out of it
        if (rank == NL - 1 && K == NL && twin) sm.q[j].tie = ks;
      }
    }
    __syncwarp();
  }
  T k[U][V], tau[U];
  int p[U][V];
#pragma unroll
  for (int j = 0; j < U; ++j) {
    const int jj = j < n ? j : n - 1;
    const int a0 = sm.q[jj].win;
#pragma unroll
    for (int v = 0; v < V; ++v) {
      const int slot = sm.win.tag[j][lane + 32 * v];
      k[j][v] = sm.win.key[jj][slot];
      p[j][v] = k[j][v] < inf_of<T>() ? a0 + slot : -1;
    }
    tau[j] = j < n ? list_key<T, V>(k[j], K - 1) : T(-INFINITY);
  }

  // ---- the unit's box
  float blo[3] = {INFINITY, INFINITY, INFINITY}, bhi[3] = {-INFINITY, -INFINITY, -INFINITY};
#pragma unroll
  for (int j = 0; j < U; ++j) {
    const T qv[3] = {sm.q[j].x, sm.q[j].y, sm.q[j].z};
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      blo[c] = fminf(blo[c], lo_of(qv[c]));
      bhi[c] = fmaxf(bhi[c], hi_of(qv[c]));
    }
  }

  // ---- groups of 32 tiles: the nearest one first, its tiles by their bound
  // (so that the thresholds fall early), then the others whose bound is at or
  // below the largest threshold
  const int groups = (it.ntile + 31) >> 5;
  home = min(home, groups - 1);
  if (groups > 2) {
    int best = 0x7fffffff, bestg = 0;  // bound (its bits, 0 for none) and group of this lane
    for (int g = lane; g < groups; g += 32) {
      const int lb = __float_as_int(fmaxf(plane_bound<T>(it.gbox, it.gplane, g, blo, bhi), 0.f));
      if (lb < best || (lb == best && g == home)) {
        best = lb;
        bestg = g;
      }
    }
    const int least = __reduce_min_sync(kFull, best);
    const unsigned at_home = __ballot_sync(kFull, best == least && bestg == home);
    if (!at_home) home = __shfl_sync(kFull, bestg, __ffs(__ballot_sync(kFull, best == least)) - 1);
  }
  unsigned gmask = 0;      // groups gbase .. gbase + 31 still to visit
  int gbase = -32, nt = 0;
  {
    const int t = home * 32 + lane;
    float lb = INFINITY;
    if (t < it.ntile) lb = plane_bound<T>(it.tbox, it.tplane, t, blo, bhi);
    T tmax = tau[0];
#pragma unroll
    for (int j = 1; j < U; ++j) tmax = fmax(tmax, tau[j]);
    const bool keep = t < it.ntile && !((T)lb > tmax);
    int v[1] = {keep ? tagged<5>(fmaxf(lb, 0.f), lane) : 0x7fffffff};
    nt = __popc(__ballot_sync(kFull, keep));
    if (nt > 1) sort_group<32, 1>(v, lane);
    else if (keep) sm.tiles[0] = t;
    if (nt > 1 && lane < nt) sm.tiles[lane] = home * 32 + (v[0] & 31);
  }
#pragma unroll 1
  for (bool done = false;;) {
    if (nt == 0 && done) break;
    __syncwarp();

    // ---- the listed tiles' sub-boxes, 32 at a time
    const int nsub = nt * kSubBoxes;
#pragma unroll 1
    for (int r0 = 0; r0 < nsub; r0 += 32) {
      const bool in = r0 + lane < nsub;
      const int code = in ? sm.tiles[(r0 + lane) >> 2] * kSubBoxes + (lane & 3) : 0;  // sub-box of this lane
      const float4* sb = it.sbox + (int64_t)(code >> 2) * 8 + (code & 3);
      const float4 b0 = __ldg(sb), b1 = __ldg(sb + 4);
      const float mn[3] = {b0.x, b0.y, b0.z}, mx[3] = {b1.x, b1.y, b1.z};
      float lb[U];
      unsigned need[U], todo = 0;
#pragma unroll
      for (int j = 0; j < U; ++j) {
        const UnitQuery<T> uq = sm.q[j];
        const float lo[3] = {lo_of(uq.x), lo_of(uq.y), lo_of(uq.z)}, hi[3] = {hi_of(uq.x), hi_of(uq.y), hi_of(uq.z)};
        lb[j] = box_bound<T>(mn, mx, b0.w, lo, hi);
        // not those of the window
        need[j] = __ballot_sync(kFull, in && !((T)lb[j] > tau[j]) &&
                                           (unsigned)(code * 32 - uq.win) >= (unsigned)W);
        todo |= need[j];
      }
      while (todo) {
        const int b_lo = __ffs(todo) - 1;
        const unsigned rest = todo & (todo - 1);
        const int b_hi = rest ? __ffs(rest) - 1 : b_lo;
        const int mine = lane < 16 ? b_lo : b_hi;
        const unsigned both = (1u << b_lo) | (1u << b_hi);
        const bool half = lane < 16 || rest;
        // pair of this lane: pairs of a tile are 64 apart from field to field
        const int pid = __shfl_sync(kFull, code, mine) * 16 + (lane & 15);
        const int pos = 2 * pid;
        const P2* tp = it.pairs + (int64_t)(pid >> 6) * (64 * kRecLen) + (pid & 63);
        P2 pr[kRecLen];
#pragma unroll
        for (int m = 0; m < kRecLen - 1; ++m) pr[m] = __ldg(tp + m * 64);
        todo = 0;
#pragma unroll
        for (int j = 0; j < U; ++j) {
          if (need[j] & both) {
            const UnitQuery<T> uq = sm.q[j];
            const P2 s = pair_keys(uq.x, uq.y, uq.z, pr);
            const bool live = half && ((need[j] >> mine) & 1u);
            const unsigned m0 = __ballot_sync(kFull, live && s.x <= tau[j]),
                           m1 = __ballot_sync(kFull, live && s.y <= tau[j]);
            need[j] &= ~both;
            if (m0 | m1) {
              auto take = [&](unsigned m, T key, int odd) {
                while (m) {
                  const int l = 31 - __clz(m);  // in any order: equal keys are left to the replay
                  m ^= 1u << l;
                  const T nk = __shfl_sync(kFull, key, l);
                  const int np = __shfl_sync(kFull, pos, l) + odd;
                  if (nk <= tau[j]) {
                    if (nk == tau[j]) {
                      sm.q[j].tie = fmin(sm.q[j].tie, nk);
                      continue;
                    }
                    const T last = tau[j];
                    list_push<T, V>(k[j], p[j], nk, np, lane);
                    tau[j] = list_key<T, V>(k[j], K - 1);
                    // the entry that left a full list
                    if (K == NL && last == tau[j]) sm.q[j].tie = fmin(sm.q[j].tie, last);
                  }
                }
              };
              take(m0, s.x, 0);
              take(m1, s.y, 1);
              need[j] &= __ballot_sync(kFull, !((T)lb[j] > tau[j]));
            }
          }
          todo |= need[j];
        }
      }
    }
    if (done) break;
    __syncwarp();  // the tile list is rewritten
    nt = 0;
    T tmax = tau[0];
#pragma unroll
    for (int j = 1; j < U; ++j) tmax = fmax(tmax, tau[j]);
    while (nt <= kTileList - 32) {
      while (gmask == 0) {
        gbase += 32;
        if (gbase >= groups) break;
        const int g = gbase + lane;
        bool keep = g < groups && g != home;
        if (groups > 2 && keep) keep = !((T)plane_bound<T>(it.gbox, it.gplane, g, blo, bhi) > tmax);
        gmask = __ballot_sync(kFull, keep);
      }
      if (gmask == 0) {
        done = true;
        break;
      }
      const int t = (gbase + __ffs(gmask) - 1) * 32 + lane;
      gmask &= gmask - 1;
      const bool keep = t < it.ntile && !((T)plane_bound<T>(it.tbox, it.tplane, t, blo, bhi) > tmax);
      const unsigned b = __ballot_sync(kFull, keep);
      if (keep) sm.tiles[nt + __popc(b & ((1u << lane) - 1u))] = t;
      nt += __popc(b);
    }
  }

  // ---- lists to shared memory (the windows are no longer needed)
  __syncwarp();
#pragma unroll
  for (int j = 0; j < U; ++j)
#pragma unroll
    for (int v = 0; v < V; ++v) sm.list[j][lane + 32 * v] = Entry<T>{k[j][v], p[j][v]};
  __syncwarp();

  // ---- flags, then dists / idxs / w_out; each entry becomes (weight, index).
  // Groups of 16 lanes (K <= 16) or 32 take a query each.
  unsigned skip = __ballot_sync(kFull, !valid);  // queries without outputs here
  const int gk = K <= 16 ? 4 : 5;
  const unsigned gbits = gk == 4 ? 0xffffu << (lane & 16) : kFull;
#pragma unroll 1
  for (int j0 = 0; j0 < n; j0 += 32 >> gk) {
    const int j = min(j0 + (lane >> gk), n - 1), e0 = lane & ((1 << gk) - 1);
    const bool mine = j0 + (lane >> gk) < n;
    Entry<T>* list = sm.list[j];
    const bool nanq = __shfl_sync(kFull, nan_fill, j);
    bool fl = nanq || sm.q[j].tie <= list[K - 1].key, bad = false;
    T kk[V];
    int idx[V];
#pragma unroll
    for (int v = 0; v < V; ++v) {
      const int e = e0 + 32 * v;
      idx[v] = 0;
      kk[v] = T(0);
      if (e < K) {
        const Entry<T> en = list[e];
        kk[v] = en.key;
        fl = fl || en.pos < 0 || (e + 1 < NL && list[e + 1].key == en.key);
        if (en.pos >= 0 && en.pos < npos) {
          const P2 pad = __ldg(it.pairs + (int64_t)(en.pos >> 7) * (64 * kRecLen) + kRecPad * 64 + ((en.pos & 127) >> 1));
          idx[v] = rec_index(en.pos & 1 ? pad.y : pad.x);
          bad = bad || (unsigned)idx[v] >= (unsigned)P;  // tiles carry indices of their own cloud: never taken
        }
      }
    }
    const int row_q = __shfl_sync(kFull, qi, j);
    const unsigned bad_m = __ballot_sync(kFull, bad && mine) & gbits;
    const unsigned out_m = __ballot_sync(kFull, (fl || bad) && mine) & gbits;
    const bool dropped = out_m || ((skip >> j) & 1u);
    if (out_m && e0 == 0 && !((skip >> j) & 1u)) {
      if (bad_m)
        atomicOr(a.status, kStatusBadIndex);
      else
        a.flag_list[atomicAdd(a.flag_count, 1)] = (int)(it.row0 + row_q);
    }
    if (mine && !dropped) {
#pragma unroll
      for (int v = 0; v < V; ++v) {
        const int e = e0 + 32 * v;
        if (e < K) {
          const int64_t o = (int64_t)row_q * K + e;
          const T w = weight_of(kk[v]);
          it.dists[o] = kk[v];
          it.idxs[o] = (int64_t)idx[v];
          it.w_out[o] = w;
          list[e] = Entry<T>{w, idx[v]};
          if (it.adj_count) atomicAdd(&it.adj_count[idx[v]], 1);
        }
      }
    }
    // queries dropped by any group are skipped below
    const unsigned d = __ballot_sync(kFull, mine && dropped && e0 == 0);
    if (d & 1u) skip |= 1u << j0;
    if (gk == 4 && (d >> 16)) skip |= 1u << (j0 + 1);
  }
  __syncwarp();

  // ---- f_out = sum_k w_k f[idx_k], in k order with fma.  Groups of 2^g lanes,
  // 16 bytes a lane, take the unit's queries side by side, a slice of columns
  // at a time: the queries share most of their neighbours, so a slice of a
  // row one of them has loaded is still in L1 when the next one asks for it.
  using V16 = typename Group16<T>::type;
  const int cols = a.vec ? a.F / (int)(16 / sizeof(T)) : a.F;
  int g = 0;
  while (g < 5 && (1 << g) < cols && (n << g) < 32) ++g;
  const int sub = lane >> g, c0 = lane & ((1 << g) - 1), per = 32 >> g;
  const uint32_t stride = (uint32_t)a.F * (uint32_t)sizeof(T);
#pragma unroll 1
  for (int j0 = 0; j0 < n; j0 += per) {
    const int j = min(j0 + sub, n - 1);
    const int64_t row = __shfl_sync(kFull, qi, j);
    if (j0 + sub >= n || ((skip >> j) & 1u)) continue;
    const Entry<T>* list = sm.list[j];
#pragma unroll 1
    for (int c = c0; c < cols; c += 1 << g) {
      if (a.vec) {
        const char* fb = reinterpret_cast<const char*>(it.f) + 16 * (size_t)c;
        T acc[16 / sizeof(T)];
#pragma unroll
        for (int u = 0; u < (int)(16 / sizeof(T)); ++u) acc[u] = T(0);
        constexpr int RB = 8;  // rows in flight
        int k0 = 0;
#pragma unroll 1
        for (; k0 + RB <= K; k0 += RB) {
          V16 v[RB];
          T w[RB];
#pragma unroll
          for (int u = 0; u < RB; ++u) {
            const Entry<T> en = list[k0 + u];
            w[u] = en.key;
            v[u] = __ldg(reinterpret_cast<const V16*>(fb + (uint64_t)(uint32_t)en.pos * stride));
          }
#pragma unroll
          for (int u = 0; u < RB; ++u) fma_group(v[u], w[u], acc);
        }
        for (; k0 < K; ++k0) {
          const Entry<T> en = list[k0];
          fma_group(__ldg(reinterpret_cast<const V16*>(fb + (uint64_t)(uint32_t)en.pos * stride)), en.key, acc);
        }
        reinterpret_cast<V16*>(it.f_out + row * a.F)[c] = group_of(acc);
      } else {
        T acc = T(0);
#pragma unroll 8
        for (int k = 0; k < K; ++k) {
          const Entry<T> en = list[k];
          acc = fma_rn(__ldg(it.f + (int64_t)en.pos * a.F + c), en.key, acc);
        }
        it.f_out[row * a.F + c] = acc;
      }
    }
  }
}

// Uniform calls: CTA i, one warp, serves the sorted queries [i % nb * qpw, ...)
// of batch element i / nb, a unit at a time.  CTAs of one warp, since units
// take very different times (queries off the surface visit many tiles): with
// 8, 4, 2 and 1 warps a CTA the search of 65536 surface queries measured 646,
// 484, 491 and 435 us, of 524288 2.37, 1.97, 2.09 and 1.74 ms, the table
// workload 68, 68, 69 and 60 us.
template <typename T, int V>
__global__ void __launch_bounds__(32, WarpSearchShape<T, V>::warps)
    search_warp_kernel(WarpSearchParams<T> a, int nb, int qpw) {
  __shared__ WarpShared<T, V> sm;
  const int64_t b = blockIdx.x / nb;
  int s0 = (blockIdx.x - (int)b * nb) * qpw;
  const int s1 = min(s0 + qpw, a.Q);
  Item<T> it;
  it.q = a.q + b * a.Q * 3;
  it.perm_q = a.perm_q + b * a.Q;
  it.rec = a.rec + b * a.P * kRecLen;
  it.pairs = reinterpret_cast<const typename Pair<T>::type*>(a.pairs) + b * a.ntile * (kTilePoints / 2) * kRecLen;
  it.tplane = (int64_t)a.B * a.ntile;
  it.tbox = a.tbox + b * a.ntile;
  it.gplane = (int64_t)a.B * a.ngroup;
  it.gbox = a.gbox + b * a.ngroup;
  it.sbox = a.sbox + b * a.ntile * 8;
  it.f = a.f + b * a.P * a.F;
  it.f_out = a.f_out + b * a.Q * a.F;
  it.w_out = a.w_out + b * a.Q * a.K;
  it.dists = a.dists + b * a.Q * a.K;
  it.idxs = a.idxs + b * a.Q * a.K;
  it.row0 = b * a.Q;
  it.adj_count = a.adj_count ? a.adj_count + b * a.P : nullptr;
  it.qseed = a.qseed + b * a.Q;
  it.cell_start = nullptr;
  it.cbox = nullptr;
  it.cbits = 0;
  it.Q = a.Q;
  it.P = a.P;
  it.K = a.K;
  it.ntile = a.ntile;
  for (; s0 < s1; s0 += kUnit<T, V>) {
    search_unit<T, V>(a, it, s0, min(kUnit<T, V>, s1 - s0), sm);
    __syncwarp();
  }
}

// Ragged calls (FP32, K <= 32): a persistent CTA of one warp takes a
// unit of one segment's sorted queries at a time from a counter until the
// table's work items (qpc queries each) run out.  Item i belongs to the last
// segment whose item_off <= i.  Single units whatever qpc is, for the same
// reason: 24 clouds of 1024 to 32768 points took 1.43 ms with fetches of 8
// queries, 1.03 ms with 4.
constexpr int kFetch = kUnit<float, 1>;
__global__ void __launch_bounds__(32, WarpSearchShape<float, 1>::warps)
    search_warp_ragged_kernel(WarpSearchParams<float> a, int qpc) {
  __shared__ WarpShared<float, 1> sm;
  if (*a.status) return;  // the table failed validation
  const SegHeader* sh = static_cast<const SegHeader*>(a.segs);
  const SegDesc* sd = seg_descs(a.segs);
  const CloudSetHeader* ch = reinterpret_cast<const CloudSetHeader*>(a.cs);
  const CloudDesc* cd = cloud_descs(a.cs);
  const int nseg = sh->nseg, n_items = sh->n_items, parts = qpc / kFetch;
  for (;;) {
    int fetch = 0;
    if (threadIdx.x == 0) fetch = atomicAdd(a.item_counter, 1);
    fetch = __shfl_sync(kFull, fetch, 0);
    const int item = fetch / parts, part = fetch - item * parts;
    if (item >= n_items) break;
    if (fetch < 0) {  // the counter starts at 0 and only grows: never taken
      if (threadIdx.x == 0) atomicOr(a.status, kStatusBadIndex);
      break;
    }
    const SegDesc g = sd[seg_of_item(sd, nseg, item)];
    const CloudDesc c = cd[g.cloud];
    if (g.K < 1 || g.K > 32 || g.K > a.K || g.K > c.P || c.ntile > a.ntile || sh->qpc != qpc) {
      if (threadIdx.x == 0) atomicOr(a.status, kStatusBadTable);
      continue;
    }
    int s0 = (item - g.item_off) * qpc + part * kFetch;
    const int s1 = min(s0 + kFetch, g.Q);
    Item<float> it;
    it.q = a.q + g.q_off * 3;
    it.perm_q = a.perm_q + g.q_off;
    it.rec = reinterpret_cast<const float*>(a.cs + ch->rec_off) + c.p_off * kRecLen;
    it.pairs = reinterpret_cast<const float2*>(a.cs + ch->pairs_off) + c.tile_off * (kTilePoints / 2) * kRecLen;
    it.tplane = ch->total_tiles;
    it.tbox = reinterpret_cast<const float*>(a.cs + ch->tbox_off) + c.tile_off;
    it.gplane = tile_groups(ch->total_tiles, ch->C);
    it.gbox = reinterpret_cast<const float*>(a.cs + ch->gbox_off) + first_group(c.tile_off, g.cloud);
    it.sbox = reinterpret_cast<const float4*>(a.cs + ch->sbox_off) + c.tile_off * 8;
    it.f = a.f + c.p_off * a.F;
    it.f_out = a.f_out + g.q_off * a.F;
    it.w_out = a.w_out + g.e_off;
    it.dists = a.dists + g.e_off;
    it.idxs = a.idxs + g.e_off;
    it.row0 = g.q_off;
    it.adj_count = nullptr;
    it.qseed = nullptr;
    it.cell_start = reinterpret_cast<const int*>(a.cs + ch->celloff_off) + c.cell_off;
    it.cbox = reinterpret_cast<const float*>(a.cs + ch->bnd_off) + (int64_t)g.cloud * 8;
    it.cbits = c.bits;
    it.Q = g.Q;
    it.P = c.P;
    it.K = g.K;
    it.ntile = c.ntile;
    for (; s0 < s1; s0 += kUnit<float, 1>) {
      search_unit<float, 1>(a, it, s0, min(kUnit<float, 1>, s1 - s0), sm);
      __syncwarp();
    }
  }
}

template <typename T, int V>
int launch_v(const WarpSearchParams<T>& a, int shape, cudaStream_t st) {
  const int qpw = search_qpw(shape);
  const int64_t nb = ((int64_t)a.Q + qpw - 1) / qpw;
  if (nb * a.B > 0x7fffffff) return KNNAG_ERR_TOO_LARGE;
  profile_begin(st);
  search_warp_kernel<T, V><<<(unsigned)(nb * a.B), 32, 0, st>>>(a, (int)nb, qpw);
  profile_end(st);
  note_launches(1);
  return cudaGetLastError() == cudaSuccess ? KNNAG_OK : KNNAG_ERR_CUDA;
}

}  // namespace

template <typename T>
int launch_search_warp(const WarpSearchParams<T>& a, int shape, cudaStream_t st) {
  if (a.K <= 32) return launch_v<T, 1>(a, shape, st);
  if (a.K <= 64) return launch_v<T, 2>(a, shape, st);
  if (a.K <= kWarpSearchMaxK) return launch_v<T, 4>(a, shape, st);
  return KNNAG_ERR_ARG;
}
template int launch_search_warp<float>(const WarpSearchParams<float>&, int, cudaStream_t);
template int launch_search_warp<double>(const WarpSearchParams<double>&, int, cudaStream_t);

int launch_search_warp_ragged(const WarpSearchParams<float>& a, int shape, int64_t cap_items, cudaStream_t st) {
  int dev = 0;
  cudaGetDevice(&dev);
  int64_t grid = (int64_t)num_sms(dev) * WarpSearchShape<float, 1>::warps;
  const int64_t fetches = cap_items * (search_qpc(shape) / kFetch);
  if (grid > fetches) grid = fetches;
  if (grid < 1) grid = 1;
  profile_begin(st);
  search_warp_ragged_kernel<<<(unsigned)grid, 32, 0, st>>>(a, search_qpc(shape));
  profile_end(st);
  note_launches(1);
  return cudaGetLastError() == cudaSuccess ? KNNAG_OK : KNNAG_ERR_CUDA;
}

}  // namespace knnag
