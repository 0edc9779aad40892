// Device helpers of the tensor-core filtered search (knn_search_tc.cu) and its
// plan (knn_search.cu): the sorted candidate list, the seed thresholds and the
// tile lower bound.
#pragma once

#include "knn_common.cuh"
#include "knn_internal.h"

namespace knnag {

// Insert (k, i) into the sorted list when k is below its top.  The list is
// ascending, so lt[s] = k < keys[s] is false up to the insertion point and
// true after it; every slot takes its left neighbour (lt[s-1]), the new
// entry (lt[s] only) or stays -- all comparisons are independent, so the
// insertion is a few instructions deep instead of a chain through the list.
// The entry that falls off the top is remembered when it was a real entry
// equal to the new top (a tie the exactness flags must see).
template <int L>
__device__ __forceinline__ void list_insert(float (&keys)[L], int (&vals)[L], float k, int i, float& tie_key) {
  bool lt[L];
#pragma unroll
  for (int s = 0; s < L; ++s) lt[s] = k < keys[s];
  const float out_k = keys[L - 1];
  const int out_i = vals[L - 1];
#pragma unroll
  for (int s = L - 1; s > 0; --s) {
    keys[s] = lt[s - 1] ? keys[s - 1] : (lt[s] ? k : keys[s]);
    vals[s] = lt[s - 1] ? vals[s - 1] : (lt[s] ? i : vals[s]);
  }
  keys[0] = lt[0] ? k : keys[0];
  vals[0] = lt[0] ? i : vals[0];
  if (lt[L - 1] && out_i >= 0 && out_k == keys[L - 1]) tie_key = fminf(tie_key, out_k);
}

// Seed thresholds of a warp's NQ queries (NQ = 8, 16 or 32).  Any K+1
// distinct points bound a query's (K+1)-th smallest key from above by their
// own (K+1)-th smallest key, so keys above that can be dropped from the start
// instead of streaming through the list.  The points are a window of NS
// points of the sorted order around `my_seed` (held by lane j for query j:
// the middle of the query's cell, so the window is near it and the bound
// tight); the half-warp (the warp for NS = 64) of a query evaluates two
// points per lane and sorts the NS keys (bitonic, NaN as +inf), and the lane
// holding element K writes the bound into tab[j].w (tab[j] holds the query's
// x, y, z) for every valid query.  Nothing is written when P < NS.
template <int KMAX, int NQ>
__device__ __forceinline__ void seed_warp(float4* tab, int my_seed, bool valid, const float* pairs, int P, int K,
                                          int lane) {
  constexpr int NS = KMAX <= 16 ? 32 : 64;  // >= K + 1
  constexpr int LG = NS / 2;                // lanes per query
  constexpr int GPR = 32 / LG;              // queries per round
  constexpr int PPT = kTilePoints / 2;
  constexpr unsigned FULL = 0xffffffffu;
  static_assert((NQ / GPR) % 2 == 0, "two rounds per iteration");
  if (P >= NS) {
    const int gl = lane % LG;  // lane within the query's group
    const float2* pairs2 = reinterpret_cast<const float2*>(pairs);
    // two rounds per iteration: both windows' loads in flight together,
    // then the two sorts interleaved (NQ / GPR is even)
#pragma unroll 1
    for (int r = 0; r < NQ / GPR; r += 2) {
      int jj[2];
      bool qok[2];
      float2 pr[2][kRecLen];
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        jj[u] = (r + u) * GPR + lane / LG;  // warp-local query of this group
        const int center = __shfl_sync(FULL, my_seed, jj[u]);
        qok[u] = __shfl_sync(FULL, valid, jj[u]);
        int a0 = center - NS / 2;
        a0 = (a0 < 0 ? 0 : (a0 > P - NS ? P - NS : a0)) & ~1;
        const int pos = a0 + 2 * gl;  // even, pos + 1 < P
        const float2* tp = pairs2 + (int64_t)(pos >> 7) * (PPT * kRecLen) + ((pos & (kTilePoints - 1)) >> 1);
#pragma unroll
        for (int f = 0; f < kRecLen; ++f) pr[u][f] = __ldg(tp + f * PPT);
      }
      float v0[2], v1[2];
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const float4 qq = tab[jj[u]];
        const float2 s2 =
            key_pair(make_float2(qq.x, qq.x), make_float2(qq.y, qq.y), make_float2(qq.z, qq.z), pr[u]);
        v0[u] = s2.x == s2.x ? s2.x : INFINITY;
        v1[u] = s2.y == s2.y ? s2.y : INFINITY;
      }
      // element e = 2 * gl + h; ascending bitonic network over NS elements
#pragma unroll
      for (int kk = 2; kk <= NS; kk <<= 1) {
        const bool up = ((2 * gl) & kk) == 0;
#pragma unroll
        for (int j = kk >> 1; j > 0; j >>= 1) {
#pragma unroll
          for (int u = 0; u < 2; ++u) {
            if (j == 1) {
              const float lo = fminf(v0[u], v1[u]), hi = fmaxf(v0[u], v1[u]);
              v0[u] = up ? lo : hi;
              v1[u] = up ? hi : lo;
            } else {
              const float o0 = __shfl_xor_sync(FULL, v0[u], j >> 1), o1 = __shfl_xor_sync(FULL, v1[u], j >> 1);
              const bool take_min = (((2 * gl) & j) == 0) == up;
              v0[u] = take_min ? fminf(v0[u], o0) : fmaxf(v0[u], o0);
              v1[u] = take_min ? fminf(v1[u], o1) : fmaxf(v1[u], o1);
            }
          }
        }
      }
#pragma unroll
      for (int u = 0; u < 2; ++u)
        if (qok[u] && gl == (K >> 1)) tab[jj[u]].w = (K & 1) ? v1[u] : v0[u];
    }
  }
}

// Lower bound on the key of any query in box [bmin, bmax] against any point
// of a tile (its box ti[0..5], bound factor mu = ti[6]): see key_bound;
// -inf when the tile has no bound (mu < 0).
__device__ __forceinline__ float tile_lower_bound(const float* ti, const float* bmin, const float* bmax) {
  float d2 = 0.f;
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const float g = fmaxf(fmaxf(ti[c] - bmax[c], bmin[c] - ti[3 + c]), 0.f);
    d2 = __fmaf_rn(g, g, d2);
  }
  const float lb = key_bound<float>(ti[6], d2);
  return ti[6] >= 0.f ? fmaxf(lb, 0.f) : -INFINITY;
}

}  // namespace knnag
