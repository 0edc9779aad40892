// Spatial ordering for the search: points and queries of every batch element
// are counting-sorted by the Hilbert-curve index of a uniform grid cell, the search
// tiles are packed in that order (each record keeps its original point
// index), and every 128-point tile gets an axis-aligned box and a lower bound
// on the key of any query against any of its points:
//     key(q, i) >= mu_tile * dist(q, box_tile)^2,
//     mu_tile = min over the tile's points of  lambda_min(R^T diag(sigma) R)
//               - 1e-5 * sum_a |sigma_a| |R_a|^2,
// where lambda_min is computed in double and the second term covers the
// rounding of the FP32 key (|key_fp32 - key_exact| <= ~12 * 2^-24 *
// |q - p|^2 * sum_a |sigma_a| |R_a|^2, as long as the rotated offsets' squares
// are normal floats: at distances that count for a bound, above 1e-15, their
// lost digits are covered too where |R_a| >= 3e-5; a point with a shorter row
// gets 0).  mu is rounded down to FP32, FLT_MAX at most.  With every sigma >= 0
// every key is >= 0, so mu = 0 still bounds; a tile holding a negative or
// non-finite value has no bound at all (its keys may be negative): mu = NaN, in
// the tile infos -1.
// The searches skip tiles, and 32-point sub-boxes of them, whose bound exceeds
// the thresholds; the order of points inside a cell
// (atomic scatter) never changes a result, only the work done.
#include <cooperative_groups.h>
#include <math.h>

#include <algorithm>

#include "knn_common.cuh"
#include "knn_internal.h"

namespace knnag {

// Element groups of a counting sort: the batch elements of a uniform batch
// (group g = elements [g*n, (g+1)*n), cells [g*8^bits, ...)), the clouds of
// a cloud set, or the segments of a segment table (whose bounds are their
// cloud's).  Positions of group g in the sorted order start where its first
// element does, because the scan runs over [group][cell].
struct GroupRange {
  int64_t start;
  int n, cell_off, bits, bnd;
};
struct GroupMap {
  int n, bits;               // uniform batches
  const CloudDesc* clouds;   // cloud set (points)
  const SegDesc* segs;       // segment table (queries)
  const SegHeader* seg_hdr;  // live segment count
  const char* cs;            // cloud set whose bounds the segments use
  const int* status;         // segments: nothing is done once this is nonzero
};
// Bounds array of a map: the cloud set's own for segments, else `bnd`.
__device__ __forceinline__ const float* group_bounds(const GroupMap& m, const float* bnd) {
  return m.cs ? reinterpret_cast<const float*>(m.cs + reinterpret_cast<const CloudSetHeader*>(m.cs)->bnd_off) : bnd;
}
__device__ __forceinline__ bool group_range(const GroupMap& m, int g, GroupRange& r) {
  if (m.segs) {
    if ((m.status && *m.status) || g >= m.seg_hdr->nseg) return false;
    const SegDesc& s = m.segs[g];
    r = GroupRange{s.q_off, s.Q, s.qcell_off, s.qbits, s.cloud};
  } else if (m.clouds) {
    const CloudDesc& c = m.clouds[g];
    r = GroupRange{c.p_off, c.P, c.cell_off, c.bits, g};
  } else {
    r = GroupRange{(int64_t)g * m.n, m.n, g << (3 * m.bits), m.bits, g};
  }
  return true;
}

// Per group of points: bounding box, bnd[g] = {min xyz, max xyz}.
__global__ void __launch_bounds__(512) point_bounds_kernel(const float* __restrict__ rec, GroupMap m,
                                                           float* __restrict__ bnd) {
  __shared__ float red[6][16];
  const int b = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  GroupRange r;
  group_range(m, b, r);
  float mn[3] = {INFINITY, INFINITY, INFINITY}, mx[3] = {-INFINITY, -INFINITY, -INFINITY};
#pragma unroll 4
  for (int i = tid; i < r.n; i += blockDim.x) {
    const float* rr = rec + (r.start + i) * kRecLen;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      const float v = -rr[kNPX + a];
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
    bnd[b * 8 + tid] = v;
  }
}

// A counting-sort job: the elements of the groups of `m` (points from
// records, or queries from q) and where their cells start in the shared
// count / offset arrays.  One launch can run two jobs (blockIdx.z), e.g. the
// points and the queries of a batch, whose cells are then scanned together.
struct CellJob {
  const float* xyz;
  int stride, negate;
  GroupMap m;
  int cell_base;
  int nparts;  // > 0: bnd holds nparts partial boxes per group, reduced here
  // queries of a uniform batch sorted together with its points (whose cells
  // come first in the scan): seed[position - seed_sub] = the middle of the
  // element's cell in its group's sorted points
  int* seed;
  int64_t seed_sub;
};

// Seed position of an element in cell c (global index in the scanned
// arrays) of the query job j: the middle of the same cell's points, as a
// position in the group's sorted points.  The points' cells of group r sit
// at r.cell_off + (c - j.cell_base); off[] is the exclusive scan.
__device__ __forceinline__ int seed_of(const CellJob& j, const GroupRange& r, const int* off, int c) {
  const int pc = c - j.cell_base;
  return ((off[pc] + off[pc + 1]) >> 1) - off[r.cell_off];
}

// The box of group r: bnd's entry, or the reduction of its nparts partial
// boxes (into shared memory, by the first six warps of the CTA; all threads
// of the CTA must call this).
__device__ __forceinline__ const float* job_bounds(const CellJob& j, const float* bnd, const GroupRange& r,
                                                   float* gbs) {
  if (j.nparts <= 0) return group_bounds(j.m, bnd) + r.bnd * 8;
  const int a = threadIdx.x >> 5, lane = threadIdx.x & 31;  // warp a: plane a of the partial boxes
  if (a < 6) {
    float v = a < 3 ? INFINITY : -INFINITY;
    for (int i = lane; i < j.nparts; i += 32) {
      const float w = __ldg(bnd + ((int64_t)r.bnd * j.nparts + i) * 8 + a);
      v = a < 3 ? fminf(v, w) : fmaxf(v, w);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float w = __shfl_xor_sync(0xffffffffu, v, o);
      v = a < 3 ? fminf(v, w) : fmaxf(v, w);
    }
    if (lane == 0) gbs[a] = v;
  }
  __syncthreads();
  return gbs;
}

// Cell histogram of the elements of group blockIdx.y of job blockIdx.z.
__global__ void cell_count_kernel(CellJob j0, CellJob j1, const float* __restrict__ bnd, int* __restrict__ count) {
  __shared__ float gbs[6];
  const CellJob& j = blockIdx.z ? j1 : j0;
  GroupRange r;
  if (!group_range(j.m, blockIdx.y, r)) return;
  const float s = j.negate ? -1.f : 1.f;
  const float* gb = job_bounds(j, bnd, r, gbs);
  int* cnt = count + j.cell_base + r.cell_off;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < r.n; i += gridDim.x * blockDim.x) {
    const float* v = j.xyz + (r.start + i) * j.stride;
    atomicAdd(&cnt[cell_of(s * v[0], s * v[1], s * v[2], gb, r.bits)], 1);
  }
}

// perm[offset[cell] + rank] = index within the group.
__global__ void cell_scatter_kernel(CellJob j0, CellJob j1, const float* __restrict__ bnd,
                                    const int* __restrict__ offset, int* __restrict__ cursor, int* __restrict__ perm) {
  __shared__ float gbs[6];
  const CellJob& j = blockIdx.z ? j1 : j0;
  GroupRange r;
  if (!group_range(j.m, blockIdx.y, r)) return;
  const float s = j.negate ? -1.f : 1.f;
  const float* gb = job_bounds(j, bnd, r, gbs);
  const int base = j.cell_base + r.cell_off;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < r.n; i += gridDim.x * blockDim.x) {
    const float* v = j.xyz + (r.start + i) * j.stride;
    const int c = base + (int)cell_of(s * v[0], s * v[1], s * v[2], gb, r.bits);
    const int pos = offset[c] + atomicAdd(&cursor[c], 1);
    perm[pos] = i;
    if (j.seed) j.seed[pos - j.seed_sub] = seed_of(j, r, offset, c);
  }
}

// The scatter with the scan folded in, for at most kScatterScanMax cells:
// every CTA scans the cell counts into shared memory itself (a few KB
// read from L2), so no separate scan launch sits between the count and the
// scatter; `cursor` (zeroed beforehand) ranks the elements of a cell.
constexpr int kScatterScanMax = 8192;

__global__ void __launch_bounds__(256) cell_scatter_scan_kernel(CellJob j0, CellJob j1, const float* __restrict__ bnd,
                                                                const int* __restrict__ count, int nc,
                                                                int* __restrict__ cursor, int* __restrict__ perm) {
  __shared__ int soff[kScatterScanMax];
  __shared__ int wsum[8];
  __shared__ float gbs[6];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int per = (nc + 255) / 256;  // <= 32 consecutive counts per thread
  int local = 0;
  for (int u = 0; u < per; ++u) {
    const int i = tid * per + u;
    if (i < nc) {
      const int v = count[i];
      soff[i] = v;
      local += v;
    }
  }
  int incl = local;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int t = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += t;
  }
  if (lane == 31) wsum[warp] = incl;
  __syncthreads();
  int run = incl - local;
  for (int w = 0; w < warp; ++w) run += wsum[w];
  for (int u = 0; u < per; ++u) {
    const int i = tid * per + u;
    if (i < nc) {
      const int v = soff[i];
      soff[i] = run;
      run += v;
    }
  }
  __syncthreads();
  const CellJob& j = blockIdx.z ? j1 : j0;
  GroupRange r;
  if (!group_range(j.m, blockIdx.y, r)) return;
  const float s = j.negate ? -1.f : 1.f;
  const float* gb = job_bounds(j, bnd, r, gbs);
  const int base = j.cell_base + r.cell_off;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < r.n; i += gridDim.x * blockDim.x) {
    const float* v = j.xyz + (r.start + i) * j.stride;
    const int c = base + (int)cell_of(s * v[0], s * v[1], s * v[2], gb, r.bits);
    const int pos = soff[c] + atomicAdd(&cursor[c], 1);
    perm[pos] = i;
    if (j.seed) j.seed[pos - j.seed_sub] = seed_of(j, r, soff, c);
  }
}

// Point groups of the tile kernels: uniform (group b: records [b*P, ...),
// tiles [b*ntile, ...)) or the clouds of a cloud set.
struct TileGroup {
  int64_t p0, t0;
  int P, ntile;
};
__device__ __forceinline__ TileGroup tile_group(const CloudDesc* cd, int b, int P, int ntile) {
  if (cd) return TileGroup{cd[b].p_off, cd[b].tile_off, cd[b].P, cd[b].ntile};
  return TileGroup{(int64_t)b * P, (int64_t)b * ntile, P, ntile};
}

// Smallest eigenvalue of a symmetric 3x3 matrix (closed form), double.
__device__ double sym3_min_eig(double a00, double a11, double a22, double a01, double a02, double a12) {
  const double p1 = a01 * a01 + a02 * a02 + a12 * a12;
  if (p1 == 0.0) return fmin(a00, fmin(a11, a22));
  const double qm = (a00 + a11 + a22) / 3.0;
  const double b00 = a00 - qm, b11 = a11 - qm, b22 = a22 - qm;
  const double p2 = b00 * b00 + b11 * b11 + b22 * b22 + 2.0 * p1;
  const double p = sqrt(p2 / 6.0);
  const double ip = 1.0 / p;
  const double c00 = b00 * ip, c11 = b11 * ip, c22 = b22 * ip, c01 = a01 * ip, c02 = a02 * ip, c12 = a12 * ip;
  double r = 0.5 * (c00 * (c11 * c22 - c12 * c12) - c01 * (c01 * c22 - c12 * c02) + c02 * (c01 * c12 - c11 * c02));
  r = fmin(1.0, fmax(-1.0, r));
  const double phi = acos(r) / 3.0;
  return qm + 2.0 * p * cos(phi + 2.0943951023931957);  // + 2 pi / 3
}

// Tensor-core filter operands of one tile, by the tile-info CTA (thread k:
// sorted point k, `real` unless padding; `tile` holds the records field-major,
// red[w][0..5] the box of warp w's points).  With o the tile's box centre,
// p' = p - o and M = R^T diag(sigma) R (in double), the point's features
//   psi = (M00, M11, M22, 2 M01, 2 M02, 2 M12, -2 (M p')_0..2, p'^T M p')
// meet a query's phi = (x^2, y^2, z^2, xy, xz, yz, x, y, z, 1), (x,y,z) =
// q - o, in phi . psi = (q - p)^T M (q - p), the key in exact arithmetic.
// Row k of the B operand holds (hi(psi), lo(psi), hi(psi), 0, 0), hi = psi
// with its low 13 mantissa bits cleared (a TF32 value), lo = psi - hi (exact);
// the search's A rows hold (hi(phi), hi(phi), lo(phi), 0, 0), so one K = 32
// TF32 product sums hi.hi + hi.lo + lo.hi.  Padding rows: psi = (0, .., 1e30).
// tcinfo: o (3) | 2^-12 max|psi_k| (10) | 1e-5 max nu (13) | max |p'|_1 (14)
// | 2^-20 max sum|M_ab| (15), nu = sum_a |sigma_a| |R_a|^2; entry 13 is +inf
// when a value of the tile is not finite (no bound: every point is a
// candidate).  The search turns these into its error bound.
__device__ void tc_tile_operand(const float* tile, float (*red)[8], int k, bool real, float* __restrict__ ops,
                                float* __restrict__ info) {
  __shared__ float red2[kTilePoints / 32][16];
  const int lane = k & 31, warp = k >> 5;
  float o[3];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    float lo = INFINITY, hi = -INFINITY;
    for (int w = 0; w < kTilePoints / 32; ++w) {
      lo = fminf(lo, red[w][a]);
      hi = fmaxf(hi, red[w][3 + a]);
    }
    o[a] = (lo <= hi && isfinite(lo) && isfinite(hi)) ? 0.5f * lo + 0.5f * hi : 0.0f;
  }
  float psi[10];
  float nu = 0.f, lam = 0.f, p1 = 0.f;
  bool bad = false;
  if (real) {
    double r[kRecLen];
#pragma unroll
    for (int m = 0; m < kRecLen; ++m) r[m] = tile[m * kTilePoints + k];
    double pp[3], M[3][3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}}, nud = 0.0;
#pragma unroll
    for (int a = 0; a < 3; ++a) pp[a] = -r[kNPX + a] - (double)o[a];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      const double sg = r[kS0 + a];
      double rn = 0.0;
#pragma unroll
      for (int m = 0; m < 3; ++m) {
        const double ra = r[kR00 + 3 * a + m];
        rn += ra * ra;
#pragma unroll
        for (int n2 = 0; n2 < 3; ++n2) M[m][n2] += sg * ra * r[kR00 + 3 * a + n2];
      }
      nud += fabs(sg) * rn;
    }
    double mp[3], pmp = 0.0, lamd = 0.0;
#pragma unroll
    for (int m = 0; m < 3; ++m) {
      mp[m] = M[m][0] * pp[0] + M[m][1] * pp[1] + M[m][2] * pp[2];
      pmp += pp[m] * mp[m];
#pragma unroll
      for (int n2 = 0; n2 < 3; ++n2) lamd += fabs(M[m][n2]);
    }
    const double pd[10] = {M[0][0], M[1][1], M[2][2], 2 * M[0][1], 2 * M[0][2], 2 * M[1][2],
                           -2 * mp[0], -2 * mp[1], -2 * mp[2], pmp};
#pragma unroll
    for (int j = 0; j < 10; ++j) {
      psi[j] = (float)pd[j];
      if (!isfinite(psi[j])) bad = true;
    }
#pragma unroll
    for (int m = 0; m < kRecLen - 1; ++m)
      if (!isfinite(r[m])) bad = true;
    nu = (float)(nud * (1.0 + 1e-6));
    lam = (float)(lamd * (1.0 + 1e-6));
    p1 = (float)((fabs(pp[0]) + fabs(pp[1]) + fabs(pp[2])) * (1.0 + 1e-6));
    if (!isfinite(nu) || !isfinite(lam) || !isfinite(p1)) bad = true;
  } else {
#pragma unroll
    for (int j = 0; j < 9; ++j) psi[j] = 0.f;
    psi[9] = 1e30f;
  }
  // B row k: (hi, lo, hi, 0, 0) in the core-matrix layout: 8-row groups of
  // 8 chunks of 4 values, 128 B per (group, chunk)
  float row[kTcK];
#pragma unroll
  for (int j = 0; j < 10; ++j) {
    const float h = tf32_hi(psi[j]);
    row[j] = h;
    row[10 + j] = psi[j] - h;
    row[20 + j] = h;
  }
  row[30] = row[31] = 0.f;
  float4* dst = reinterpret_cast<float4*>(ops + (k >> 3) * (8 * 32) + (k & 7) * 4);
#pragma unroll
  for (int c = 0; c < kTcK / 4; ++c) dst[c * 8] = make_float4(row[4 * c], row[4 * c + 1], row[4 * c + 2], row[4 * c + 3]);
  // tile maxima of the bound terms over its real points
  float v[14];
#pragma unroll
  for (int j = 0; j < 10; ++j) v[j] = real ? fabsf(psi[j]) : 0.f;
  v[10] = nu;
  v[11] = p1;
  v[12] = lam;
  v[13] = bad ? 1.f : 0.f;
#pragma unroll
  for (int off = 16; off > 0; off >>= 1)
#pragma unroll
    for (int j = 0; j < 14; ++j) v[j] = fmaxf(v[j], __shfl_xor_sync(0xffffffffu, v[j], off));
  if (lane == 0)
#pragma unroll
    for (int j = 0; j < 14; ++j) red2[warp][j] = v[j];
  __syncthreads();
  if (k < kTcInfoFloats) {
    auto tmax = [&](int j) { return fmaxf(fmaxf(red2[0][j], red2[1][j]), fmaxf(red2[2][j], red2[3][j])); };
    const bool nonfinite = red2[0][13] != 0.f || red2[1][13] != 0.f || red2[2][13] != 0.f || red2[3][13] != 0.f;
    float out;
    if (k < 3) out = o[k];
    else if (k < 13) out = ldexpf(tmax(k - 3), -12);
    else if (k == 13) out = nonfinite ? INFINITY : 1e-5f * tmax(10);
    else if (k == 14) out = tmax(11);
    else out = ldexpf(tmax(12), -20);
    info[k] = out;
  }
}

// One CTA of 128 threads per search tile (tile blockIdx.x of group
// blockIdx.y), one sorted point per thread: packs the tile field-major --
// field f of point pair m (points 2m, 2m+1) at float2 f * 64 + m, so a lane
// reads its pair's 16 fields conflict-free and one packed f32x2 evaluation
// gives both keys -- (field kRecPad carries the original point index, -1
// for padding, whose sigma is NaN so its key is never a candidate) and
// writes tinfo[tile * kTinfoFloats]: the tile's {min xyz, max xyz, mu, 0},
// then one such box per warp's 32 points (the sub-boxes).
// It also writes the same boxes where the one-warp-per-query search reads
// them: the tile's by plane (plane m at tbox[m * tplane + tile], lanes over
// tiles read each plane coalesced) and the sub-boxes as 8 float4 per tile
// (4 x (min, mu), then 4 x (max, 0): the four lanes of a tile read 64
// contiguous bytes).  FP64 records keep FP64 tiles; the boxes are rounded
// outwards to FP32.
template <typename T>
__device__ __forceinline__ T index_bits(int idx);
template <>
__device__ __forceinline__ float index_bits<float>(int idx) { return __int_as_float(idx); }
template <>
__device__ __forceinline__ double index_bits<double>(int idx) { return (double)idx; }
__device__ __forceinline__ float round_down(float v) { return v; }
__device__ __forceinline__ float round_up_f(float v) { return v; }
__device__ __forceinline__ float round_down(double v) { return __double2float_rd(v); }
__device__ __forceinline__ float round_up_f(double v) { return __double2float_ru(v); }

// A record through L2 (load_rec's read-only path is for data that the running
// kernel does not write).
__device__ __forceinline__ void load_rec_cg(const float* p, float (&r)[kRecLen]) {
#pragma unroll
  for (int i = 0; i < kRecLen / 4; ++i) {
    const float4 x = __ldcg(reinterpret_cast<const float4*>(p) + i);
    r[4 * i + 0] = x.x;
    r[4 * i + 1] = x.y;
    r[4 * i + 2] = x.z;
    r[4 * i + 3] = x.w;
  }
}
__device__ __forceinline__ void load_rec_cg(const double* p, double (&r)[kRecLen]) {
#pragma unroll
  for (int i = 0; i < kRecLen / 2; ++i) {
    const double2 x = __ldcg(reinterpret_cast<const double2*>(p) + i);
    r[2 * i + 0] = x.x;
    r[2 * i + 1] = x.y;
  }
}

// Shared memory of one tile.
template <typename T>
struct TileScratch {
  T tile[kTilePoints * kRecLen];
  float red[kTilePoints / 32][8];
};

// Tile t of group g by 128 threads (k: 0..127; whole warps).  Every thread of
// the CTA must call it (it has a CTA barrier); those of an inactive group only
// take part in that.
template <typename T>
__device__ __forceinline__ void tile_info_body(bool active, const T* rec, const int* perm, TileGroup g,
                                               int t, int k, TileScratch<T>& sm, T* __restrict__ pairs,
                                               float* __restrict__ tinfo, float* __restrict__ tbox, int64_t tplane,
                                               float4* __restrict__ sbox) {
  const int lane = k & 31, warp = k >> 5;
  float mn[3] = {INFINITY, INFINITY, INFINITY}, mx[3] = {-INFINITY, -INFINITY, -INFINITY};
  float mu = INFINITY;
  bool bad = false;
  if (active) {
    const int pos = t * kTilePoints + k;
    T* slot = sm.tile + k;  // field f of point k at slot[f * kTilePoints]
    if (pos >= g.P) {
#pragma unroll
      for (int m = 0; m < kRecLen; ++m)
        slot[m * kTilePoints] = m == kRecPad ? index_bits<T>(-1)
                                             : ((m == kS0 || m == kS1 || m == kS2) ? T(__int_as_float(0x7fc00000)) : T(0));
    } else {
      const int idx = __ldcg(perm + g.p0 + pos);
      const T* r = rec + (g.p0 + idx) * kRecLen;
      T v[kRecLen];
      load_rec_cg(r, v);  // another CTA of the cluster may have just written it
#pragma unroll
      for (int m = 0; m < kRecLen; ++m) slot[m * kTilePoints] = m == kRecPad ? index_bits<T>(idx) : v[m];
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        const T c = -v[kNPX + a];
        mn[a] = fminf(mn[a], round_down(c));
        mx[a] = fmaxf(mx[a], round_up_f(c));
        if (!isfinite(mn[a]) || !isfinite(mx[a])) bad = true;
      }
      double M[3][3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}};
      double err = 0.0;
      bool short_row = false;
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        const double s = v[kS0 + a];
        if (!(s >= 0.0)) bad = true;  // a negative (or NaN) precision: keys may be negative
        double rn = 0.0;
#pragma unroll
        for (int m = 0; m < 3; ++m) {
          const double ra = v[kR00 + 3 * a + m];
          rn += ra * ra;
#pragma unroll
          for (int n2 = 0; n2 < 3; ++n2) M[m][n2] += s * ra * (double)v[kR00 + 3 * a + n2];
        }
        err += fabs(s) * rn;
        if (sizeof(T) == 4 && s != 0.0 && rn < 1e-9) short_row = true;
      }
      const double lam = sym3_min_eig(M[0][0], M[1][1], M[2][2], M[0][1], M[0][2], M[1][2]);
      const double scale = fabs(M[0][0]) + fabs(M[1][1]) + fabs(M[2][2]) + fabs(M[0][1]) + fabs(M[0][2]) + fabs(M[1][2]);
      const double m = lam - 1e-9 * scale - 1e-5 * err;
      if (!isfinite(m)) bad = true;
      mu = fminf(mu, m > 0.0 && isfinite(m) && !short_row ? __double2float_rd(m * (1.0 - 1e-6)) : 0.0f);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        mn[a] = fminf(mn[a], __shfl_xor_sync(0xffffffffu, mn[a], o));
        mx[a] = fmaxf(mx[a], __shfl_xor_sync(0xffffffffu, mx[a], o));
      }
      mu = fminf(mu, __shfl_xor_sync(0xffffffffu, mu, o));
    }
    bad = __any_sync(0xffffffffu, bad);
    if (lane == 0) {
      for (int a = 0; a < 3; ++a) {
        sm.red[warp][a] = mn[a];
        sm.red[warp][3 + a] = mx[a];
      }
      sm.red[warp][6] = mu;
      sm.red[warp][7] = bad ? 1.0f : 0.0f;
      float* o = tinfo + (g.t0 + t) * kTinfoFloats + 8 * (1 + warp);  // this warp's sub-box
      for (int a = 0; a < 3; ++a) {
        o[a] = mn[a];
        o[3 + a] = mx[a];
      }
      o[6] = bad ? -1.0f : mu;  // +inf: no points (the box is empty)
      o[7] = 0.0f;
      sbox[(g.t0 + t) * 8 + warp] = make_float4(mn[0], mn[1], mn[2], bad ? NAN : mu);
      sbox[(g.t0 + t) * 8 + 4 + warp] = make_float4(mx[0], mx[1], mx[2], 0.f);
    }
  }
  __syncthreads();
  if (!active) return;
  const float4* src = reinterpret_cast<const float4*>(sm.tile);
  float4* dst = reinterpret_cast<float4*>(pairs + (g.t0 + t) * kTilePoints * kRecLen);
  for (int i = k; i < (int)(kTilePoints * kRecLen * sizeof(T) / 16); i += kTilePoints) dst[i] = src[i];
  if (k == 0) {
    for (int w = 1; w < kTilePoints / 32; ++w) {
      for (int a = 0; a < 3; ++a) {
        mn[a] = fminf(mn[a], sm.red[w][a]);
        mx[a] = fmaxf(mx[a], sm.red[w][3 + a]);
      }
      mu = fminf(mu, sm.red[w][6]);
      bad = bad || sm.red[w][7] != 0.0f;
    }
    float* o = tinfo + (g.t0 + t) * kTinfoFloats;
    for (int a = 0; a < 3; ++a) {
      o[a] = mn[a];
      o[3 + a] = mx[a];
    }
    o[6] = bad ? -1.0f : (mu < INFINITY ? mu : 0.0f);  // -1: the tile has no key bound
    o[7] = 0.0f;
    for (int m = 0; m < 6; ++m) tbox[m * tplane + g.t0 + t] = o[m];
    tbox[6 * tplane + g.t0 + t] = bad ? NAN : o[6];
  }
}

template <typename T>
__global__ void __launch_bounds__(kTilePoints) tile_info_kernel(const T* __restrict__ rec,
                                                                const int* __restrict__ perm,
                                                                const CloudDesc* __restrict__ cd, int P, int ntile,
                                                                T* __restrict__ pairs, float* __restrict__ tinfo,
                                                                float* __restrict__ tbox, int64_t tplane,
                                                                float4* __restrict__ sbox, float* __restrict__ tcops,
                                                                float* __restrict__ tcinfo) {
  const TileGroup g = tile_group(cd, blockIdx.y, P, ntile);
  const int t = blockIdx.x, k = threadIdx.x;
  if (t >= g.ntile) return;
  __shared__ __align__(16) TileScratch<T> sm;
  tile_info_body<T>(true, rec, perm, g, t, k, sm, pairs, tinfo, tbox, tplane, sbox);
  if constexpr (sizeof(T) == 4)
    if (tcops)
      tc_tile_operand(sm.tile, sm.red, k, t * kTilePoints + k < g.P, tcops + (g.t0 + t) * kTcOpsFloats,
                      tcinfo + (g.t0 + t) * kTcInfoFloats);
}

// ------------------------------------------------------ index in one launch
//
// The whole index of a small uniform call -- packed records, bounds, the
// counting sort of points and queries, tiles -- by one cluster of
// kIndexCtas CTAs per batch element: the steps that are launches of their own
// below are separated by cluster barriers here.  For elements of up to 4096
// points (the coarse grid's cells fit shared memory) and 32768 queries.
// What bounds it: latency, a handful of dependent memory round trips.  The four
// launches took 21 us at B = 2, Q = 1000, P = 500 and 26 us at B = 2, Q = 12288,
// P = 4096, gaps included; one takes 13 and 20, and a whole forward call of the
// first size went from 40 us to 33.
constexpr int kIndexCtas = 8;
constexpr int kIndexThreads = 1024;
constexpr int kIndexPoints = 4096;
constexpr int kIndexCells = 512;  // 8^spatial_bits(kIndexPoints)
constexpr int kIndexElements = 8;
constexpr int kIndexPerThread = 4;
constexpr int kIndexQueries = kIndexCtas * kIndexThreads * kIndexPerThread;
constexpr int kIndexTiles = kIndexPoints / kTilePoints / kIndexCtas;  // tiles of a CTA

template <typename T>
struct IndexShared {
  TileScratch<T> tile[kIndexTiles];
  float box[6];                        // of this CTA's points
  float red[6][kIndexThreads / 32];
  int count[2][kIndexCells];           // this CTA's points and queries per cell
  int start[2][kIndexCells];           // where they go; then the cursors
  int first[kIndexCells + 1];          // of the element's sorted points, per cell
  int wsum[2][kIndexThreads / 32];
};

template <typename T>
struct IndexParams {
  const T *p, *sigma, *R, *q;
  int Q, P, bits, ntile;
  T* rec;
  int *zero_words, n_zero;
  int* zero_rows;  // as pack_points_bounded_kernel
  int64_t zero_rows2;
  int *perm_p, *perm_q, *seed;
  T* pairs;
  float *tinfo, *tbox;
  int64_t tplane;
  float4* sbox;
};

template <typename T>
__global__ void __launch_bounds__(kIndexThreads) index_cluster_kernel(IndexParams<T> a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  IndexShared<T>& sm = *reinterpret_cast<IndexShared<T>*>(smem_raw);
  cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
  const int rank = (int)cluster.block_rank();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t b = blockIdx.x / kIndexCtas;
  const int cells = 1 << (3 * a.bits);
  if (blockIdx.x == 0 && tid < a.n_zero) a.zero_words[tid] = 0;
  static_assert(2 * kIndexCells == kIndexThreads, "a thread per cell of either kind");
  sm.count[tid / kIndexCells][tid % kIndexCells] = 0;
  // ---- this CTA's points: records, box
  const int share = (a.P + kIndexCtas - 1) / kIndexCtas;  // at most kIndexThreads
  const int pi = tid < share && rank * share + tid < a.P ? rank * share + tid : -1;
  float xyz[3] = {0.f, 0.f, 0.f};
  {
    float v[6] = {INFINITY, INFINITY, INFINITY, -INFINITY, -INFINITY, -INFINITY};
    if (pi >= 0) {
      const int64_t i = b * a.P + pi;
      pack_one<T>(a.p, a.sigma, a.R, i, a.rec);
      if (a.zero_rows) a.zero_rows[i] = a.zero_rows[i + a.zero_rows2] = 0;
#pragma unroll
      for (int m = 0; m < 3; ++m) {
        xyz[m] = (float)a.p[i * 3 + m];
        v[m] = fminf(v[m], xyz[m]);  // NaN leaves the box alone
        v[3 + m] = fmaxf(v[3 + m], xyz[m]);
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
      for (int m = 0; m < 6; ++m) {
        const float w = __shfl_xor_sync(0xffffffffu, v[m], o);
        v[m] = m < 3 ? fminf(v[m], w) : fmaxf(v[m], w);
      }
    if (lane == 0)
#pragma unroll
      for (int m = 0; m < 6; ++m) sm.red[m][warp] = v[m];
    __syncthreads();
    if (warp < 6) {
      float w = sm.red[warp][lane];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const float x = __shfl_xor_sync(0xffffffffu, w, o);
        w = warp < 3 ? fminf(w, x) : fmaxf(w, x);
      }
      if (lane == 0) sm.box[warp] = w;
    }
  }
  cluster.sync();
  // ---- the element's box; cells of this CTA's points and queries
  float box[6] = {INFINITY, INFINITY, INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
  for (int r = 0; r < kIndexCtas; ++r) {
    const float* o = cluster.map_shared_rank(sm.box, r);
#pragma unroll
    for (int m = 0; m < 6; ++m) box[m] = m < 3 ? fminf(box[m], o[m]) : fmaxf(box[m], o[m]);
  }
  int pcell = 0, qcell[kIndexPerThread];
  if (pi >= 0) {
    pcell = (int)cell_of(xyz[0], xyz[1], xyz[2], box, a.bits);
    atomicAdd(&sm.count[0][pcell], 1);
  }
#pragma unroll
  for (int u = 0; u < kIndexPerThread; ++u) {
    const int qi = (u * kIndexCtas + rank) * kIndexThreads + tid;
    qcell[u] = 0;
    if (qi < a.Q) {
      const T* v = a.q + (b * a.Q + qi) * 3;
      qcell[u] = (int)cell_of((float)v[0], (float)v[1], (float)v[2], box, a.bits);
      atomicAdd(&sm.count[1][qcell[u]], 1);
    }
  }
  cluster.sync();
  // ---- scan: thread c < 2 * kIndexCells takes cell c of the points or queries
  {
    const int kind = tid >= kIndexCells, c = tid - kind * kIndexCells;
    int before = 0, total = 0;
#pragma unroll
    for (int r = 0; r < kIndexCtas; ++r) {
      const int n = c < cells ? cluster.map_shared_rank(&sm, r)->count[kind][c] : 0;
      if (r < rank) before += n;
      total += n;
    }
    int incl = total;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int n = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += n;
    }
    if (lane == 31) sm.wsum[0][warp] = incl;
    __syncthreads();
    if (warp == 0) {  // 16 warps of points, 16 of queries
      const int n = sm.wsum[0][lane];
      int w = n;
#pragma unroll
      for (int o = 1; o < 16; o <<= 1) {
        const int x = __shfl_up_sync(0xffffffffu, w, o);
        if ((lane & 15) >= o) w += x;
      }
      sm.wsum[1][lane] = w - n;
    }
    __syncthreads();
    const int off = sm.wsum[1][warp] + incl - total;
    sm.start[kind][c] = off + before;
    if (kind == 0) {
      sm.first[c] = off;
      if (c == kIndexCells - 1) sm.first[kIndexCells] = off + total;
    }
  }
  __syncthreads();
  // ---- scatter
  if (pi >= 0) a.perm_p[b * a.P + atomicAdd(&sm.start[0][pcell], 1)] = pi;
#pragma unroll
  for (int u = 0; u < kIndexPerThread; ++u) {
    const int qi = (u * kIndexCtas + rank) * kIndexThreads + tid;
    if (qi < a.Q) {
      const int64_t pos = b * a.Q + atomicAdd(&sm.start[1][qcell[u]], 1);
      a.perm_q[pos] = qi;
      a.seed[pos] = (sm.first[qcell[u]] + sm.first[qcell[u] + 1]) >> 1;  // the middle of the cell's points
    }
  }
  cluster.sync();
  // ---- tiles: 128 threads each
  const int slot = tid / kTilePoints, t = rank + slot * kIndexCtas;
  const bool active = slot < kIndexTiles && t < a.ntile;
  tile_info_body<T>(active, a.rec, a.perm_p, TileGroup{b * a.P, b * a.ntile, a.P, a.ntile}, t, tid % kTilePoints,
                    sm.tile[slot < kIndexTiles ? slot : 0], a.pairs, a.tinfo, a.tbox, a.tplane, a.sbox);
}

// Boxes of groups of 32 tiles (warp blockIdx.x of batch element or cloud
// blockIdx.y): the search tests a group before its tiles.  mu is the least of
// the group's tiles, NaN where one has no bound.
__global__ void __launch_bounds__(32) group_box_kernel(const CloudDesc* __restrict__ cd, int ntile, int ngroup,
                                                       const float* __restrict__ tbox, int64_t tplane,
                                                       float* __restrict__ gbox, int64_t gplane) {
  const int b = blockIdx.y, gi = blockIdx.x, lane = threadIdx.x;
  const int64_t t0 = cd ? cd[b].tile_off : (int64_t)b * ntile;
  const int nt = cd ? cd[b].ntile : ntile;
  if (gi * 32 >= nt) return;
  const int t = gi * 32 + lane;
  float v[7];
#pragma unroll
  for (int m = 0; m < 7; ++m) v[m] = t < nt ? tbox[m * tplane + t0 + t] : (m >= 3 && m < 6 ? -INFINITY : INFINITY);
  const bool none = __any_sync(0xffffffffu, v[6] != v[6]);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
#pragma unroll
    for (int m = 0; m < 7; ++m) {
      const float w = __shfl_xor_sync(0xffffffffu, v[m], o);
      v[m] = m >= 3 && m < 6 ? fmaxf(v[m], w) : fminf(v[m], w);
    }
  if (lane == 0) {
    const int64_t g0 = (cd ? first_group(t0, b) : (int64_t)b * ngroup) + gi;
#pragma unroll
    for (int m = 0; m < 6; ++m) gbox[m * gplane + g0] = v[m];
    gbox[6 * gplane + g0] = none ? NAN : v[6];
  }
}

int point_bits(int P) {
  int bits = spatial_bits(P);
  if (P > 4096)
    while (bits < 10 && (int64_t(1) << (3 * bits)) < P) ++bits;
  return bits;
}

int spatial_bits(int P) {
  int bits = 1;
  while (bits < 10 && (int64_t(1) << (3 * bits)) * 8 < P) ++bits;
  return bits;
}

namespace {
unsigned grid_x(int64_t n, int sms, int groups) {
  const int64_t cap = std::max<int64_t>(1, (int64_t)sms * 16 / std::max(1, groups));
  return (unsigned)std::max<int64_t>(1, std::min<int64_t>((n + 255) / 256, cap));
}
}  // namespace

// qf, pf: the coordinates the cells are taken from (FP32): the queries, and
// for FP64 the rounded points (FP32 points are read from the records).
template <typename T>
int launch_spatial_index(const float* qf, const float* pf, const T* rec, int B, int Q, int P, int P_pad, char* ws,
                         const FwdLayout& L, cudaStream_t st, bool tc_ops) {
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const int bits = L.bits, cells = 1 << (3 * bits);
  float* bnd = reinterpret_cast<float*>(ws + L.bounds);
  int* cnt = reinterpret_cast<int*>(ws + L.cell_count);
  int* off = reinterpret_cast<int*>(ws + L.cell_offset);
  int* perm = reinterpret_cast<int*>(ws + L.perm_p);  // perm_q follows perm_p directly
  T* pairs = reinterpret_cast<T*>(ws + L.pairs);
  float* tinfo = reinterpret_cast<float*>(ws + L.tinfo);
  const int ntile = P_pad / kTilePoints;
  GroupMap pm{P, bits, nullptr, nullptr, nullptr, nullptr, nullptr};
  GroupMap qm{Q, bits, nullptr, nullptr, nullptr, nullptr, nullptr};
  // the packing kernel wrote bound_parts(B) partial boxes per element (reduced
  // by the cell kernels) and zeroed the cell counts.  Points and queries in
  // one counting sort: their cells are scanned together, so the queries'
  // positions start after all points' and land in perm_q, which follows perm_p
  const int64_t nc = 2 * (int64_t)B * cells;
  const int nparts = bound_parts(B);
  const CellJob jp = sizeof(T) == 4 ? CellJob{reinterpret_cast<const float*>(rec) + kNPX, kRecLen, 1, pm, 0, nparts}
                                    : CellJob{pf, 3, 0, pm, 0, nparts};
  const CellJob jq{qf, 3, 0, qm, B * cells, nparts, reinterpret_cast<int*>(ws + L.qseed), (int64_t)B * P};
  const dim3 grid(grid_x(P > Q ? P : Q, sms, B), B, 2);
  cell_count_kernel<<<grid, 256, 0, st>>>(jp, jq, bnd, cnt);
  if (nc <= kScatterScanMax) {
    // the packing kernel zeroed the offsets region too: it is the cursor here
    cell_scatter_scan_kernel<<<grid, 256, 0, st>>>(jp, jq, bnd, cnt, (int)nc, off, perm);
    note_launches(1);
  } else {
    int rc = launch_exclusive_scan(cnt, (int)nc, off, st);
    if (rc) return rc;
    cell_scatter_kernel<<<grid, 256, 0, st>>>(jp, jq, bnd, off, cnt, perm);
  }
  tile_info_kernel<T><<<dim3(ntile, B), kTilePoints, 0, st>>>(rec, perm, nullptr, P, ntile, pairs, tinfo,
                                                            reinterpret_cast<float*>(ws + L.tbox), (int64_t)B * ntile,
                                                            reinterpret_cast<float4*>(ws + L.sbox),
                                                            tc_ops ? reinterpret_cast<float*>(ws + L.tcops) : nullptr,
                                                            tc_ops ? reinterpret_cast<float*>(ws + L.tcinfo) : nullptr);
  note_launches(3);  // + 1 scan, counted by launch_exclusive_scan
  const int ngroup = (ntile + 31) / 32;
  if (ngroup > 2 && !tc_ops) {  // with one or two groups the search takes them all
    group_box_kernel<<<dim3(ngroup, B), 32, 0, st>>>(nullptr, ntile, ngroup, reinterpret_cast<const float*>(ws + L.tbox),
                                                     (int64_t)B * ntile, reinterpret_cast<float*>(ws + L.gbox),
                                                     (int64_t)B * ngroup);
    note_launches(1);
  }
  return cudaGetLastError() == cudaSuccess ? KNNAG_OK : KNNAG_ERR_CUDA;
}

template int launch_spatial_index<float>(const float*, const float*, const float*, int, int, int, int, char*,
                                         const FwdLayout&, cudaStream_t, bool);
template int launch_spatial_index<double>(const float*, const float*, const double*, int, int, int, int, char*,
                                          const FwdLayout&, cudaStream_t, bool);

// Elements that a cluster's shared memory and registers hold, and no more of
// them than find room at the same time (8 CTAs of a whole SM each, side by
// side): a graph-replayed forward at Q = 1000, P = 500 took 38 us with one
// launch and 40 with four at B = 8, but 55 and 49 at B = 16, 85 and 78 at 32.
bool index_in_one_launch(int B, int Q, int P) {
  return P <= kIndexPoints && Q <= kIndexQueries && B <= kIndexElements;
}

template <typename T>
int launch_index_cluster(const T* p, const T* sigma, const T* R, const T* q, int B, int Q, int P, T* rec, char* ws,
                         const FwdLayout& L, cudaStream_t st, int* zero_words, int n_zero, int* zero_rows,
                         int64_t zero_rows2) {
  IndexParams<T> a{};
  a.p = p;
  a.sigma = sigma;
  a.R = R;
  a.q = q;
  a.Q = Q;
  a.P = P;
  a.bits = L.bits;
  a.ntile = L.P_pad / kTilePoints;
  a.rec = rec;
  a.zero_words = zero_words;
  a.n_zero = n_zero;
  a.zero_rows = zero_rows;
  a.zero_rows2 = zero_rows2;
  a.perm_p = reinterpret_cast<int*>(ws + L.perm_p);
  a.perm_q = reinterpret_cast<int*>(ws + L.perm_q);
  a.seed = reinterpret_cast<int*>(ws + L.qseed);
  a.pairs = reinterpret_cast<T*>(ws + L.pairs);
  a.tinfo = reinterpret_cast<float*>(ws + L.tinfo);
  a.tbox = reinterpret_cast<float*>(ws + L.tbox);
  a.tplane = (int64_t)B * a.ntile;
  a.sbox = reinterpret_cast<float4*>(ws + L.sbox);
  const size_t smem = sizeof(IndexShared<T>);
  if (smem > 48 * 1024 && cudaFuncSetAttribute(index_cluster_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               (int)smem) != cudaSuccess)
    return KNNAG_ERR_CUDA;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)B * kIndexCtas);
  cfg.blockDim = dim3(kIndexThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = kIndexCtas;
  attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  if (cudaLaunchKernelEx(&cfg, index_cluster_kernel<T>, a) != cudaSuccess) return KNNAG_ERR_CUDA;
  note_launches(1);
  return cudaGetLastError() == cudaSuccess ? KNNAG_OK : KNNAG_ERR_CUDA;
}
template int launch_index_cluster<float>(const float*, const float*, const float*, const float*, int, int, int, float*,
                                         char*, const FwdLayout&, cudaStream_t, int*, int, int*, int64_t);
template int launch_index_cluster<double>(const double*, const double*, const double*, const double*, int, int, int,
                                          double*, char*, const FwdLayout&, cudaStream_t, int*, int, int*, int64_t);

// Cloud-set index: bounds, Hilbert order, sorted tiles and tile boxes of
// every cloud (records already packed); the cell offsets stay in the cloud
// set.  Scratch: cell counts [total_cells], point permutation [total_p].
int launch_cloudset_index(char* cs, const CloudSetHeader& h, const CloudDesc* cd_dev, int max_p, int max_ntile,
                          int* cnt, int* perm_p, cudaStream_t st) {
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const int C = h.C;
  const float* rec = reinterpret_cast<const float*>(cs + h.rec_off);
  int* off = reinterpret_cast<int*>(cs + h.celloff_off);
  float* bnd = reinterpret_cast<float*>(cs + h.bnd_off);
  float* pairs = reinterpret_cast<float*>(cs + h.pairs_off);
  float* tinfo = reinterpret_cast<float*>(cs + h.tinfo_off);
  GroupMap pm{0, 0, cd_dev, nullptr, nullptr, nullptr, nullptr};
  point_bounds_kernel<<<C, 512, 0, st>>>(rec, pm, bnd);
  if (cudaMemsetAsync(cnt, 0, (size_t)h.total_cells * 4, st) != cudaSuccess) return KNNAG_ERR_CUDA;
  const CellJob jp{rec + kNPX, kRecLen, 1, pm, 0, 0};
  const dim3 grid(grid_x(max_p, sms, C), C, 1);
  cell_count_kernel<<<grid, 256, 0, st>>>(jp, jp, bnd, cnt);
  int rc = launch_exclusive_scan(cnt, h.total_cells, off, st);
  if (rc) return rc;
  cell_scatter_kernel<<<grid, 256, 0, st>>>(jp, jp, bnd, off, cnt, perm_p);
  tile_info_kernel<float><<<dim3(max_ntile, C), kTilePoints, 0, st>>>(
      rec, perm_p, cd_dev, 0, 0, pairs, tinfo, reinterpret_cast<float*>(cs + h.tbox_off), h.total_tiles,
      reinterpret_cast<float4*>(cs + h.sbox_off), nullptr, nullptr);
  note_launches(4);  // + 1 scan
  if (max_ntile > 64) {  // the search reads the boxes of clouds with more than two groups
    group_box_kernel<<<dim3((max_ntile + 31) / 32, C), 32, 0, st>>>(
        cd_dev, 0, 0, reinterpret_cast<const float*>(cs + h.tbox_off), h.total_tiles,
        reinterpret_cast<float*>(cs + h.gbox_off), tile_groups(h.total_tiles, C));
    note_launches(1);
  }
  return cudaGetLastError() == cudaSuccess ? KNNAG_OK : KNNAG_ERR_CUDA;
}

// Query order of a segment table: every segment's queries counting-sorted by
// the Hilbert index of a grid cell over its cloud's box.  cnt/off hold cap_cells
// (+1) cells (the encoded total is at most that); perm_q gets, at each
// segment's rows, the segment-local query indices in sorted order.  Sizes
// come from the device copy of the table, so the launches replay on new
// tables of the same capacity.
int launch_query_order(const float* q, const char* cs, const void* segs_dev, int cap_segs, int64_t cap_q,
                       int cap_cells, int* cnt, int* off, int* perm_q, const int* status, cudaStream_t st) {
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  GroupMap qm{0, 0, nullptr, seg_descs(segs_dev), static_cast<const SegHeader*>(segs_dev), cs, status};
  if (cudaMemsetAsync(cnt, 0, (size_t)cap_cells * 4, st) != cudaSuccess) return KNNAG_ERR_CUDA;
  const dim3 grid(grid_x(cap_q, sms, cap_segs), cap_segs, 1);
  const CellJob jq{q, 3, 0, qm, 0, 0};
  cell_count_kernel<<<grid, 256, 0, st>>>(jq, jq, nullptr, cnt);
  int rc = launch_exclusive_scan(cnt, cap_cells, off, st);
  if (rc) return rc;
  cell_scatter_kernel<<<grid, 256, 0, st>>>(jq, jq, nullptr, off, cnt, perm_q);
  note_launches(2);
  return cudaGetLastError() == cudaSuccess ? KNNAG_OK : KNNAG_ERR_CUDA;
}

}  // namespace knnag
