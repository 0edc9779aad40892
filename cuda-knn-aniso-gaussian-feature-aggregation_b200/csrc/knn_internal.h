// Internal parameter blocks and workspace layout shared by the .cu files of
// libknn_aniso.so.  Not part of the C ABI.
#pragma once

#include <cuda_runtime.h>
#include <nvtx3/nvToolsExt.h>
#include <stddef.h>
#include <stdint.h>

#include "knn_aniso.h"
#include "knn_ragged.h"

namespace knnag {

// NVTX range over one host-side stage of a call (the kernels it enqueues
// show up under it in a timeline profiler; without one attached the push
// and pop are no-ops).  Names start with "knnag:".
struct NvtxRange {
  explicit NvtxRange(const char* name) { nvtxRangePushA(name); }
  ~NvtxRange() { nvtxRangePop(); }
  NvtxRange(const NvtxRange&) = delete;
  NvtxRange& operator=(const NvtxRange&) = delete;
};

template <typename T>
struct ExactParams {
  const T* q;
  const T* rec;  // per-point records [B*P*16]
  const T* f;
  // isotropic forward only (key = squared Euclidean distance): raw points,
  // sigma [B,P,iso_stride] (component 0 scales the key in the weight); the
  // weight sum goes to w_out[B,Q,1]
  const T* iso_p;
  const T* iso_sigma;
  int iso_stride;
  int B, Q, P, F, K;
  const int* list;         // replay: the flagged queries' rows, list[0 .. *list_count)
  const int* list_count;
  T* f_out;
  T* w_out;
  T* dists;
  int64_t* idxs;
  // ragged calls (FP32): per-query sizes and offsets from the segment table,
  // records from the cloud set.  Nothing is done when *status is nonzero (a
  // table that failed validation).
  const char* cs;
  const void* segs;
  int* status;
  // optional (uniform calls): per point row b*P + i, the number of written
  // entries that select it (the adjacency's first pass), zeroed beforehand
  int* adj_count;
};

struct SearchParams {
  const float* q;
  const int* perm_q;   // sorted position -> query index, per batch element
  const float* tinfo;  // per tile kTinfoFloats: its box and its sub-boxes (box, mu, pad)
  int ntile;           // tiles per batch element (ragged: the most of any cloud)
  const float* pairs;  // pair-interleaved tiles [B][P_pad/2][32]
  const float* rec;    // per-point records [B*P*16]
  const float* f;
  int B, Q, P, P_pad, F, K;
  int vec4;            // f and f_out rows may be read/written as float4
  float* f_out;
  float* w_out;
  float* dists;
  int64_t* idxs;
  int* status;
  int* flag_count;
  int* flag_list;      // flagged queries: global query rows
  // ragged calls: records, tiles and boxes come from the cloud set, sizes
  // and offsets from the segment table; work items are taken in order from
  // item_counter
  const char* cs;
  const void* segs;
  int* item_counter;
  // Test hook of the timeout path (knnag_debug_set_search_stall): the tile
  // copy of visit `stall_visit` is armed on its mbarrier but never issued,
  // so the waits on it run out after `wait_spins` sleeps; -1 (no stall)
  // and the default budget otherwise.
  int stall_visit;
  int wait_spins;
  // optional (uniform calls): entries per point row, counted as written
  int* adj_count;
  // optional (uniform calls): per batch element [Q], sorted query position
  // -> a position in the sorted point order near the query (the middle of
  // its cell's points), where the seed window of the threshold is taken
  const int* qseed;
  // optional (uniform calls): the plan kernels' outputs, read by the search:
  // seed thresholds per sorted query [B*Q], the CTA items (batch element,
  // first and end sorted query, 0), and the per-block estimates
  float* tau0;
  int4* items;
  int* plan_est;
  // tensor-core filtered search (uniform calls): per tile the B operand of
  // the approximate-key GEMM [B*ntile][kTcOpsFloats] and its error-bound
  // terms [B*ntile][kTcInfoFloats], written by the tile-info kernel
  const float* tcops;
  const float* tcinfo;
};

// One-warp-per-query search (knn_search_warp.cu).
template <typename T>
struct WarpSearchParams {
  const T* q;
  const int* perm_q;   // sorted position -> query index, per batch element
  const int* qseed;    // uniform calls: per sorted query, a near position in the sorted points
  const T* rec;        // per-point records [B*P*16]
  const T* pairs;      // field-major tiles [B][ntile][16][64 pairs][2]
  const float* tbox;   // tile boxes, 7 planes of B*ntile: min xyz, max xyz, mu
  const float* gbox;   // boxes of groups of 32 tiles, 7 planes of B*ngroup
  const float4* sbox;  // per tile 4 x (min xyz, mu), then 4 x (max xyz, 0) of its sub-boxes
  const T* f;
  int B, Q, P, F, K, ntile, ngroup;  // ragged: K and ntile are the most of any segment / cloud
  int vec;             // f and f_out rows may be accessed 16 bytes at a time
  T* f_out;
  T* w_out;
  T* dists;
  int64_t* idxs;
  int* status;
  int* flag_count;
  int* flag_list;      // flagged queries: global query rows
  int* adj_count;      // optional (uniform calls): entries per point row, counted as written
  // ragged calls: everything per cloud comes from the cloud set, sizes and
  // offsets from the segment table, work items from item_counter
  const char* cs;
  const void* segs;
  int* item_counter;
};
constexpr int kWarpSearchMaxK = 128;
// Most tiles per cloud a search takes (P <= 2 097 152), as before this
// kernel: larger clouds are refused with KNNAG_ERR_TOO_LARGE (FP32, K <= 32)
// or go to the exact kernel (FP64, K > 32), which takes any size.
constexpr int kSearchMaxTiles = 16384;
// Warps (CTAs of one warp) per SM the registers are held to.  More warps hide
// more of each one's latency, fewer spill less: 24, 28 and 32 warps took 62,
// 64 and 62 us (table workload), 431, 433 and 420 us (65536 surface queries,
// K = 32), 1.78, 1.74 and 1.67 ms (524288 sphere queries).
template <typename T, int V>
struct WarpSearchShape {
  static constexpr int warps = sizeof(T) == 4 ? (V == 1 ? 32 : 16) : 8;
};
template <typename T>
int launch_search_warp(const WarpSearchParams<T>& a, int shape, cudaStream_t st);
int launch_search_warp_ragged(const WarpSearchParams<float>& a, int shape, int64_t cap_items, cudaStream_t st);

// Launch shape of the search.  The C ABI's launch-shape code s
// (knnag_set_search_splits, the segment tables' `splits`) selects the queries
// a warp of a uniform call takes: 16, 8, 4, 4, 4, 2 and 1 for s = 1, 2, 4, 8,
// 16, 32 and 64.  In segment tables it sets the size of the work items (128,
// 64, 32, 32, 32, 16 and 8 queries), which the search takes a unit at a time.
inline constexpr int search_qpc(int shape) {
  return shape == 1 ? 128 : shape == 2 ? 64 : shape == 32 ? 16 : shape == 64 ? 8 : 32;
}
inline constexpr int search_qpw(int shape) { return search_qpc(shape) / 8; }
inline bool search_shape_ok(int shape) {
  return shape == 1 || shape == 2 || shape == 4 || shape == 8 || shape == 16 || shape == 32 || shape == 64;
}
// Launch-shape code of the uniform search that filters candidates with
// approximate keys from the tensor cores (search_tc_kernel: 128 queries per
// CTA, one thread per query); uniform calls only (segment tables take the
// codes above).
constexpr int kShapeTensorFilter = 128;
inline bool search_setting_ok(int shape) { return search_shape_ok(shape) || shape == kShapeTensorFilter; }

// ------------------------------------------------------------- workspace
// Forward workspace: [status, flag_count] | flag_list [B*Q] | records (when
// the caller passed no points buffer) | pair tiles (FP32 fast path).
struct FwdLayout {
  size_t status, flag_list, rec, pairs, total;
  // spatial index (FP32 search path): bound parts [B*bound_parts(B)*8], cell counts / offsets
  // [B*cells(+1)], point and query permutations, tile boxes [B*ntile*8]
  size_t bounds, cell_count, cell_offset, perm_p, perm_q, tinfo;
  size_t qseed;  // [B*Q] ints: seed positions of the sorted queries
  size_t tau0, plan_est, items;  // search plan: seeds [B*Q], estimates, CTA items
  size_t tcops, tcinfo;          // tensor-core filter: per tile B operand and bound terms
  size_t tbox, gbox, sbox;       // boxes of tiles, groups of tiles, sub-boxes (see WarpSearchParams)
  size_t pf, qf;                 // FP64: points and queries rounded to FP32 (what the cells are taken from)
  int P_pad, bits;
};
// Whether a call is served through the spatial index (else by the exact
// kernel).  FP64 and K > 32 had only the exact kernel and its small
// workspace: they take the index where its padded tiles at most double the
// points and the launches' grids hold the batch.  A few FP64 queries of a small
// cloud and few neighbours stay with the exact kernel, one or two per SM and hardly
// a turn of MinK each: 296 queries take 12 us there and 23 through the index at P =
// 128, K = 1, 25 and 27 at P = 200, K = 8, 23 and 27 at P = 128, K = 16, but 29 and
// 29 at P = 200, K = 16; 740 of them 27 and 25 at P = 128, K = 8.  MinK's turns grow
// with the points where these come ever nearer (P = 200: 57 and 21), so P is bound too.
inline bool forward_indexed(int B, int Q, int P, int K, int dtype) {
  if (dtype == KNNAG_F32 && K <= 32) return true;
  if (dtype == KNNAG_F64 && (int64_t)B * Q <= 256 && P <= 256 && (int64_t)K * P <= 2048) return false;
  return K <= kWarpSearchMaxK && P >= kTilePoints && B <= 65535 && (int64_t)P <= (int64_t)kSearchMaxTiles * kTilePoints;
}
// Grid bits per axis of n elements: 8^bits cells hold at most 8 of them each on
// average.
int spatial_bits(int n);
// The same for P points: at least one cell per point beyond 4096 points.
// Points that fill no volume (surfaces, clusters) crowd into few cells, whose
// inner order is random; with the finer grid a query of the 131072-point
// sphere visits 14 instead of 15 sub-boxes and the unit of four 18 instead of
// 22, one of a cluster mixture (P = 30000, K = 32) 37 instead of 51.  Up to
// 4096 points the coarse grid keeps the scan inside the scatter launch.
int point_bits(int P);
// tc_ops: also write the tensor-core filter's per-tile operands (L.tcops, L.tcinfo)
template <typename T>
int launch_spatial_index(const float* qf, const float* pf, const T* rec, int B, int Q, int P, int P_pad, char* ws,
                         const FwdLayout& L, cudaStream_t st, bool tc_ops = false);
// The records and the whole index in one launch, for elements that one cluster
// of CTAs holds (knn_spatial.cu); also zeroes the status words and the
// adjacency's counts.
bool index_in_one_launch(int B, int Q, int P);
template <typename T>
int launch_index_cluster(const T* p, const T* sigma, const T* R, const T* q, int B, int Q, int P, T* rec, char* ws,
                         const FwdLayout& L, cudaStream_t st, int* zero_words, int n_zero, int* zero_rows,
                         int64_t zero_rows2);
int launch_exclusive_scan(int* count, int n, int* out, cudaStream_t st);
int launch_cloudset_index(char* cs, const CloudSetHeader& h, const CloudDesc* cd_dev, int max_p, int max_ntile,
                          int* cnt, int* perm_p, cudaStream_t st);
int launch_query_order(const float* q, const char* cs, const void* segs_dev, int cap_segs, int64_t cap_q,
                       int cap_cells, int* cnt, int* off, int* perm_q, const int* status, cudaStream_t st);

// Ragged forward workspace: [status, flag_count, item_counter] | flag_list
// [cap_q] | perm_q [cap_q] | query cell counts / offsets [cap_cells (+1)],
// cap_cells = cap_q + 8 * cap_segs (a segment of Q queries has at most
// max(Q, 8) cells).
struct RaggedLayout {
  size_t status, flag_list, perm_q, cell_count, cell_offset, total;
  int64_t cap_cells;
};
RaggedLayout ragged_layout(int cap_segs, int64_t cap_q);
int launch_validate_segments(const char* cs, const void* segs, int cap_segs, int64_t cap_q, int64_t cap_e, int max_k,
                             int ntile_cap, int qpc, int* status, cudaStream_t st);
int ragged_forward_impl(const char* cs, const void* segs, const float* q, const float* f, int F, int cap_segs,
                        int64_t cap_q, int64_t cap_e, int max_k, int ntile_cap, int splits, float* f_out, float* w_out,
                        float* dists, int64_t* idxs, void* workspace, cudaStream_t st);
int ragged_grad_q_impl(const char* cs, const void* segs, const float* q, const float* f, int F, const float* gfo,
                       const float* f_row_sums, const int64_t* idxs, int64_t cap_q, float* dq, const int* status,
                       cudaStream_t st);
int launch_row_sums(const void* f, int64_t rows, int F, int dtype, void* out, cudaStream_t st);
// Every query (of segments with K > 32: ragged calls) by the exact kernel.
template <typename T>
int launch_exact(const ExactParams<T>& a, cudaStream_t st);
// The queries of a.list (knn_replay.cu), K <= kWarpSearchMaxK; max_points: the
// most points of any of their clouds.
template <typename T>
int launch_replay_list(const ExactParams<T>& a, int max_points, cudaStream_t st);
int variants_precomputed(const void* q, const void* f, const void* rec, const int64_t* idxs, int B, int Q, int P,
                         int F, int K, int dtype, void* f_out, void* w_out, void* dists, cudaStream_t st);
int variants_lookup(const void* q, const void* p, const void* f, const void* rec, const int64_t* table, int tstride, int B, int Q,
                    int P, int F, int K, int dtype, int* nearest, void* f_out, void* w_out, void* dists,
                    int64_t* idxs, cudaStream_t st);
FwdLayout fwd_layout(int B, int Q, int P, int K, int dtype, bool own_rec, bool indexed);
// The layout a workspace of `bytes` holds: the indexed one where the call is
// served through the index and it fits, else the exact kernel's (FP64 and
// K > 32 only); L.total > bytes when neither fits.
FwdLayout fwd_layout_in(int B, int Q, int P, int K, int dtype, bool own_rec, size_t bytes, bool* indexed);

// Adjacency (CSR) layout: rowptr [B*P+1] | cursor [B*P] (the counts) | unsorted
// [N] | entries [N] | fill [B*P] (the fused fill's cursors; few rows only).
struct AdjLayout {
  size_t rowptr, cursor, unsorted, entries, fill, total;
};
AdjLayout adj_layout(int B, int Q, int P, int K);

// Tensor-core filtered search of a uniform FP32 call (knn_search_tc.cu);
// KNNAG_ERR_TOO_LARGE when its shared memory does not fit (the caller then
// takes the CUDA-core search).
int launch_search_tc(const SearchParams& a, cudaStream_t st);
// Whether the tensor-core search's shared memory fits for `ntile` tiles.
bool search_tc_fits(int ntile);
// The search plan (knn_search.cu) for blocks of qpc sorted queries, nb per
// batch element: seed thresholds into a.tau0, the blocks' estimates into
// a.plan_est, the CTA items, heaviest first, into a.items.
int launch_search_plan(const SearchParams& a, int qpc, int nb, cudaStream_t st);
// Most blocks the plan orders (its estimates are staged in shared memory).
int search_plan_max_blocks();
int num_sms(int dev);

// Process-wide split count of the uniform search (0: automatic), set by
// knnag_set_search_splits (defined in knn_capi.cu).
int search_splits_setting();
// Process-wide test hook of the search's bounded waits, set by
// knnag_debug_set_search_stall (defined in knn_capi.cu): writes the
// stall_visit / wait_spins fields of a SearchParams.
void apply_search_debug(SearchParams& sp);

// Instrumentation shared by the .cu files (defined in knn_capi.cu).
void note_launches(int n);
void profile_begin(cudaStream_t st);
void profile_end(cudaStream_t st);

inline size_t align256(size_t x) { return (x + 255) / 256 * 256; }

// Backward workspace: status | records | adjacency | per-entry coefficients.
struct BwdLayout {
  size_t status, rec, adj, coef, rowsum, total;  // rowsum: sum over columns of f per point (scalar grad_f_out)
};
BwdLayout bwd_layout(int B, int Q, int P, int F, int K, int dtype);

// Arguments of one backward call (order 1 or 2).
struct BwdArgs {
  int order;
  const void *ggq, *gfo, *q, *p, *f, *sigma, *R, *w_in;
  const int64_t* idxs;
  int B, Q, P, F, K, dtype, needs;
  const void *points, *adjacency, *coef_in;
  void *dgfo, *dq, *dp, *df, *dsigma, *dR, *coef_out;
  void* workspace;
};
int backward_impl(const BwdArgs& x, cudaStream_t st);

// Packs the point records; block 0 also zeroes zero_words[0..n_zero) (a
// call's status words) so no separate memset is needed.
int launch_pack_points(const void* p, const void* sigma, const void* R, int B, int P, int dtype, void* rec,
                       cudaStream_t st, int* zero_words = nullptr, int n_zero = 0, int* zero_rows = nullptr,
                       int64_t zero_rows2 = 0);
// Chunks per batch element of the packing kernel that also bounds the points:
// chunk c of element b writes its box to parts[(b * bound_parts(B) + c) * 8 ...]
// (min xyz, max xyz), which the cell kernels reduce.  128 for few elements (with
// 32, a quarter of the SMs packed B = 1, P = 131072 in 33 us; 128 take 12), for
// many no more than the chip's eight CTAs per SM: at B = 512, P = 64 128
// chunks an element take 91 us, 32 29 us, the two of this rule 5 us.
inline int bound_parts(int B) {
  int n = 128;
  while (n > 1 && (int64_t)n * B > 8 * 148) n /= 2;
  return n;
}
template <typename T>
int launch_pack_points_bounded(const T* p, const T* sigma, const T* R, const T* q, int B, int Q, int P, T* rec,
                               float* parts, float* pf, float* qf, cudaStream_t st, int* zero_words, int n_zero,
                               int* zero_rows, int64_t zero_rows2, int* zero_cells, int64_t n_cells);
// adjacency: optional buffer (adj_layout) whose per-point entry counts the
// forward writes, for launch_build_adjacency(..., counted = true)
int forward_impl(const void* q, const void* p, const void* f, const void* sigma, const void* R, int B, int Q,
                 int P, int F, int K, int dtype, void* f_out, void* w_out, void* dists, int64_t* idxs,
                 void* points, void* workspace, size_t workspace_bytes, cudaStream_t st, void* adjacency = nullptr);
int launch_build_adjacency(const int64_t* idxs, int B, int Q, int P, int K, void* adjacency, cudaStream_t st,
                           bool counted = false);

}  // namespace knnag
