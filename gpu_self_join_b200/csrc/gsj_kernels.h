// Host-side launchers of the self-join kernels (internal interface between
// gsj_api.cu and the kernel translation units).
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

#include "gsj_common.cuh"

namespace gsj {

// Resident CTAs per SM for a launch: the larger of the occupancy calculation
// and the same fit computed from the SM's limits (shared memory with the
// per-block reservation, registers in 256-register warp units, threads),
// since the calculation can come out below what the SM holds.  Results are
// cached per (device, kernel, block size, dynamic shared memory).
cudaError_t blocks_per_sm(const void* kern, int threads, size_t smem, int* per_sm);
// Lets launches of `kern` take up to the device's limit of dynamic shared memory
// (an error when `smem` is above it).  The attribute belongs to the kernel, not to
// a launch: set to each launch's own size, another thread's context could lower
// it between this thread's setting and launch, which then failed.
cudaError_t allow_smem(const void* kern, size_t smem);


template <typename T>
cudaError_t launch_variance(const T* in, uint64_t N, uint32_t n, T denom, T* var_out, cudaStream_t st);
template <typename T>
cudaError_t launch_minmax(const T* in, uint64_t N, uint32_t n, uint32_t k, const uint32_t* perm, T* part,
                          uint32_t nparts, T* out, cudaStream_t st);
// Grid origin per indexed dim, passed to kernels by value.
template <typename T>
struct MinVals {
    T v[kMaxK];
};
// `perm` (column of each dim) may be null where columns keep their order.
// Cell key per point (K = uint32_t when the grid has fewer than 2^32 cells)
// and the point ids 0..N-1.  *bad (zeroed by the caller) is raised when a
// point's cell index reaches its dimension's extent.
template <typename T, typename K>
cudaError_t launch_cell_keys(const T* in, uint64_t N, uint32_t n, const uint32_t* perm, const GridGeom& g,
                             const MinVals<T>& minArr, T eps, K* keys, uint32_t* vals, uint32_t* bad,
                             cudaStream_t st);
template <typename T>
cudaError_t launch_gather_points(const T* in, uint64_t N, uint32_t n, uint32_t npad, const uint32_t* perm,
                                 const uint32_t* ids, T* pts, cudaStream_t st);
// Dense grids: the slot-prefix table ds[0 .. total] (16-byte aligned).  The
// others: the hash table of the grid rows that hold a cell (n0: the grid's
// cells in dim 0; all entries empty).
cudaError_t launch_dense_slots(const uint64_t* cell_key, const uint32_t* cell_start, uint32_t M, uint64_t total,
                               uint32_t* ds, cudaStream_t st);
cudaError_t launch_row_table(const uint64_t* cell_key, uint32_t M, uint32_t n0, uint4* htab, uint64_t hmask,
                             cudaStream_t st);
cudaError_t launch_cell_plan(const uint64_t* cell_key, uint32_t M, const GridGeom& g, const uint32_t* ds,
                             uint2* plan, cudaStream_t st);
// The same for the warp join on a hashed grid with k <= 3 (a: cell table, grid and
// neighbour offsets), the rows of the unicomp half-space with `stamp`.
// On fewer cells than kRowPlanCells the join's own warps have lanes and time for it,
// and the launch costs more than it gives (whole joins, us, without / with: 3-D float
// 2,000 cells 290 / 299, 4,000 352 / 370, 30,000 379 / 391, 100,000 445 / 445; double
// 2,000 274 / 284, 30,000 367 / 360, 100,000 488 / 433; 2-D double 30,000 356 / 338).
constexpr uint32_t kRowPlanCells = 32768;
template <typename T>
cudaError_t launch_row_plan(const JoinArgs<T>& a, bool stamp, uint2* plan, cudaStream_t st);
cudaError_t launch_item_counts(const uint32_t* cell_start, const uint32_t* order, uint32_t M, uint32_t qchunk,
                               uint32_t* nchunks, uint32_t* sizes, cudaStream_t st);
cudaError_t launch_make_items(const uint32_t* order, const uint32_t* nchunks, const uint32_t* item_off,
                              uint32_t M, uint2* items, cudaStream_t st);
// The 3^k neighbour offsets (JoinArgs::nbtab).
cudaError_t launch_neighbour_table(const GridGeom& g, uint32_t noff, uint4* tab, cudaStream_t st);
cudaError_t launch_iota(uint32_t* out, uint32_t M, cudaStream_t st);

// The warp-per-item join: appends packed pair keys into `o` (its rechecks
// counter receives the exact number of keys; with o.emit false only that
// count is taken) and visits items 0, o.stride, ..., (nvisit - 1) * o.stride.
// `model` is one of Model; `stamp` selects the unicomp traversal.  heavy.count
// and heavy.claim must be zero.  The launcher picks the specialisation.
struct TileOut;
// Slices of the items that are too long for one warp: found by the first launch,
// processed by a second one.  The items that find the list full are processed
// where they are found.
struct HeavyList {
    uint2* list;                // [cap] (visit, slice)
    unsigned long long* count;  // slices found, the dropped ones of a full list included: a
                                // join may find more than 2^32
    uint32_t* claim;            // the second launch's work counter
    uint32_t cap;               // 1 .. kHeavyCap
    uint32_t unit;              // steps of a slice (join_unit_steps)
};
constexpr uint32_t kHeavyCap = 1u << 20;
uint32_t join_unit_steps(double cand, int num_sms);
struct WarpLaunch {
    int num_sms;
    cudaStream_t st;
    int* launches;    // advanced by the kernels launched
    uint64_t* warps;  // not null: nothing is launched, *warps = warps of the pass's launches
};
template <typename T>
cudaError_t launch_join_emit(const JoinArgs<T>& a, const TileOut& o, const HeavyList& heavy, uint32_t nvisit,
                             int model, bool stamp, const WarpLaunch& w);

// ROWS path: dense low-dimensional grids (k <= 3, n <= 4), full neighbourhood.
// slot_cell[s] = cell of slot s; a.plan holds 3^(k-1) rows a cell.
// Count pass (a.work_counter zeroed): counts_by_id[ids[s]] = list length.
template <typename T>
cudaError_t launch_rows_count(const JoinArgs<T>& a, const uint32_t* slot_cell, uint32_t* counts_by_id, int num_sms,
                              cudaStream_t st);
// Fill pass (a.work_counter zeroed, a.offsets/table/table_cap/err_flag set):
// the lists of the queries at slots qslots[0 .. nq) (slots 0 .. nq-1 when
// qslots is null) into the point-id-ordered table; the list of point id i lands
// at a.table[offsets[i] - base].  pairs, cands: the whole join's result pairs and
// candidates, which choose the kernel.
template <typename T>
cudaError_t launch_rows_fill(const JoinArgs<T>& a, const uint32_t* slot_cell, const uint32_t* qslots, uint32_t nq,
                             uint64_t base, uint64_t pairs, uint64_t cands, int num_sms, cudaStream_t st);
// Result batches by point-id range: bound[0..nb] (ids) and boff[0..nb] (their
// table offsets), each batch's lists at most `step` + the longest list
// entries; per-slot batch keys (with the slot index as value, for a stable
// sort by batch); the start of each batch in the sorted slot list.
cudaError_t launch_batch_bounds(const uint64_t* offsets, uint32_t N, uint64_t step, uint32_t nb, uint32_t* bound,
                                unsigned long long* boff, cudaStream_t st);
cudaError_t launch_slot_batch(const uint32_t* ids, uint32_t N, const uint32_t* bound, uint32_t nb, uint32_t* bkey,
                              uint32_t* slot, cudaStream_t st);
cudaError_t launch_group_starts(const uint32_t* sorted_bkey, uint32_t N, uint32_t nb, uint32_t* gstart,
                                cudaStream_t st);
// *out = max of in[0 .. n) (*out zeroed by the caller).
cudaError_t launch_max_u32(const uint32_t* in, uint64_t n, uint32_t* out, cudaStream_t st);

// SORT variant (gsj_join_sort.cu): a count pass (fill == false: list lengths
// into counts_by_id, candidates into a.cand_cnt) and a fill pass (a.offsets,
// a.table, a.err_flag set) of the reference's pruned per-cell scans; the
// points of each cell must be in sort-dimension order.  `model` is one of Model.
template <typename T>
cudaError_t launch_sort_join(const JoinArgs<T>& a, const uint32_t* slot_cell, uint32_t* counts_by_id, int model,
                             bool fill, int num_sms, cudaStream_t st);
// out[s] = in[ids[s] * n + col]: the sort dimension's values in slot order.
template <typename T>
cudaError_t launch_sort_values(const T* in, uint64_t N, uint32_t n, uint32_t col, const uint32_t* ids, T* out,
                               cudaStream_t st);

// Tile join of high-dimensional float data (5 <= n <= kTileMaxN, k <= 6):
// a CTA per item of up to kTileQ query slots; hits become packed
// (query id << shift | candidate id) keys in a pair buffer.
constexpr int kTileQ = 64;            // queries per tile-join work item
constexpr uint32_t kTileMaxN = 128;   // dimensions held in shared memory
struct TileOut {
    unsigned long long* pairs;    // [cap] packed pairs
    unsigned long long cap;       // pairs beyond cap are counted, not written
    unsigned long long* cursor;   // pairs found so far (zeroed by the caller)
    uint32_t shift;               // bits of a point id
    uint32_t stride;              // items visited: 0, stride, 2*stride, ...
    bool emit;                    // false: count only (the sampling pass)
    unsigned long long* rechecks; // screened join: pairs sent to the exact check
};
bool tile_supported(uint32_t n, uint32_t npad, uint32_t k, int model, uint32_t ilp);
// Visits items 0, stride, ..., (nvisit-1)*stride; a.work_counter must be zero.
cudaError_t launch_tile_join(const JoinArgs<float>& a, const TileOut& o, bool stamp, int model, uint32_t nvisit,
                             int num_sms, cudaStream_t st);

// Tensor-core screened tile join (gsj_join_screen.cu): BF16 tcgen05 dot
// products with a proven rejection bound, exact FP32 check of the rest.
constexpr int kScreenQ = 128;         // queries per screened work item (MMA M)
constexpr uint32_t kScreenPathDims = 16;  // a screened join reports GSJ_PATH_SCREEN from here on, GSJ_PATH_TILE below
struct ScreenConst {
    float r0;             // >= sqrt(thr) with the reference sum's rounding room
    float c1, c0;         // FP32 accumulation bound per unit squared norm, per unit r0^2
    uint32_t kpad;        // dimensions + 4 padded to the MMA K step (16)
    const uint4* rows;    // [ceil(N/8)][kpad/8][8] BF16 rows in groups of 8 slots (gsj_join_screen.cu)
    const uint32_t* qg;   // [N] the query side's (-G_hi, -G_lo), packed BF16
};
// BF16 rows and query terms of all points (slot order) for the screen: centre
// = per-dimension mean of the finite values (deterministic two-level FP64
// sum); `partial` holds kScreenPrepBlocks x n x 2 doubles, `centre` n floats,
// `rows` screen_rows_count(N, kpad) uint4s.
constexpr uint32_t kScreenPrepBlocks = 592;
uint64_t screen_rows_count(uint64_t N, uint32_t kpad);
cudaError_t launch_screen_prep(const float* pts, uint32_t N, uint32_t n, uint32_t npad, const ScreenConst& sc,
                               double* partial, float* centre, uint4* rows, uint32_t* qg, cudaStream_t st);
bool screen_supported(uint32_t n, uint32_t npad, uint32_t k, int model, uint32_t ilp, float thr);
ScreenConst make_screen_const(uint32_t n, float thr);
// Screen pass: the undecided pairs go to o.pairs as 16-byte records {query
// slot, slot of column 0, mask of 32 columns, mask of the columns outside the
// query's cell (unicomp)}, in blocks of kScreenBlock records that consumer warps
// reserve on o.cursor and fill one after another; a block's end that cannot take
// all records of a warp's 32 queries (up to 31) stays unused (mask 0); o.cap
// counts records; o.rechecks receives the exact number of undecided pairs.
// Without emission o.cursor receives the number of records.
constexpr uint32_t kScreenBlock = 256;
// Keys of the warp join: its warps reserve blocks of kKeyBlock entries; the unused
// tails hold kKeyPad, which no key equals.
constexpr unsigned long long kKeyPad = ~0ull;
constexpr uint64_t kKeyBlock = 1024;
cudaError_t launch_tile_screen(const JoinArgs<float>& a, const TileOut& o, const ScreenConst& sc, bool stamp,
                               int model, uint32_t nvisit, int num_sms, cudaStream_t st);
// Exact check of the undecided pairs; hits go to o as packed (query id, candidate id) keys.
cudaError_t launch_screen_recheck(const JoinArgs<float>& a, const uint4* recs, unsigned long long nrec,
                                  const TileOut& o, bool stamp, int model, int num_sms, cudaStream_t st);

// Brute-force neighbour counts over all N^2 pairs (the reference's algorithm
// 1, kernel.cu:486-515) with the sequential model: counts[q] and the total.
template <typename T>
cudaError_t launch_bruteforce(const T* pts, uint32_t N, uint32_t n, T thr, uint32_t* counts,
                              unsigned long long* total, cudaStream_t st);

}  // namespace gsj
