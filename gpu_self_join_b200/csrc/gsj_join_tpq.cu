// Join of dense low-dimensional grids (k <= 3, n <= 4): the ROWS path.
//
// Low-dimensional workloads have tiny cells (a 2-D mixture of 20M points
// averages 3 points per non-empty cell), so any per-cell set-up done by a
// whole warp costs more than the distance tests.  Each query's candidates are
// the 3^(k-1) contiguous slot ranges of its cell plan (k_cell_plan), the full
// neighbourhood of kernel.cu:292-302, taken in a fixed order: candidate f of
// query s is the f-th slot of the concatenated ranges.
//
// k_rows_join takes 32 consecutive query slots a warp (a few cells) and cell by
// cell puts 128 candidates of the cell in the lanes' registers, coordinates and
// ids, four a lane; every query of the cell is then tested against 32 candidates
// at a time, a vote giving the hits.  The count pass adds up the votes; the fill
// pass, which runs once the lists have their places, repeats the tests and lets
// the lanes with a hit store their ids to consecutive list places.
//
// Repeating the test (4 instructions in 2-D) costs less than keeping its result:
// the earlier form had the count pass record every decision as a bit (a thread
// per query, 60 % of the lanes active, since neighbouring queries have candidate
// rows of different lengths) and the fill pass replay the bits of two queries a
// warp step, loading each hit's id on its own; the masks also needed a per-slot
// layout (a pass over the cells and a scan), 0.5 GB of traffic and a host
// read-back of their size between the index and the join.  Bound by instruction
// issue (0.77 of the slots in the fill).  Measured, count + fill (and the mask
// layout before): 2-D 20M points 1.28 + 3.00 + 0.23 -> 0.93 + 2.80 ms; 3-D
// double 250k 0.120 + 0.126 -> 0.080 + 0.101 ms.  Four CTAs an SM (64 registers)
// for float: 2-D 20M 3.03 / 2.80 / 3.01 / 2.80 ms with 3 / 4 / 5 / 6; double
// spills there (3-D 250k 0.101 / 0.114 with 2 / 4).
//
// Sparse cells leave most of a warp's lanes without a candidate and pay the cell's
// set-up for one or two queries: k_rows_thread, a thread per query, takes their
// count and, for short lists, their fill (launch_rows has the lines and both sides).
// Against the passes with masks, whole joins on the device: 3-D double 5M points at 1.6 a cell 1.87
// -> 1.29 ms, 2-D 10M at 1.2 2.08 -> 1.68, 4-D with 2 dims indexed 500k at 600 2.99 ->
// 2.68; 2-D at 2 to 3 points a cell is 4 % above them.
// The chunks are claimed dynamically (one atomic per warp, the next claim
// issued before the current chunk is processed), since chunk costs vary with the
// local density by orders of magnitude.
#include <cstdint>
#include <cuda_runtime.h>
#include <type_traits>

#include "gsj_common.cuh"
#include "gsj_dist.cuh"
#include "gsj_fp.cuh"
#include "gsj_kernels.h"

namespace gsj {

namespace {

// Next 32-slot chunk of the warp (lane 0 claims; the caller broadcasts it).
__device__ __forceinline__ uint32_t claim32(uint32_t* ctr, int lane) {
    uint32_t v = 0;
    if (lane == 0) v = atomicAdd(ctr, 32u);
    return v;
}

}  // namespace

// Coordinates of one point row (NT values of a row padded to npad = 1, 2 or
// 4 entries, so the vector forms are aligned).
template <typename T, int NT>
__device__ __forceinline__ void load_row(const T* __restrict__ p, T (&r)[NT]) {
    if constexpr (std::is_same<T, float>::value && NT == 2) {
        const float2 v = *reinterpret_cast<const float2*>(p);
        r[0] = v.x;
        r[1] = v.y;
    } else if constexpr (std::is_same<T, float>::value && NT >= 3) {
        const float4 v = *reinterpret_cast<const float4*>(p);
        r[0] = v.x;
        r[1] = v.y;
        r[2] = v.z;
        if constexpr (NT == 4) r[3] = v.w;
    } else if constexpr (std::is_same<T, double>::value && NT >= 2) {
        const double2 v = *reinterpret_cast<const double2*>(p);
        r[0] = v.x;
        r[1] = v.y;
        if constexpr (NT >= 3) {
            const double2 w = *reinterpret_cast<const double2*>(p + 2);
            r[2] = w.x;
            if constexpr (NT == 4) r[3] = w.y;
        }
    } else {
#pragma unroll
        for (int l = 0; l < NT; l++) r[l] = p[l];
    }
}

template <typename T>
__device__ __forceinline__ T quiet_nan();
template <>
__device__ __forceinline__ float quiet_nan<float>() {
    return __int_as_float(0x7fffffff);
}
template <>
__device__ __forceinline__ double quiet_nan<double>() {
    return __longlong_as_double(0x7fffffffffffffffll);
}

// k_rows_join's passes: the count, and the fill where many or few of the candidates
// are within eps.
enum RowsPass : int { kCountOnly = 0, kFill = 1, kFillFew = 2 };

// Where a query's list goes: read back with one 16-byte broadcast.
struct alignas(16) FillList {
    unsigned long long dst;
    uint32_t len, pad;
};

// Queries: the slots qslots[0 .. nq) (slots 0 .. nq-1 when qslots is null).
// Count pass: counts_by_id[id] = list length.  Fill pass: the list of point id i
// goes to a.table[offsets[i] - base]; a list that would leave the table or
// differ from its counted length raises *err_flag and is not written past it.
template <typename T, int NT, int NR, int POL, int FILL>
__global__ void __launch_bounds__(256, sizeof(T) == 4 ? 4 : 1) k_rows_join(const JoinArgs<T> a, const uint32_t* __restrict__ slot_cell,
                                                   uint32_t* __restrict__ counts_by_id,
                                                   const uint32_t* __restrict__ qslots, uint32_t nq, uint64_t base) {
    constexpr int G = 4;                             // candidates a lane holds
    static_assert(G == 4, "the tile counts below");
    __shared__ T sq[8][32 * NT];                     // the chunk's query rows (blockDim.x <= 256)
    __shared__ FillList slist[FILL ? 8 : 1][32];
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned lt;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(lt));
    const uint32_t npad = a.npad;
    const T thr = a.thr;
    unsigned long long cand = 0;
    uint32_t cur = __shfl_sync(FULL, claim32(a.work_counter, lane), 0);
    while (cur < nq) {
        const uint32_t nxt = claim32(a.work_counter, lane);  // in flight while this chunk runs
        const uint32_t nv = min(32u, nq - cur);
        const bool valid = (uint32_t)lane < nv;
        const uint32_t s = valid ? (qslots ? qslots[cur + (uint32_t)lane] : cur + (uint32_t)lane) : 0u;
        const uint32_t id = a.ids[s];
        const uint32_t cell = valid ? slot_cell[s] : 0xffffffffu;
        T own[NT];
        load_row<T, NT>(a.pts + (size_t)s * npad, own);
        uint32_t len = 0;
        uint2 e[NR <= 3 ? NR : 1];
        if (NR <= 3) {
#pragma unroll
            for (int r = 0; r < (NR <= 3 ? NR : 1); r++)
                e[r] = valid ? a.plan[(size_t)cell * NR + r] : make_uint2(0u, 0u);
        }
        __syncwarp();  // the previous chunk's reads of the staging are done
#pragma unroll
        for (int l = 0; l < NT; l++) sq[warp][lane * NT + l] = own[l];
        if (FILL) {
            unsigned long long dst = 0;
            if (valid) {
                dst = a.offsets[id] - base;
                len = (uint32_t)(a.offsets[id + 1] - a.offsets[id]);
                if (dst + len > a.table_cap) {
                    *a.err_flag = 1u;
                    len = 0u;
                }
            }
            slist[warp][lane] = FillList{dst, len, 0u};
        }
        __syncwarp();
        const uint32_t prev = __shfl_up_sync(FULL, cell, 1);
        unsigned heads = __ballot_sync(FULL, valid && (lane == 0 || cell != prev));
        uint32_t run = 0;  // hits of this lane's query so far
        while (heads) {
            // queries [j0, j1) of one cell
            const uint32_t j0 = (uint32_t)__ffs(heads) - 1u;
            heads &= heads - 1u;
            const uint32_t j1 = heads ? (uint32_t)__ffs(heads) - 1u : nv;
            // candidate f is slot f + adj[r] of the last row r with pre[r] <= f
            uint32_t adj[NR], pre[NR], total = 0;
            uint2 er = make_uint2(0u, 0u);
            if (NR > 3) {
                const uint32_t c = __shfl_sync(FULL, cell, (int)j0);
                if (lane < NR) er = a.plan[(size_t)c * NR + lane];
            }
#pragma unroll
            for (int r = 0; r < NR; r++) {
                const uint32_t st = __shfl_sync(FULL, NR <= 3 ? e[NR <= 3 ? r : 0].x : er.x, NR <= 3 ? (int)j0 : r);
                const uint32_t n = __shfl_sync(FULL, NR <= 3 ? e[NR <= 3 ? r : 0].y : er.y, NR <= 3 ? (int)j0 : r);
                pre[r] = total;
                adj[r] = st - total;
                total += n;
            }
            if (!FILL) cand += (unsigned long long)total * (j1 - j0);
            for (uint32_t f0 = 0; f0 < total; f0 += 32u * G) {
                T cx[G][NT];
                uint32_t cid[G];
#pragma unroll
                for (int t = 0; t < G; t++) {
                    const uint32_t f = f0 + 32u * (uint32_t)t + (uint32_t)lane;
                    uint32_t d = adj[0];
#pragma unroll
                    for (int r = 1; r < NR; r++)
                        if (f >= pre[r]) d = adj[r];
                    const bool in = f < total;
                    if (f0 + 32u * (uint32_t)t < total) {
                        const uint32_t slot = in ? f + d : s;
                        load_row<T, NT>(a.pts + (size_t)slot * npad, cx[t]);
                        if (FILL) cid[t] = FILL == kFillFew ? slot : a.ids[slot];
                        if (!in) cx[t][0] = quiet_nan<T>();  // within no threshold
                    }
                }
                // the cell's queries against the group's W tiles of 32 candidates
                auto test = [&](auto tiles) {
                    constexpr int W = decltype(tiles)::value;
                    for (uint32_t j = j0; j < j1; j++) {
                        T q[NT];
#pragma unroll
                        for (int l = 0; l < NT; l++) q[l] = sq[warp][j * NT + l];
                        if (FILL == kFillFew) {
                            bool any = false;
#pragma unroll
                            for (int t = 0; t < W; t++) any |= sqdist_seq_reg<T, NT, POL>(q, cx[t]) <= thr;
                            if (!__any_sync(FULL, any)) continue;
                        }
                        uint32_t rj = f0 ? __shfl_sync(FULL, run, (int)j) : 0u;
                        FillList fl{};
                        if (FILL) fl = slist[FILL ? warp : 0][j];
                        uint32_t* list = FILL ? a.table + fl.dst : nullptr;
#pragma unroll
                        for (int t = 0; t < W; t++) {
                            const bool hit = sqdist_seq_reg<T, NT, POL>(q, cx[t]) <= thr;
                            const unsigned b = __ballot_sync(FULL, hit);
                            if (FILL) {
                                const uint32_t pos = rj + (uint32_t)__popc(b & lt);
                                if (hit && pos < fl.len) list[pos] = FILL == kFillFew ? a.ids[cid[t]] : cid[t];
                            }
                            rj += (uint32_t)__popc(b);
                        }
                        if ((uint32_t)lane == j) run = rj;
                    }
                };
                const uint32_t left = total - f0;
                if (left > 96u) test(std::integral_constant<int, 4>{});
                else if (left > 64u) test(std::integral_constant<int, 3>{});
                else if (left > 32u) test(std::integral_constant<int, 2>{});
                else test(std::integral_constant<int, 1>{});
            }
        }
        if (FILL) {
            if (valid && run != len) *a.err_flag = 1u;
        } else if (valid) {
            counts_by_id[id] = run;
        }
        cur = __shfl_sync(FULL, nxt, 0);
    }
    if (!FILL && lane == 0 && cand) atomicAdd(a.cand_cnt, cand);
}

// A thread per query: the slots of a warp are consecutive in cell order, so lanes
// of one cell walk the same ranges (broadcast loads).  Passes as for k_rows_join.
template <typename T, int NT, int NR, int POL, bool FILL>
__global__ void __launch_bounds__(256) k_rows_thread(const JoinArgs<T> a, const uint32_t* __restrict__ slot_cell,
                                                     uint32_t* __restrict__ counts_by_id,
                                                     const uint32_t* __restrict__ qslots, uint32_t nq, uint64_t base) {
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const uint32_t npad = a.npad;
    const T thr = a.thr;
    unsigned long long cand = 0;
    uint32_t cur = __shfl_sync(FULL, claim32(a.work_counter, lane), 0);
    while (cur < nq) {
        const uint32_t nxt = claim32(a.work_counter, lane);  // in flight while this chunk runs
        const uint32_t i = cur + (uint32_t)lane;
        if (i < nq) {
            const uint32_t s = FILL && qslots ? qslots[i] : i;
            const uint32_t cell = slot_cell[s];
            T q[NT];
            load_row<T, NT>(a.pts + (size_t)s * npad, q);
            uint32_t cnt = 0, len = 0;
            uint32_t* list = nullptr;
            if (FILL) {
                const uint32_t id = a.ids[s];
                const unsigned long long dst = a.offsets[id] - base;
                len = (uint32_t)(a.offsets[id + 1] - a.offsets[id]);
                if (dst + len > a.table_cap) {
                    *a.err_flag = 1u;
                    len = 0u;
                }
                list = a.table + dst;
            }
#pragma unroll
            for (int r = 0; r < NR; r++) {
                const uint2 e = a.plan[(size_t)cell * NR + r];
                const T* cp = a.pts + (size_t)e.x * npad;
                if (!FILL) cand += e.y;
#pragma unroll 4
                for (uint32_t u = 0; u < e.y; u++) {
                    T cr[NT];
                    load_row<T, NT>(cp, cr);
                    cp += npad;
                    const bool hit = sqdist_seq_reg<T, NT, POL>(q, cr) <= thr;
                    if (FILL && hit && cnt < len) list[cnt] = a.ids[e.x + u];
                    cnt += hit ? 1u : 0u;
                }
            }
            if (!FILL) counts_by_id[a.ids[s]] = cnt;
            else if (cnt != len) *a.err_flag = 1u;
        }
        cur = __shfl_sync(FULL, nxt, 0);
    }
    if (FILL) return;
    // one atomic per warp for the candidate statistic
    for (int o = 16; o > 0; o >>= 1) cand += __shfl_down_sync(FULL, cand, o);
    if (lane == 0 && cand) atomicAdd(a.cand_cnt, cand);
}

// Resident CTAs of a kernel, for persistent grids.
static int resident_blocks(const void* kern, int threads, size_t smem, int num_sms) {
    int per_sm = 0;
    if (blocks_per_sm(kern, threads, smem, &per_sm) != cudaSuccess || per_sm < 1) per_sm = 1;
    return num_sms * per_sm;
}

// Launches one of the forms over nq queries.
template <typename T, typename K>
static cudaError_t launch_form(K kern, const JoinArgs<T>& a, const uint32_t* slot_cell, uint32_t* counts_by_id,
                               const uint32_t* qslots, uint32_t nq, uint64_t base, int num_sms, cudaStream_t st) {
    const int threads = a.shape_threads ? (int)a.shape_threads : 256;
    uint64_t blocks = (uint64_t)resident_blocks((const void*)kern, threads, 0, num_sms);
    const uint64_t needed = ((uint64_t)nq + threads - 1) / threads;
    if (blocks > needed) blocks = needed ? needed : 1;
    kern<<<(unsigned)blocks, threads, 0, st>>>(a, slot_cell, counts_by_id, qslots, nq, base);
    return cudaGetLastError();
}

// From about this many queries on a thread per query fills the chip (148 SMs hold
// 303,104 threads): the lines below were drawn on both sides of it, from 3,000
// points to 4 million.
constexpr uint32_t kManyQueries = 400000u;

template <typename T, int NT, int NR, bool FILL>
static cudaError_t launch_rows(const JoinArgs<T>& a, const uint32_t* slot_cell, uint32_t* counts_by_id,
                               const uint32_t* qslots, uint32_t nq, uint64_t base, uint64_t pairs, uint64_t cands,
                               int num_sms, cudaStream_t st) {
    constexpr int POL = sizeof(T) == 8 ? kPolF64 : kPolF32;
    if constexpr (!FILL) {
        // Sparse cells leave the lanes of k_rows_join's cells half empty and pay its
        // set-up for few queries.  Count pass, cell form / thread per query (ms, uniform
        // points, points a non-empty cell): nine rows: 3-D 2M at 5.0 0.293 / 0.267, 5.9 0.312 /
        // 0.306, 7.0 0.314 / 0.344, 250k at 4.0 0.057 / 0.053, 5.9 0.064 / 0.068, 4-D 1M at
        // 6.0 0.181 / 0.177, 6.8 0.189 / 0.195; in double 3-D 2M at 5.0 0.480 / 0.428, 5.9
        // 0.496 / 0.484, 250k at 3.1 0.074 / 0.068, 5.0 0.074 / 0.089, 4-D 1M at 4.1 0.234 /
        // 0.246.  Three rows: 2-D 4M at 7.0 0.228 / 0.158, 10 0.226 / 0.195, in double at 7.0
        // 0.269 / 0.250, 8.0 0.271 / 0.277, a 2-D mixture 8M at 9.1 1.14 / 1.18; 4-D 1M at 6.0 0.080 / 0.074, 7.0 0.080 / 0.082, in
        // double at 6.0 0.119 / 0.119.  One row: 1-D 4M at 10 0.129 / 0.119, in double 0.160 /
        // 0.123.  Fewer points than the chip holds threads for leave a thread's serial
        // candidates in plain sight, in double above all: us for 3-D double 10k at 3.8 31.0 /
        // 37.1, 100k at 3.9 47.3 / 47.2, at 4.8 47.4 / 51.4, 2-D double 10k at 5.0 14.5 / 16.4,
        // 300k at 6.0 32.8 / 35.2; 3-D float 10k at 5.8 22.8 / 20.6, 300k at 5.9 65.6 / 67.9.
        const bool many = a.n_points >= kManyQueries;
        const uint32_t line = sizeof(T) == 8 ? (many ? (NR == 9 ? 5u : NR == 1 ? 10u : NT <= 2 ? 7u : 6u)
                                                     : (NR == 9 ? 4u : 5u))
                              : NR == 1      ? (many ? 10u : 7u)
                              : NR == 3 && NT <= 2 ? 8u
                                                   : 6u;
        if (a.n_points < line * (uint64_t)a.num_cells)
            return launch_form<T>(k_rows_thread<T, NT, NR, POL, false>, a, slot_cell, counts_by_id, qslots, nq, base,
                                  num_sms, st);
        return launch_form<T>(k_rows_join<T, NT, NR, POL, kCountOnly>, a, slot_cell, counts_by_id, qslots, nq, base,
                              num_sms, st);
    } else {
        const uint64_t N = a.n_points;
        // Fill pass, cell form against thread per query (ms): 2-D 4M points, 1.6 a cell
        // and 4.1 result pairs a point 0.497 / 0.277, 2.3 and 7.3 0.402 / 0.418, 3.2 and
        // 10.4 0.361 / 0.542; 3-D 2M at 1.6 and 5.2 0.359 / 0.201, 3.1 and 13.4 0.369 /
        // 0.348, 4.0 and 17.5 0.403 / 0.437 (double 1.6 0.620 / 0.262); 1-D 4M at 2.3
        // and 5.2 0.324 / 0.292, 4.1 and 9.2 0.259 / 0.482.  So sparse cells take a
        // thread per query while it stores few ids, each to a sector of its own; with
        // many candidates a point (4-D 500k, 130 of them and 1.5 pairs: 0.145 / 0.148,
        // double 0.162 / 0.195) the cell form is the better one again, and on fewer points
        // sooner (us; 3-D 100k, 28 candidates and 5.1 pairs 53.8 / 48.0, 54 and 9.1 51.7 /
        // 58.3, in double 51.5 / 53.3 and 49.3 / 65.7; 2-D 100k, 19 and 7.3 33.5 / 24.6).
        const bool many = N >= kManyQueries;
        if (N < (sizeof(T) == 8 ? 5u : 7u) * (uint64_t)a.num_cells &&
            pairs <= (NR == 1 ? 6u : NR == 3 ? 7u : many ? 14u : 6u) * N && cands <= (many ? 96u : 32u) * N)
            return launch_form<T>(k_rows_thread<T, NT, NR, POL, true>, a, slot_cell, counts_by_id, qslots, nq, base,
                                  num_sms, st);
        // Where few candidates are within eps one vote a query skips four tiles, and an id
        // is loaded for a hit alone.  Every candidate's id / the hits' ids, by the share
        // of hits: 4-D 500k 0.0009 2.36 / 1.23 ms, 0.0084 0.348 / 0.286, 0.0117 0.145 /
        // 0.144, 0.022 0.068 / 0.070, 2-D 4M 0.36 0.46 / 0.54; double 4-D 0.0009 2.64 /
        // 2.21, 2-D 0.0021 0.247 / 0.213, 0.0044 2.22 / 2.24, 0.0084 0.334 / 0.392.
        if (pairs * (sizeof(T) == 8 ? 256u : 64u) < cands)
            return launch_form<T>(k_rows_join<T, NT, NR, POL, kFillFew>, a, slot_cell, counts_by_id, qslots, nq, base,
                                  num_sms, st);
        return launch_form<T>(k_rows_join<T, NT, NR, POL, kFill>, a, slot_cell, counts_by_id, qslots, nq, base,
                              num_sms, st);
    }
}

template <typename T, int NR, bool FILL>
static cudaError_t rows_nr(const JoinArgs<T>& a, const uint32_t* slot_cell, uint32_t* counts_by_id,
                           const uint32_t* qslots, uint32_t nq, uint64_t base, uint64_t pairs, uint64_t cands,
                           int num_sms, cudaStream_t st) {
    switch (a.n) {
        case 1: return launch_rows<T, 1, NR, FILL>(a, slot_cell, counts_by_id, qslots, nq, base, pairs, cands, num_sms, st);
        case 2: return launch_rows<T, 2, NR, FILL>(a, slot_cell, counts_by_id, qslots, nq, base, pairs, cands, num_sms, st);
        case 3: return launch_rows<T, 3, NR, FILL>(a, slot_cell, counts_by_id, qslots, nq, base, pairs, cands, num_sms, st);
        case 4: return launch_rows<T, 4, NR, FILL>(a, slot_cell, counts_by_id, qslots, nq, base, pairs, cands, num_sms, st);
        default: return cudaErrorInvalidValue;
    }
}

template <typename T, bool FILL>
static cudaError_t rows_any(const JoinArgs<T>& a, const uint32_t* slot_cell, uint32_t* counts_by_id,
                            const uint32_t* qslots, uint32_t nq, uint64_t base, uint64_t pairs, uint64_t cands,
                            int num_sms, cudaStream_t st) {
    if (a.n < 1 || a.n > 4 || a.ilp != 0 || a.g.k > 3 || !a.plan) return cudaErrorInvalidValue;
    if (nq == 0) return cudaSuccess;
    if (a.g.k == 1) return rows_nr<T, 1, FILL>(a, slot_cell, counts_by_id, qslots, nq, base, pairs, cands, num_sms, st);
    if (a.g.k == 2) return rows_nr<T, 3, FILL>(a, slot_cell, counts_by_id, qslots, nq, base, pairs, cands, num_sms, st);
    return rows_nr<T, 9, FILL>(a, slot_cell, counts_by_id, qslots, nq, base, pairs, cands, num_sms, st);
}

template <typename T>
cudaError_t launch_rows_count(const JoinArgs<T>& a, const uint32_t* slot_cell, uint32_t* counts_by_id, int num_sms,
                              cudaStream_t st) {
    return rows_any<T, false>(a, slot_cell, counts_by_id, nullptr, a.n_points, 0, 0, 0, num_sms, st);
}

template <typename T>
cudaError_t launch_rows_fill(const JoinArgs<T>& a, const uint32_t* slot_cell, const uint32_t* qslots, uint32_t nq,
                             uint64_t base, uint64_t pairs, uint64_t cands, int num_sms, cudaStream_t st) {
    return rows_any<T, true>(a, slot_cell, nullptr, qslots, nq, base, pairs, cands, num_sms, st);
}

template cudaError_t launch_rows_count<float>(const JoinArgs<float>&, const uint32_t*, uint32_t*, int, cudaStream_t);
template cudaError_t launch_rows_count<double>(const JoinArgs<double>&, const uint32_t*, uint32_t*, int,
                                               cudaStream_t);
template cudaError_t launch_rows_fill<float>(const JoinArgs<float>&, const uint32_t*, const uint32_t*, uint32_t,
                                             uint64_t, uint64_t, uint64_t, int, cudaStream_t);
template cudaError_t launch_rows_fill<double>(const JoinArgs<double>&, const uint32_t*, const uint32_t*, uint32_t,
                                              uint64_t, uint64_t, uint64_t, int, cudaStream_t);

// ---------------------------------------------------------------- result batches
// Batch b of the host-result pipeline holds the point ids [bound[b],
// bound[b+1]): its lists are the table range [boff[b], boff[b+1]) with boff[b]
// = offsets[bound[b]].  bound[b] = the last id whose list starts at or below
// b * step, so with step = segment capacity minus the longest list every batch
// fits one segment; bound[0] = 0, bound[nb] = N.
__global__ void k_batch_bounds(const uint64_t* __restrict__ offsets, uint32_t N, uint64_t step, uint32_t nb,
                               uint32_t* __restrict__ bound, unsigned long long* __restrict__ boff) {
    const uint32_t b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b > nb) return;
    if (b == 0 || b == nb) {
        bound[b] = b == 0 ? 0u : N;
        boff[b] = b == 0 ? 0ull : offsets[N];
        return;
    }
    const unsigned long long target = (unsigned long long)b * step;
    uint32_t lo = 0, hi = N;  // first i in [0, N) with offsets[i] > target (N if none)
    while (lo < hi) {
        const uint32_t mid = lo + (hi - lo) / 2u;
        if (offsets[mid] > target) hi = mid;
        else lo = mid + 1u;
    }
    bound[b] = lo > 0 ? lo - 1u : 0u;
    boff[b] = offsets[bound[b]];
}

// Batch index of every slot's point id (binary search over the bounds), and
// the slot index as the value of the stable sort by batch.
__global__ void k_slot_batch(const uint32_t* __restrict__ ids, uint32_t N, const uint32_t* __restrict__ bound,
                             uint32_t nb, uint32_t* __restrict__ bkey, uint32_t* __restrict__ slot) {
    const uint32_t s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= N) return;
    const uint32_t id = ids[s];
    uint32_t lo = 0, hi = nb;  // last b with bound[b] <= id
    while (hi - lo > 1u) {
        const uint32_t mid = (lo + hi) / 2u;
        if (bound[mid] <= id) lo = mid;
        else hi = mid;
    }
    bkey[s] = lo;
    slot[s] = s;
}

// Start of each batch's slots in the batch-sorted slot list: gstart[b] =
// first position whose batch key is >= b, gstart[nb] = N.
__global__ void k_group_starts(const uint32_t* __restrict__ sorted_bkey, uint32_t N, uint32_t nb,
                               uint32_t* __restrict__ gstart) {
    const uint32_t b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b > nb) return;
    uint32_t lo = 0, hi = N;
    while (lo < hi) {
        const uint32_t mid = lo + (hi - lo) / 2u;
        if (sorted_bkey[mid] >= b) hi = mid;
        else lo = mid + 1u;
    }
    gstart[b] = lo;
}

// *out = max(in[0 .. n)) (*out zeroed by the caller).
__global__ void k_max_u32(const uint32_t* __restrict__ in, uint64_t n, uint32_t* __restrict__ out) {
    uint32_t m = 0;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
        m = max(m, in[i]);
    for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_down_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0 && m) atomicMax(out, m);
}

cudaError_t launch_batch_bounds(const uint64_t* offsets, uint32_t N, uint64_t step, uint32_t nb, uint32_t* bound,
                                unsigned long long* boff, cudaStream_t st) {
    k_batch_bounds<<<(nb + 1 + 127) / 128, 128, 0, st>>>(offsets, N, step, nb, bound, boff);
    return cudaGetLastError();
}

cudaError_t launch_slot_batch(const uint32_t* ids, uint32_t N, const uint32_t* bound, uint32_t nb, uint32_t* bkey,
                              uint32_t* slot, cudaStream_t st) {
    k_slot_batch<<<(N + 255) / 256, 256, 0, st>>>(ids, N, bound, nb, bkey, slot);
    return cudaGetLastError();
}

cudaError_t launch_group_starts(const uint32_t* sorted_bkey, uint32_t N, uint32_t nb, uint32_t* gstart,
                                cudaStream_t st) {
    k_group_starts<<<(nb + 1 + 127) / 128, 128, 0, st>>>(sorted_bkey, N, nb, gstart);
    return cudaGetLastError();
}

cudaError_t launch_max_u32(const uint32_t* in, uint64_t n, uint32_t* out, cudaStream_t st) {
    uint64_t blocks = (n + 255) / 256;
    if (blocks > 1184) blocks = 1184;
    k_max_u32<<<(unsigned)(blocks ? blocks : 1), 256, 0, st>>>(in, n, out);
    return cudaGetLastError();
}

}  // namespace gsj
