// Candidate-cell distance join (subsystem (b)).
//
// Replaces kernelNDGridIndexGlobal / evaluateCell / evalPoint
// (kernel.cu:132-480, kernelloops.h, stamploops.h).  The reference runs one
// thread per query point, repeats the neighbour-cell search (2 binary searches
// per cell) for every query, and appends every hit with a global atomicAdd.
// Here one warp owns a work item: up to 32 consecutive query slots of one
// non-empty cell.  The warp
//   1. enumerates the cell's 3^(k-1) neighbour rows once, lanes in parallel (a
//      row's up to three cells are one contiguous slot range, row_slots), and
//      compacts the non-empty ones (ballot) into a per-warp list in shared memory -
//      with STAMP only the unicomp half-space of stamploops.h;
//   2. stages the queries in shared memory;
//   3. walks the concatenated candidate slots 32 at a time, one candidate per
//      lane, and tests every query against the 32 candidates with the
//      reference's exact arithmetic (s <= thr is sqrt(s) <= eps, see
//      gsj_threshold_*).
// Every hit becomes a packed (query id, candidate id) key appended to the pair
// buffer, with STAMP also the reverse key of a hit in another cell (the
// reference emits (q,c) twice there, kernel.cu:367-375); the buffer becomes the
// neighbour table afterwards (the reference's pair buffers + sort_by_key,
// GPU.cu:863-980).  One traversal per join; a sampling run over every stride-th
// item sizes the buffer first.
//
// Two kernels: k_join_reg for float rows of up to 16 values (candidate rows in
// registers, hits through a per-warp queue, heavy items cut into slices), k_join
// for the rest (double, longer rows, ILP chains that a register form would have
// to reorder).
#include <algorithm>
#include <cstdint>
#include <cuda_runtime.h>

#include "gsj_common.cuh"
#include "gsj_fp.cuh"
#include "gsj_dist.cuh"
#include "gsj_kernels.h"

namespace gsj {

__device__ __forceinline__ unsigned lanemask_lt() {
    unsigned m;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}

__host__ __device__ constexpr uint32_t align16(uint32_t x) { return (x + 15u) & ~15u; }

__host__ __device__ constexpr uint32_t npad_for(uint32_t n, uint32_t tsize) {
    return n <= 2 ? n : ((n + (16u / tsize) - 1u) / (16u / tsize)) * (16u / tsize);
}

struct WarpSmem {
    uint32_t q_off, qid_off, nbs_off, nbp_off, cand_off, total;
};

__host__ __device__ inline WarpSmem warp_smem_layout(uint32_t npad, uint32_t tsize, uint32_t nb_cap, bool generic) {
    WarpSmem w{};
    uint32_t o = 0;
    w.q_off = o;
    o = align16(o + 32u * npad * tsize);
    w.qid_off = o;
    o = align16(o + 32u * 4u);
    w.nbs_off = o;
    o = align16(o + nb_cap * 4u);
    w.nbp_off = o;
    o = align16(o + (nb_cap + 1u) * 4u);
    w.cand_off = o;
    if (generic) o = align16(o + 32u * (npad + 1u) * tsize);
    w.total = o;
    return w;
}

// The warp appends its hits as packed (query id << shift |
// candidate id) keys, and with unicomp the reverse key of a hit in another
// cell, into blocks of kEmitBlk entries it reserves on o.cursor (unused tails
// padded with kKeyPad, which sorts after every key); emitted counts the
// keys exactly.  hit / cr are this lane's flags, b / cb their ballots.
constexpr uint32_t kEmitBlk = (uint32_t)kKeyBlock;

__device__ __forceinline__ void emit_keys(const TileOut& o, unsigned long long& blk_base, uint32_t& blk_used,
                                          unsigned long long& emitted, bool hit, bool cr, unsigned b, unsigned cb,
                                          unsigned lt, int lane, uint64_t qid, uint64_t cid) {
    const uint32_t cnt = (uint32_t)__popc(b) + (uint32_t)__popc(cb);
    emitted += cnt;
    if (!o.emit) return;
    if (blk_used + cnt > kEmitBlk) {
        for (uint32_t e = blk_used + (uint32_t)lane; e < kEmitBlk; e += 32u)
            if (blk_base + e < o.cap) o.pairs[blk_base + e] = kKeyPad;
        unsigned long long nb = 0;
        if (lane == 0) nb = atomicAdd(o.cursor, (unsigned long long)kEmitBlk);
        blk_base = __shfl_sync(0xffffffffu, nb, 0);
        blk_used = 0;
    }
    if (hit) {
        unsigned long long p = blk_base + blk_used + (unsigned)__popc(b & lt) + (unsigned)__popc(cb & lt);
        if (p < o.cap) o.pairs[p] = (qid << o.shift) | cid;
        p++;
        if (cr && p < o.cap) o.pairs[p] = (cid << o.shift) | qid;
    }
    blk_used += cnt;
}

// Slot of candidate f = f0 + lane in the concatenated neighbour ranges
// (nb_pref: exclusive prefix of the range sizes, nb_pref[nnb] = total).  `ent`
// is the range holding f0 (warp-uniform).  Every range holds at least one
// candidate, so the warp's 32 candidates lie in ranges ent .. ent + 31: lane j
// loads nb_pref[ent + j] and each lane finds its range with a 5-step search
// over those values; `ent` then moves to the range of f0 + 32 (at most one
// range past lane 31's).
__device__ __forceinline__ uint32_t cand_slot(const uint32_t* nb_start, const uint32_t* nb_pref, uint32_t nnb,
                                              uint32_t& ent, uint32_t f0, uint32_t lane, uint32_t total) {
    const unsigned FULL = 0xffffffffu;
    const uint32_t f = f0 + lane;
    const uint32_t p = ent + lane <= nnb ? nb_pref[ent + lane] : 0xffffffffu;
    uint32_t lo = 0;
#pragma unroll
    for (uint32_t step = 16; step >= 1; step >>= 1) {
        const uint32_t c = lo + step;
        if (__shfl_sync(FULL, p, c) <= f) lo = c;
    }
    const uint32_t my = ent + lo;
    const uint32_t pf = __shfl_sync(FULL, p, lo);
    const uint32_t e31 = __shfl_sync(FULL, my, 31);
    ent = (e31 + 1u <= nnb && nb_pref[e31 + 1u] <= f0 + 32u) ? e31 + 1u : e31;
    return f < total ? nb_start[my] + (f - pf) : 0u;
}

// The neighbour rows of `cell` (first slot cs; kernel.cu:180-303; stamploops.h
// for STAMP) as slot ranges in nb_start and the exclusive prefix of their sizes
// in nb_pref (nb_pref[rows] = total).  Returns the number of rows; the whole
// warp calls.  PLAN: a.plan holds them (as a template argument: a branch on the
// pointer cost the 8-D register form 1 %).
template <typename T, bool STAMP, bool PLAN>
__device__ __forceinline__ uint32_t enumerate_rows(const JoinArgs<T>& a, uint32_t cell, uint32_t cs, uint32_t nrow,
                                                   uint32_t* nb_start, uint32_t* nb_pref, int lane, unsigned lt,
                                                   uint32_t& total) {
    const unsigned FULL = 0xffffffffu;
    if (PLAN) {  // at most 9 rows, looked up before (k_row_plan)
        uint2 e = make_uint2(0u, 0u);
        if ((uint32_t)lane < nrow) e = a.plan[(size_t)cell * nrow + (uint32_t)lane];
        const unsigned m = __ballot_sync(FULL, e.y != 0u);
        uint32_t x = e.y;
#pragma unroll
        for (int s = 1; s < 16; s <<= 1) {
            const uint32_t y = __shfl_up_sync(FULL, x, s);
            if (lane >= s) x += y;
        }
        total = __shfl_sync(FULL, x, 15);
        const uint32_t nnb = (uint32_t)__popc(m);
        if (e.y) {
            const uint32_t pos = (uint32_t)__popc(m & lt);
            nb_start[pos] = e.x;
            nb_pref[pos] = x - e.y;
        }
        if (lane == 0) nb_pref[nnb] = total;
        return nnb;
    }
    // own cell coordinates, from the first query of the cell with the formula the
    // keys were built with (main.cu:744, kernel.cu:184)
    uint32_t own[kMaxK];
#pragma unroll
    for (int j = 0; j < kMaxK; j++)
        own[j] = (j < (int)a.g.k) ? FP<T>::to_uint_rz(FP<T>::div(FP<T>::sub(a.pts[(size_t)cs * a.npad + j], a.minv[j]),
                                                                 a.eps))
                                  : 0u;
    uint32_t lowmask, highmask, oddmask;
    cell_masks(own, a.g, lowmask, highmask, oddmask);
    const uint64_t own_lin = a.cell_key[cell];
    uint32_t nnb = 0, run = 0;
    // the next round's first loads are in flight while a round is finished
    RowProbe next;
    neighbour_row<T, STAMP>(a, (uint32_t)lane < nrow, (uint32_t)lane, own_lin, own[0], lowmask, highmask, oddmask,
                            next);
    for (uint32_t b0 = 0; b0 < nrow; b0 += 32) {
        const uint32_t r = b0 + 32u + (uint32_t)lane;
        const RowProbe cur = next;
        neighbour_row<T, STAMP>(a, r < nrow, r, own_lin, own[0], lowmask, highmask, oddmask, next);
        uint32_t st, v;
        row_slots(a, cur, st, v);
        const unsigned m = __ballot_sync(FULL, v != 0u);
        uint32_t x = v;
#pragma unroll
        for (int s = 1; s < 32; s <<= 1) {
            const uint32_t y = __shfl_up_sync(FULL, x, s);
            if (lane >= s) x += y;
        }
        if (v) {
            const uint32_t pos = nnb + (uint32_t)__popc(m & lt);
            nb_start[pos] = st;
            nb_pref[pos] = run + x - v;
        }
        nnb += (uint32_t)__popc(m);
        run += __shfl_sync(FULL, x, 31);
    }
    if (lane == 0) nb_pref[nnb] = run;
    total = run;
    return nnb;
}

template <typename T, int NT, int MODEL, int POL, bool STAMP, bool PLAN>
__global__ void __launch_bounds__(256, sizeof(T) == 4 ? 4 : 1) k_join(const JoinArgs<T> a, uint32_t nrow,
                                                                       const TileOut o, uint32_t nvisit) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    constexpr bool GENERIC = (NT == 0);
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    const uint32_t npad = a.npad;
    const WarpSmem L = warp_smem_layout(npad, sizeof(T), nrow, GENERIC);
    unsigned char* wb = smem_raw + (size_t)warp * L.total;
    T* q_s = reinterpret_cast<T*>(wb + L.q_off);
    uint32_t* qid_s = reinterpret_cast<uint32_t*>(wb + L.qid_off);
    uint32_t* nb_start = reinterpret_cast<uint32_t*>(wb + L.nbs_off);
    uint32_t* nb_pref = reinterpret_cast<uint32_t*>(wb + L.nbp_off);
    T* cand_s = reinterpret_cast<T*>(wb + L.cand_off);
    const unsigned lt = lanemask_lt();
    unsigned long long cand_total = 0;
    unsigned long long blk_base = 0, emitted = 0;
    uint32_t blk_used = kEmitBlk;

    // Work items are claimed one at a time: items in cell order are as heavy
    // as their cells are dense, so claiming runs of consecutive items left one
    // warp with a run of the densest cells long after the others had finished
    // (on a 5M-point 6-D Gaussian mixture the heaviest run of 32 items held 7.5x
    // a warp's mean share).  The next claim is issued before the current item
    // is processed and read after it, so its latency hides behind the item.
    // Item i is items[i * o.stride] (a stride above 1 samples every stride-th item).
    uint32_t claim = 0;
    if (lane == 0) claim = atomicAdd(a.work_counter, 1u);
    for (;;) {
        const uint32_t item = __shfl_sync(FULL, claim, 0);
        if (item >= nvisit) break;
        if (lane == 0) claim = atomicAdd(a.work_counter, 1u);
        const uint2 wi = a.items[(size_t)item * o.stride];
        const uint32_t cs = a.cell_start[wi.x], ce = a.cell_start[wi.x + 1];
        const uint32_t q0 = cs + wi.y * kQChunk;
        const uint32_t qn = min((uint32_t)kQChunk, ce - q0);
        uint32_t total;
        const uint32_t nnb = enumerate_rows<T, STAMP, PLAN>(a, wi.x, cs, nrow, nb_start, nb_pref, lane, lt, total);

        // ---- queries
        for (uint32_t e = lane; e < qn * npad; e += 32) q_s[e] = a.pts[(size_t)q0 * npad + e];
        if (lane < qn) qid_s[lane] = a.ids[q0 + lane];
        __syncwarp();
        cand_total += (unsigned long long)total * qn;
        const uint64_t my_qid = lane < qn ? qid_s[lane] : 0u;

        if constexpr (!GENERIC) {
            // ---- register path (n <= 8): up to G tiles of 32 candidates live in
            // registers; queries outside, tiles inside, so each query's
            // coordinates are loaded once per group of tiles.
            constexpr int G = 4;
            constexpr int NR = NT > 0 ? NT : 1;
            uint32_t ent = 0;
            for (uint32_t g0 = 0; g0 < total; g0 += 32u * G) {
                T cx[G][NR];
                uint32_t cid[G];
                bool cval[G], ccross[G];
                const uint32_t ntile = min((uint32_t)G, (total - g0 + 31u) / 32u);
#pragma unroll
                for (int t = 0; t < G; t++) {
                    const uint32_t f = g0 + (uint32_t)t * 32u + lane;
                    cval[t] = f < total;
                    cid[t] = 0u;
                    ccross[t] = false;
                    if ((uint32_t)t >= ntile) continue;
                    const uint32_t slot = cand_slot(nb_start, nb_pref, nnb, ent, g0 + (uint32_t)t * 32u, lane, total);
                    if (cval[t]) cid[t] = a.ids[slot];
                    ccross[t] = STAMP && cval[t] && (slot < cs || slot >= ce);  // outside the own cell
                    const T* row = a.pts + (size_t)slot * npad;
#pragma unroll
                    for (int l = 0; l < NR; l++) cx[t][l] = row[l];
                }
                for (uint32_t j = 0; j < qn; j++) {
                    T q[NR];
#pragma unroll
                    for (int l = 0; l < NR; l++) q[l] = q_s[(size_t)j * npad + l];
                    const uint64_t qid = __shfl_sync(FULL, my_qid, j);
#pragma unroll
                    for (int t = 0; t < G; t++) {
                        if ((uint32_t)t < ntile) {
                            const T s = sqdist_seq_reg<T, NR, POL>(q, cx[t]);
                            const bool hit = cval[t] && (s <= a.thr);
                            const unsigned b = __ballot_sync(FULL, hit);
                            if (b) {
                                const bool cr = STAMP && ccross[t] && hit;
                                const unsigned cb = __ballot_sync(FULL, cr);
                                emit_keys(o, blk_base, blk_used, emitted, hit, cr, b, cb, lt, lane, qid, cid[t]);
                            }
                        }
                    }
                }
            }
        } else {
            // ---- generic n: one tile of 32 candidate rows staged in shared memory
            uint32_t ent = 0;
            for (uint32_t t0 = 0; t0 < total; t0 += 32) {
                const uint32_t f = t0 + lane;
                const bool valid = f < total;
                const uint32_t slot = cand_slot(nb_start, nb_pref, nnb, ent, t0, lane, total);
                uint32_t corig = 0;
                bool cross = false;
                if (valid) {
                    cross = STAMP && (slot < cs || slot >= ce);  // outside the own cell
                    corig = a.ids[slot];
                }
                {
                    const T* row = a.pts + (size_t)slot * npad;
                    T* dst = cand_s + (size_t)lane * (npad + 1u);
                    for (uint32_t l = 0; l < a.n; l++) dst[l] = row[l];
                    __syncwarp();
                }
                for (uint32_t j = 0; j < qn; j++) {
                    const T* q = q_s + (size_t)j * npad;
                    const T s =
                        sqdist_generic<T, MODEL, POL>(q, cand_s + (size_t)lane * (npad + 1u), a.n, a.ilp, a.thr, valid);
                    const bool hit = valid && (s <= a.thr);
                    const unsigned b = __ballot_sync(FULL, hit);
                    if (b) {
                        const bool cr = STAMP && cross && hit;
                        const unsigned cb = __ballot_sync(FULL, cr);
                        emit_keys(o, blk_base, blk_used, emitted, hit, cr, b, cb, lt, lane,
                                  __shfl_sync(FULL, my_qid, j), corig);
                    }
                }
                __syncwarp();
            }
        }
        __syncwarp();
    }
    if (lane == 0 && cand_total) atomicAdd(a.cand_cnt, cand_total);
    if (o.emit && blk_used < kEmitBlk)
        for (uint32_t e = blk_used + (uint32_t)lane; e < kEmitBlk; e += 32u)
            if (blk_base + e < o.cap) o.pairs[blk_base + e] = kKeyPad;
    if (lane == 0 && emitted) atomicAdd(o.rechecks, emitted);
}

// ------------------------------------------------------------------ register form
// Float rows of up to NP <= 16 values.  Each lane keeps G candidate rows in
// registers, so a query costs NP/4 broadcast reads and 2 NP arithmetic
// instructions per 32 candidates, and one vote per 32 G candidates when
// nothing is within eps.  Columns from n to NP are zero in every row: a
// zero difference leaves every running sum unchanged bit for bit, so NP need not
// be n.  Lanes without a candidate hold NaN coordinates, which are within
// no threshold.
//
// Bound by instruction issue (0.71 of the slots on the 6-D mixture) and by the
// latency of the enumeration.  Measured, both launches of a join and the
// sampling pass: 6-D 5M points 40.8 -> 17.4 ms, 8-D 142k points (ILP 8 with
// SHORTCIRCUIT, formerly through shared memory) 16.8 -> 1.4 ms.  What did not
// help: 16-byte entries for single cells hashed next to their row neighbours (33
// ms, the table no longer fits the L2 and its probe chains diverge); two rows'
// lookups in flight with all their steps unrolled (the code outgrows the
// instruction cache); items of 2 to 4 neighbouring cells of a grid row (17.1 ms at
// 5M, 5 to 10 % slower on the smaller ones: what the shared enumeration saves
// goes into candidates of cells two steps away).
//
// How the terms are summed (gsj_dist.cuh, float):
//   kSumSeq    s = fma(d, d, s) (ILP 0 and 1)
//   kSumFirst  ILP >= n with either ILP model: one square per register, the
//              registers added in order: s = d0^2, s += d_l^2
//   kSumMask   SHORTCIRCUIT with 1 < ILP < n: the first dim of every ILP block is
//              fused into s, the others are squared and added
enum RegSum : int { kSumSeq = 0, kSumFirst = 1, kSumMask = 2 };

template <int NP, int SUM>
__device__ __forceinline__ float reg_sqdist(const float (&q)[NP], const float (&c)[NP], uint32_t fused) {
    float s = 0.f;
#pragma unroll
    for (int l = 0; l < NP; l++) {
        const float d = __fsub_rn(c[l], q[l]);
        if (SUM == kSumSeq || l == 0) s = __fmaf_rn(d, d, s);
        else if (SUM == kSumFirst) s = __fadd_rn(s, __fmul_rn(d, d));
        else s = ((fused >> l) & 1u) ? __fmaf_rn(d, d, s) : __fadd_rn(s, __fmul_rn(d, d));
    }
    return s;
}

template <int NP>
__device__ __forceinline__ void reg_load(const float* __restrict__ p, float (&r)[NP]) {
#pragma unroll
    for (int l = 0; l < NP; l += 4) {
        if (l + 4 <= NP) {
            const float4 v = *reinterpret_cast<const float4*>(p + l);
            r[l] = v.x;
            r[l + 1] = v.y;
            r[l + 2] = v.z;
            r[l + 3] = v.w;
        } else {  // NP = 6: rows are padded to 8
            const float2 v = *reinterpret_cast<const float2*>(p + l);
            r[l] = v.x;
            r[l + 1] = v.y;
        }
    }
}

// Entries of the per-warp hit queue: up to 31 left over and the hits of a query
// among 32 G candidates.
constexpr uint32_t kMaxTiles = 4;
constexpr uint32_t kHitQueue = 32u + 32u * kMaxTiles;

struct RegSmem {
    uint32_t q, nbs, nbp, hits, total;
};

__host__ __device__ inline RegSmem reg_smem(uint32_t np4, uint32_t nrow) {
    RegSmem t{};
    uint32_t o = 0;
    t.q = o;
    o += 32u * np4 * 4u;
    t.hits = o;
    o += kHitQueue * 8u;
    t.nbs = o;
    o += nrow * 4u;
    t.nbp = o;
    o += (nrow + 1u) * 4u;
    t.total = align16(o);
    return t;
}

// A unit is heavy.unit steps of (query, 32 G candidates); an item of more than
// twice that goes to the heavy list in slices.  A step is about 60 instructions.
// Short units balance a small join (142k points in 8-D, 32 queries an item in the
// dense cells: unsliced, the longest items held the launch for two thirds of its
// time), long ones repeat the enumeration less often: see join_unit_steps.
template <int NP, int SUM, int G, bool STAMP, bool PLAN, bool SLICES>
__global__ void __launch_bounds__(256, 4) k_join_reg(const JoinArgs<float> a, uint32_t nrow, const TileOut o,
                                                     const HeavyList heavy, uint32_t nvisit) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    constexpr uint32_t NP4 = (NP + 3) / 4 * 4;
    static_assert(G <= (int)kMaxTiles, "hit queue");
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const RegSmem L = reg_smem(NP4, nrow);
    unsigned char* wb = smem_raw + (size_t)(threadIdx.x >> 5) * L.total;
    float* q_s = reinterpret_cast<float*>(wb + L.q);
    uint2* hits = reinterpret_cast<uint2*>(wb + L.hits);  // (query slot | cross << 31, candidate slot)
    uint32_t* nb_start = reinterpret_cast<uint32_t*>(wb + L.nbs);
    uint32_t* nb_pref = reinterpret_cast<uint32_t*>(wb + L.nbp);
    const unsigned lt = lanemask_lt();
    unsigned long long cand_total = 0;
    unsigned long long blk_base = 0, emitted = 0;
    uint32_t blk_used = kEmitBlk, nq = 0;  // nq: entries in the hit queue
    uint32_t fused = 0;                    // kSumMask: dims fused into the sum
    if (SUM == kSumMask)
        for (uint32_t l = 0; l < NP; l += a.ilp) fused |= 1u << l;

    // The last `cnt` (at most 32) entries of the queue become keys, a full warp of
    // them at a time.
    auto flush = [&](uint32_t cnt) {
        __syncwarp();
        const bool v = (uint32_t)lane < cnt;
        const uint2 e = v ? hits[nq - cnt + (uint32_t)lane] : make_uint2(0u, 0u);
        const bool cr = STAMP && (e.x >> 31) != 0u;
        const unsigned b = __ballot_sync(FULL, v), cb = __ballot_sync(FULL, cr);
        const uint64_t qid = v && o.emit ? a.ids[e.x & 0x7fffffffu] : 0u, cid = v && o.emit ? a.ids[e.y] : 0u;
        emit_keys(o, blk_base, blk_used, emitted, v, cr, b, cb, lt, lane, qid, cid);
        nq -= cnt;
        __syncwarp();
    };

    const uint32_t nunits = SLICES ? (uint32_t)min(*heavy.count, (unsigned long long)heavy.cap) : nvisit;
    uint32_t* counter = SLICES ? heavy.claim : a.work_counter;
    // one claim at a time, the next one in flight while an item is processed (see k_join)
    uint32_t claim = 0;
    if (lane == 0) claim = atomicAdd(counter, 1u);
    for (;;) {
        const uint32_t unit = __shfl_sync(FULL, claim, 0);
        if (unit >= nunits) break;
        if (lane == 0) claim = atomicAdd(counter, 1u);
        uint32_t visit = unit, slice = 0;
        if (SLICES) {
            const uint2 h = heavy.list[unit];
            visit = h.x;
            slice = h.y;
            if (visit >= nvisit) continue;  // an entry of an item that found the list full
        }
        const uint2 wi = a.items[(size_t)visit * o.stride];
        const uint32_t cs = a.cell_start[wi.x], ce = a.cell_start[wi.x + 1];
        const uint32_t q0 = cs + wi.y * kQChunk;
        const uint32_t qn = min((uint32_t)kQChunk, ce - q0);
        uint32_t total;
        const uint32_t nnb = enumerate_rows<float, STAMP, PLAN>(a, wi.x, cs, nrow, nb_start, nb_pref, lane, lt, total);
        uint32_t g_lo = 0, g_hi = (total + 32u * G - 1u) / (32u * G);  // candidate groups of this unit
        const uint32_t per = (heavy.unit + qn - 1u) / qn;              // groups of a slice
        if (SLICES) {
            g_lo = slice * per;
            g_hi = min(g_hi, g_lo + per);
        } else {
            cand_total += (unsigned long long)total * qn;
            if (g_hi > 2u * per) {
                const uint32_t ns = (g_hi + per - 1u) / per;
                unsigned long long at = 0;
                if (lane == 0) at = atomicAdd(heavy.count, (unsigned long long)ns);
                at = __shfl_sync(FULL, at, 0);
                const bool fits = at + ns <= heavy.cap;
                const uint32_t room = at < heavy.cap ? min(ns, heavy.cap - (uint32_t)at) : 0u;
                for (uint32_t i = (uint32_t)lane; i < room; i += 32u)
                    heavy.list[at + i] = make_uint2(fits ? visit : 0xffffffffu, i);
                if (fits) continue;
            }
        }
        // ---- queries
        __syncwarp();
        {
            const float4* src = reinterpret_cast<const float4*>(a.pts + (size_t)q0 * NP4);
            for (uint32_t e = lane; e < qn * (NP4 / 4u); e += 32) reinterpret_cast<float4*>(q_s)[e] = src[e];
        }
        __syncwarp();

        uint32_t ent = 0;  // the neighbour row of the group's first candidate
        if (SLICES && g_lo) {
            uint32_t hi = nnb;
            while (hi - ent > 1u) {
                const uint32_t mid = (ent + hi) / 2u;
                if (nb_pref[mid] <= g_lo * 32u * G) ent = mid;
                else hi = mid;
            }
        }
        for (uint32_t g = g_lo; g < g_hi; g++) {
            float cx[G][NP];
            uint32_t slot[G];
#pragma unroll
            for (int t = 0; t < G; t++) {
                const uint32_t f0 = (g * G + (uint32_t)t) * 32u;
                slot[t] = 0u;
                if (f0 < total) slot[t] = cand_slot(nb_start, nb_pref, nnb, ent, f0, lane, total);
                reg_load<NP>(a.pts + (size_t)slot[t] * NP4, cx[t]);
                if (f0 + (uint32_t)lane >= total) cx[t][0] = __int_as_float(0x7fffffff);
            }
            for (uint32_t j = 0; j < qn; j++) {
                float q[NP];
                reg_load<NP>(q_s + (size_t)j * NP4, q);
                float s[G];
                bool any = false;
#pragma unroll
                for (int t = 0; t < G; t++) {
                    s[t] = reg_sqdist<NP, SUM>(q, cx[t], fused);
                    any = any || s[t] <= a.thr;
                }
                if (!__any_sync(FULL, any)) continue;
#pragma unroll
                for (int t = 0; t < G; t++) {
                    const bool hit = s[t] <= a.thr;
                    const unsigned b = __ballot_sync(FULL, hit);
                    // outside the own cell: the reverse pair too
                    const bool cross = STAMP && (slot[t] < cs || slot[t] >= ce);
                    if (hit)
                        hits[nq + (uint32_t)__popc(b & lt)] =
                            make_uint2((q0 + j) | (cross ? 0x80000000u : 0u), slot[t]);
                    nq += (uint32_t)__popc(b);
                }
                while (nq >= 32u) flush(32u);
            }
        }
    }
    if (nq) flush(nq);
    if (!SLICES && lane == 0 && cand_total) atomicAdd(a.cand_cnt, cand_total);
    if (o.emit && blk_used < kEmitBlk)
        for (uint32_t e = blk_used + (uint32_t)lane; e < kEmitBlk; e += 32u)
            if (blk_base + e < o.cap) o.pairs[blk_base + e] = kKeyPad;
    if (lane == 0 && emitted) atomicAdd(o.rechecks, emitted);
}

// ------------------------------------------------------------------ launch
// Grid and shared memory of a warp-per-unit kernel (`per_warp` bytes a warp).
static cudaError_t warp_grid(const void* kern, uint32_t per_warp, const uint32_t shape_warps, uint32_t shape_per_sm,
                             uint32_t nvisit, int num_sms, int& threads, size_t& smem, uint64_t& blocks) {
    const uint32_t max_smem = 200u * 1024u;
    int warps = (int)(max_smem / per_warp);
    if (warps > 8) warps = 8;
    if (shape_warps && (int)shape_warps < warps) warps = (int)shape_warps;
    if (warps < 1) return cudaErrorInvalidValue;
    threads = warps * 32;
    smem = (size_t)warps * per_warp;
    cudaError_t e = allow_smem(kern, smem);
    if (e != cudaSuccess) return e;
    int per_sm = 0;
    e = blocks_per_sm(kern, threads, smem, &per_sm);
    if (e != cudaSuccess) return e;
    if (per_sm < 1) per_sm = 1;
    if (shape_per_sm && (int)shape_per_sm < per_sm) per_sm = (int)shape_per_sm;
    // as much of the unified array as those CTAs need; the rest caches candidate
    // rows, which consecutive items (cells of one grid row) share
    const size_t need = (size_t)per_sm * (smem + 1024u);
    int pct = (int)((need * 100u + 228u * 1024u - 1u) / (228u * 1024u));
    if (pct > 100) pct = 100;
    e = cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, pct);
    if (e != cudaSuccess) return e;
    const uint64_t needed = ((uint64_t)nvisit + warps - 1) / warps;
    blocks = (uint64_t)num_sms * per_sm;
    if (blocks > needed) blocks = needed ? needed : 1;
    // every warp claims once past the last item: the counter must not wrap
    if ((uint64_t)nvisit + blocks * (uint64_t)warps >= 0xffffffffull) return cudaErrorInvalidValue;
    return cudaSuccess;
}

template <typename T, int NT, int MODEL, int POL, bool STAMP, bool PLAN = false>
static cudaError_t launch_one(const JoinArgs<T>& a, uint32_t nrow, const TileOut& o, uint32_t nvisit, const WarpLaunch& w) {
    if (!PLAN && a.plan) return launch_one<T, NT, MODEL, POL, STAMP, true>(a, nrow, o, nvisit, w);
    auto kern = k_join<T, NT, MODEL, POL, STAMP, PLAN>;
    const WarpSmem L = warp_smem_layout(a.npad, sizeof(T), nrow, NT == 0);
    int threads = 0;
    size_t smem = 0;
    uint64_t blocks = 0;
    const cudaError_t e = warp_grid((const void*)kern, L.total, a.shape_warps, a.shape_per_sm, nvisit, w.num_sms,
                                    threads, smem, blocks);
    if (e != cudaSuccess) return e;
    if (w.warps) {
        *w.warps = blocks * (uint64_t)(threads / 32);
        return cudaSuccess;
    }
    kern<<<(unsigned)blocks, threads, smem, w.st>>>(a, nrow, o, nvisit);
    *w.launches += 1;
    return cudaGetLastError();
}

template <int NP, int SUM, int G, bool STAMP, bool PLAN = false>
static cudaError_t launch_reg(const JoinArgs<float>& a, uint32_t nrow, const TileOut& o, const HeavyList& heavy,
                              uint32_t nvisit, const WarpLaunch& w) {
    if (!PLAN && a.plan)
        return launch_reg<NP, SUM, G, STAMP, true>(a, nrow, o, heavy, nvisit, w);
    auto k1 = k_join_reg<NP, SUM, G, STAMP, PLAN, false>;
    auto k2 = k_join_reg<NP, SUM, G, STAMP, PLAN, true>;
    const RegSmem L = reg_smem((NP + 3) / 4 * 4, nrow);
    int threads = 0;
    size_t smem = 0;
    uint64_t blocks = 0;
    cudaError_t e = warp_grid((const void*)k1, L.total, a.shape_warps, a.shape_per_sm, nvisit, w.num_sms, threads, smem,
                              blocks);
    if (e != cudaSuccess) return e;
    if (w.warps) *w.warps = blocks * (uint64_t)(threads / 32);
    else k1<<<(unsigned)blocks, threads, smem, w.st>>>(a, nrow, o, heavy, nvisit);
    // the slices of the heavy items, whose number only the device knows
    e = warp_grid((const void*)k2, L.total, a.shape_warps, a.shape_per_sm, heavy.cap, w.num_sms, threads, smem, blocks);
    if (e != cudaSuccess) return e;
    if (w.warps) {
        *w.warps += blocks * (uint64_t)(threads / 32);
        return cudaSuccess;
    }
    k2<<<(unsigned)blocks, threads, smem, w.st>>>(a, nrow, o, heavy, nvisit);
    *w.launches += 2;
    return cudaGetLastError();
}

// Steps of a unit for a join of about `cand` candidate evaluations (0: unknown):
// some 32 units a resident warp.  Emit stage at 32 / 64 / 128 / 256 steps: 6-D
// 200k 0.73 / 0.84 / 0.89 / 1.10 ms, 8-D 142k 1.44 / 1.42 / 1.46 / 1.50, 8-D
// 280k 5.91 / 5.35 / 5.27 / 5.19, 6-D 5M 22.8 / 19.4 / 17.8 / 17.4.
uint32_t join_unit_steps(double cand, int num_sms) {
    if (cand <= 0.0) return 128u;
    const double per_warp = cand / 128.0 / ((double)num_sms * 32.0);
    return (uint32_t)std::min(256.0, std::max(32.0, per_warp / 32.0));
}

// The register form's dispatch: false when the join takes k_join.
template <bool STAMP>
static bool try_reg(const JoinArgs<float>& a, int model, uint32_t nrow, const TileOut& o, const HeavyList& heavy,
                    uint32_t nvisit, const WarpLaunch& w, cudaError_t* e) {
    if (a.n > 16 || a.npad != npad_for(a.n, 4u) || a.npad < 4u || (a.npad & 3u)) return false;
    const bool seq = model == kSeq || a.ilp <= 1u;
    const bool first = !seq && a.ilp >= a.n;
    if (!seq && !first && model != kIlpSc) return false;  // ILP chains of several dims
#define GSJ_REG(NP, SUM, G)                                                                            \
    do {                                                                                               \
        *e = launch_reg<NP, SUM, G, STAMP>(a, nrow, o, heavy, nvisit, w);           \
        return true;                                                                                   \
    } while (0)
    if (seq) {
        if (a.n == 6) GSJ_REG(6, kSumSeq, 4);
        if (a.npad == 4) GSJ_REG(4, kSumSeq, 4);
        if (a.npad == 8) GSJ_REG(8, kSumSeq, 4);
        if (a.npad == 12) GSJ_REG(12, kSumSeq, 2);
        GSJ_REG(16, kSumSeq, 2);
    }
    if (first) {
        if (a.npad == 4) GSJ_REG(4, kSumFirst, 4);
        if (a.npad == 8) GSJ_REG(8, kSumFirst, 4);
        if (a.npad == 12) GSJ_REG(12, kSumFirst, 2);
        GSJ_REG(16, kSumFirst, 2);
    }
    if (a.npad == 4) GSJ_REG(4, kSumMask, 4);
    if (a.npad == 8) GSJ_REG(8, kSumMask, 4);
    if (a.npad == 12) GSJ_REG(12, kSumMask, 2);
    GSJ_REG(16, kSumMask, 2);
#undef GSJ_REG
}

template <typename T, int MODEL, int POL, bool STAMP>
static cudaError_t dispatch_nt(const JoinArgs<T>& a, uint32_t nrow, const TileOut& o, uint32_t nvisit, const WarpLaunch& w) {
    if constexpr (MODEL == kSeq) {
        if (a.npad == npad_for(a.n, sizeof(T))) {
            switch (a.n) {
                case 1: return launch_one<T, 1, MODEL, POL, STAMP>(a, nrow, o, nvisit, w);
                case 2: return launch_one<T, 2, MODEL, POL, STAMP>(a, nrow, o, nvisit, w);
                default: break;
            }
            if constexpr (sizeof(T) == 8) {
                switch (a.n) {
                    case 3: return launch_one<T, 3, MODEL, POL, STAMP>(a, nrow, o, nvisit, w);
                    case 4: return launch_one<T, 4, MODEL, POL, STAMP>(a, nrow, o, nvisit, w);
                    case 6: return launch_one<T, 6, MODEL, POL, STAMP>(a, nrow, o, nvisit, w);
                    case 8: return launch_one<T, 8, MODEL, POL, STAMP>(a, nrow, o, nvisit, w);
                    default: break;
                }
            }
        }
    }
    return launch_one<T, 0, MODEL, POL, STAMP>(a, nrow, o, nvisit, w);
}

template <typename T, bool STAMP>
static cudaError_t dispatch_model(const JoinArgs<T>& a, int model, uint32_t nrow, const TileOut& o,
                                  const HeavyList& heavy, uint32_t nvisit, const WarpLaunch& w) {
    constexpr int P = sizeof(T) == 8 ? kPolF64 : kPolF32;
    if constexpr (sizeof(T) == 4) {
        cudaError_t e = cudaSuccess;
        if (try_reg<STAMP>(a, model, nrow, o, heavy, nvisit, w, &e)) return e;
    }
    switch (model) {
        case kSeq: return dispatch_nt<T, kSeq, P, STAMP>(a, nrow, o, nvisit, w);
        case kIlp: return dispatch_nt<T, kIlp, P, STAMP>(a, nrow, o, nvisit, w);
        case kIlpSc: return dispatch_nt<T, kIlpSc, P, STAMP>(a, nrow, o, nvisit, w);
        default: return cudaErrorInvalidValue;
    }
}

template <typename T>
cudaError_t launch_join_emit(const JoinArgs<T>& a, const TileOut& o, const HeavyList& heavy, uint32_t nvisit,
                             int model, bool stamp, const WarpLaunch& w) {
    uint32_t nrow = 1;  // neighbour rows: 3^(k-1)
    for (uint32_t j = 1; j < a.g.k; j++) nrow *= 3u;
    if (o.stride == 0 || !heavy.list || heavy.cap == 0 || heavy.cap > kHeavyCap || heavy.unit == 0) return cudaErrorInvalidValue;
    if (nvisit == 0) return cudaSuccess;
    if ((uint64_t)(nvisit - 1) * o.stride >= a.num_items) return cudaErrorInvalidValue;
    return stamp ? dispatch_model<T, true>(a, model, nrow, o, heavy, nvisit, w)
                 : dispatch_model<T, false>(a, model, nrow, o, heavy, nvisit, w);
}

template cudaError_t launch_join_emit<float>(const JoinArgs<float>&, const TileOut&, const HeavyList&, uint32_t, int,
                                             bool, const WarpLaunch&);
template cudaError_t launch_join_emit<double>(const JoinArgs<double>&, const TileOut&, const HeavyList&, uint32_t, int,
                                              bool, const WarpLaunch&);

}  // namespace gsj
