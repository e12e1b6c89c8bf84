// Tensor-core screened tile join for high-dimensional float data.
//
// Same work decomposition and output as the tile join (gsj_join_tile.cu): a
// CTA owns up to kScreenQ = 128 consecutive query slots of one cell, walks the
// concatenated candidate slots of the cell's neighbour cells (3^k offsets,
// kernel.cu:180-303) 128 at a time and appends every pair within eps as a
// packed (query id, candidate id) key.  What changes is how a pair is decided:
//
//   1. Once per join (k_screen_rows), every point is centred on the data mean
//      o and rounded to BF16, c^ = bf16(fl(c - o)), and stored as a row
//      [c^, A_hi, A_lo, 1, 1, 0...] (K columns, a multiple of 16), with
//          r = |(c - o) - c^|                       (its own rounding, bounded above)
//          A <= |c^|^2 - 2 R0 r - 2 r^2 - c1 |c^|^2   (rounded down, two BF16 terms)
//      and, for its role as a query, G >= R0^2 + 2 R0 r + 2 r^2 - |c^|^2 +
//      c1 |c^|^2 + c0 R0^2 (rounded up, two BF16 terms).  The rows lie in
//      groups of 8 consecutive slots, each group the 8 x 16-byte core matrices of
//      a K-major shared-memory tile, so that any run of groups is one contiguous
//      copy in global and in shared memory.
//   2. One thread issues tcgen05.mma (kind::f16, BF16 x BF16 -> FP32, M = N =
//      128, K = 16 per instruction) of the query tile [-2 q^, 1, 1, -G_hi, -G_lo]
//      and a tile of 16 candidate groups: the accumulator is
//          D_ij = A_j - 2 q^_i.c^_j - G_i.
//   3. Every consumer thread reads its query's row (tcgen05.ld 32x32b) and
//      rejects candidate j when D_ij >= 0: one OR over the sign bits decides
//      whether any of 32 candidates is left.  The bound is proven, not tuned:
//      |c^ - q^| <= |c - q| + r_c + r_q, so a pair within eps by the reference's
//      arithmetic (whose FP32 sum is covered by R0 >= sqrt(thr): at most 2n+8
//      roundings of non-negative terms) has
//          |c^ - q^|^2 <= (R0 + r_c + r_q)^2
//                      <= R0^2 + 2 R0 (r_c + r_q) + 2 r_c^2 + 2 r_q^2,
//      which is A_j - 2 q^.c^ - G_i <= -(c1 (|c^|^2 + |q^|^2) + c0 R0^2) in exact
//      arithmetic, and c1, c0 exceed the FP32 accumulation error (K + 32 steps
//      of 2^-20 of the summed magnitudes, a factor 8 above FP32 rounding), so
//      D_ij < 0.  A point that is not finite (or beyond 1e15 from the centre)
//      becomes a row with q^ = 0 and A, -G = -2^120: all its pairs stay undecided
//      and no NaN can arise.
//   4. The pairs not rejected are appended as records (query slot, first of 32
//      candidate slots, 32-bit mask), one per query and 32 columns;
//      k_screen_recheck recomputes each pair in the reference's exact FP32 order
//      from the original coordinates (ILP/SHORTCIRCUIT model, kernel.cu:307-365)
//      and keeps it iff s <= thr.
// The emitted pair set is the plain path's, bit for bit.
//
// Candidates are walked in groups: the slot range of a neighbour row (the up to
// three cells x-1..x+1 of one row of the grid, consecutive in cell order) is
// widened to whole groups, and an 8-bit mask per group keeps the rows that
// belong to the range; only undecided pairs look at it.
//
// Roles: warps 0-7 consume, warp 8 copies candidate tiles (a bulk copy per run of
// consecutive groups; most tiles are one run), an elected lane of warp 9 issues the
// MMAs.  Candidate tiles rotate through up to kMaxStages buffers and two
// accumulators alternate, handed over by mbarriers (landed: a buffer's bytes have
// arrived; drained: its MMA has read it; full / empty: an accumulator).  Every
// wait is a bounded poll by a whole warp, whose lanes agree on the outcome; on
// time-out the error flag is raised and the CTA stops.
// Tensor memory (2 x 128 columns) is allocated once per CTA; the shared-memory
// request keeps at most 2 CTAs (512 columns) on an SM; it is released before
// exit.
#include <algorithm>
#include <cstdint>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "gsj_common.cuh"
#include "gsj_fp.cuh"
#include "gsj_kernels.h"

namespace gsj {

namespace {

constexpr int kSQ = kScreenQ;        // queries per item = MMA M
constexpr int kSC = 128;             // candidates per tile = MMA N
constexpr uint32_t kGrp = 8;         // candidate slots per group (rows of a core matrix)
constexpr uint32_t kTileGrps = kSC / kGrp;
constexpr int kConsumers = 256;      // warps 0-7 consume
constexpr int kCopyWarp = 8, kMmaWarp = 9;
constexpr int kSThreads = 320;
constexpr uint32_t kTmemCols = 128;  // FP32 accumulator columns (N)
constexpr uint32_t kMinSmem = 80u * 1024u;  // at most 2 CTAs (2 x 256 TMEM columns) per SM
constexpr uint32_t kWaitHintNs = 20000u, kWaitPolls = 1u << 16;
constexpr uint32_t kBlk = kScreenBlock;  // records a consumer warp reserves at a time
constexpr uint32_t kMaxStages = 8;   // candidate tiles in flight (the accumulators alternate in 2)
// Per-tile candidate metadata rotates through kMeta entries.  Tile g's entry is
// rewritten for tile g + kMeta, whose buffer is free once the MMA of tile
// g + kMeta - stages has run; that MMA waited for every consumer to have read
// the accumulator two tiles earlier, and a consumer reads an accumulator only
// after it is done with all earlier tiles.  So kMeta >= kMaxStages + 3 suffices.
constexpr uint32_t kMeta = 16;
constexpr uint32_t kMaxKpad = 144;   // 126 dimensions + 4 columns, padded to 16
constexpr uint64_t kUnitsPerCta = 16, kMaxParts = 64;  // slicing of small launches
constexpr float kFar = 1e30f;        // |c^|^2 above it: the point is screened by no bound

// Instruction descriptor of tcgen05.mma kind::f16: FP32 accumulator (bit 4),
// A and B BF16 (bits 7 and 10), both K-major, N >> 3 at bit 17, M >> 4 at bit 24.
constexpr uint32_t kIdesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(kSC >> 3) << 17) |
                            ((uint32_t)(kSQ >> 4) << 24);

__device__ __forceinline__ unsigned lanemask_lt_s() {
    unsigned m;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return (uint32_t)__cvta_generic_to_shared(p);
}

// Shared-memory matrix descriptor, K-major, no swizzle: core matrices of 8 rows
// x 16 bytes; LBO = byte distance between K-adjacent core matrices, SBO =
// between row-group-adjacent ones; version 1 (bit 46).
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
    return (uint64_t)((addr >> 4) & 0x3fffu) | ((uint64_t)((lbo >> 4) & 0x3fffu) << 16) |
           ((uint64_t)((sbo >> 4) & 0x3fffu) << 32) | (1ull << 46);
}

// Byte offset of element (r, k) of a K-major tile with kpad columns.
__device__ __forceinline__ uint32_t core_off(uint32_t r, uint32_t kc, uint32_t kpad) {
    return ((r >> 3) * (kpad >> 3) + kc) * 128u + (r & 7u) * 16u;
}

__device__ __forceinline__ void mma_bf16(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(tmem_d),
        "l"(adesc), "l"(bdesc), "r"(kIdesc), "r"(accumulate));
}

// True for one lane of a converged warp, the same one every time.
__device__ __forceinline__ bool elect_one() {
    uint32_t p;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "elect.sync _|p, 0xffffffff;\n\t"
        "selp.b32 %0, 1, 0, p;\n\t}\n"
        : "=r"(p));
    return p != 0;
}

__device__ __forceinline__ void mma_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar)
                 : "memory");
}

// try_wait suspends the thread in hardware until the phase completes or the
// hint (ns) passes, so that waiting warps leave the issue slots to the others;
// the loop bounds the total wait (about a second).
__device__ __forceinline__ bool bar_try(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
        "selp.b32 %0, 1, 0, p;\n\t}\n"
        : "=r"(ok)
        : "r"(bar), "r"(parity), "r"(kWaitHintNs)
        : "memory");
    return ok != 0;
}

// The whole warp waits; the outcome is the same for all lanes.
__device__ __forceinline__ bool warp_wait_bounded(uint32_t bar, uint32_t parity) {
    for (uint32_t it = 0; it < kWaitPolls; it++)
        if (__all_sync(0xffffffffu, bar_try(bar, parity))) return true;
    return false;
}

__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// 32 accumulator columns of the warp's 32 rows (row = lane); tmem_wait_ld
// completes the loads.
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t* r) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
        "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
          "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
          "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr));
}

// The wait names every loaded register, so that no use of them can move above it.
__device__ __forceinline__ void tmem_wait_ld(uint32_t* r) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]),
                   "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]),
                   "+r"(r[15]), "+r"(r[16]), "+r"(r[17]), "+r"(r[18]), "+r"(r[19]), "+r"(r[20]), "+r"(r[21]),
                   "+r"(r[22]), "+r"(r[23]), "+r"(r[24]), "+r"(r[25]), "+r"(r[26]), "+r"(r[27]), "+r"(r[28]),
                   "+r"(r[29])
                 :
                 : "memory");
    asm volatile("" : "+r"(r[30]), "+r"(r[31])::"memory");
}

// The same for 32 more registers, after the wait.
__device__ __forceinline__ void tmem_named(uint32_t* r) {
#pragma unroll
    for (int j = 0; j < 32; j += 8)
        asm volatile("" : "+r"(r[j]), "+r"(r[j + 1]), "+r"(r[j + 2]), "+r"(r[j + 3]), "+r"(r[j + 4]), "+r"(r[j + 5]),
                          "+r"(r[j + 6]), "+r"(r[j + 7])::"memory");
}

// The reference's squared distance of the ILP model without SHORTCIRCUIT (one
// chain per register over the dims l = j mod ILP, the chains added in order), one
// thread, stopping as soon as the running value (which only grows) is above thr.
__device__ float exact_sqdist_ilp(const float* __restrict__ q, const float* __restrict__ c, uint32_t n, uint32_t ilp,
                                  float thr) {
    float s = 0.f;
    for (uint32_t j = 0; j < ilp && j < n; j++) {
        float r = 0.f;
        for (uint32_t l = j; l < n; l += ilp) {
            const float d = __fsub_rn(c[l], q[l]);
            r = __fmaf_rn(d, d, r);
        }
        s = j == 0 ? r : __fadd_rn(s, r);
        if (s > thr) break;
    }
    return s;
}

// The other models, rows read as float4 blocks of 16 dimensions loaded before use
// (npad is a multiple of 4, the padding is 0 and adds nothing): the sequential
// model fuses every term; with SHORTCIRCUIT the terms l = 0 mod ILP are fused,
// the others rounded and added.  fused[b]: bit e, whether term 16 b + e is.
template <int MODEL>
__device__ __forceinline__ float exact_sqdist4(const float* __restrict__ q, const float* __restrict__ c, uint32_t n,
                                               const uint32_t* __restrict__ fused, float thr) {
    const float4* q4 = reinterpret_cast<const float4*>(q);
    const float4* c4 = reinterpret_cast<const float4*>(c);
    float s = 0.f;
    for (uint32_t l0 = 0; l0 < n; l0 += 16u) {
        float4 qa[4], ca[4];
#pragma unroll
        for (int b = 0; b < 4; b++) {
            if (l0 + 4u * b < n) {
                qa[b] = q4[(l0 >> 2) + b];
                ca[b] = c4[(l0 >> 2) + b];
            }
        }
        const uint32_t fm = MODEL == kIlpSc ? fused[l0 >> 4] : 0u;
#pragma unroll
        for (int b = 0; b < 4; b++) {
            if (l0 + 4u * b >= n) break;
            const float qv[4] = {qa[b].x, qa[b].y, qa[b].z, qa[b].w};
            const float cv[4] = {ca[b].x, ca[b].y, ca[b].z, ca[b].w};
#pragma unroll
            for (int e = 0; e < 4; e++) {
                const float d = __fsub_rn(cv[e], qv[e]);
                if (MODEL == kSeq || (fm & (1u << (4 * b + e)))) s = __fmaf_rn(d, d, s);
                else s = __fadd_rn(s, __fmul_rn(d, d));
            }
        }
        if (s > thr) break;
    }
    return s;
}

// Bit c: slot gs + c lies outside [lo, hi); gs is a slot or, modulo 2^32, up to
// 24 below slot 0.
__device__ __forceinline__ uint32_t outside_mask(uint32_t gs, uint32_t lo, uint32_t hi) {
    const int64_t g = gs > 0xffffffe0u ? (int64_t)gs - (1ll << 32) : (int64_t)gs;
    const int64_t a = (int64_t)lo - g, b = (int64_t)hi - g;
    const uint32_t l = a <= 0 ? 0u : a >= 32 ? 32u : (uint32_t)a, h = b <= 0 ? 0u : b >= 32 ? 32u : (uint32_t)b;
    const uint32_t below_l = l == 32u ? 0xffffffffu : (1u << l) - 1u, below_h = h == 32u ? 0xffffffffu : (1u << h) - 1u;
    return ~(below_h & ~below_l);
}

struct ScreenSmem {
    uint32_t a, nbs, nbe, nbg, mbase, mmask, misc, b, total;
};

// Byte sizes are rounded to 128 so that the tiles stay aligned; `stages`
// candidate tiles follow at b.
__host__ __device__ inline ScreenSmem screen_smem(uint32_t kpad, uint32_t nrow, uint32_t stages) {
    ScreenSmem t{};
    uint32_t o = 0;
    t.a = o;
    o += (uint32_t)kSQ * kpad * 2u;
    t.nbs = o;  // per neighbour row: first slot, end slot, exclusive prefix of the groups
    o += nrow * 4u;
    t.nbe = o;
    o += nrow * 4u;
    t.nbg = o;
    o += (nrow + 1u) * 4u;
    o = (o + 15u) & ~15u;  // read as 16-byte vectors
    t.mbase = o;  // [kMeta][16] first slot of each group of a tile
    o += kMeta * kTileGrps * 4u;
    t.mmask = o;  // [kMeta][16] bytes: rows of the group that are candidates
    o += kMeta * kTileGrps;
    o = (o + 15u) & ~15u;
    t.misc = o;   // [0] unit [1] failed [2] groups [3] candidates [4] tmem [8..17] warp counts
                  // [20..] mbarriers: full 0 1, empty 0 1, landed 0..7, drained 0..7
                  // [64..] undecided pairs and records of each consumer warp (64-bit)
    o += 96u * 4u;
    o = (o + 127u) & ~127u;
    t.b = o;
    o += stages * (uint32_t)kSC * kpad * 2u;
    t.total = o;
    return t;
}

__device__ __forceinline__ void bar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}

__device__ __forceinline__ void bar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}

__device__ __forceinline__ void bar_arrive_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}

// Untiled bulk copy global -> this CTA's shared memory (16-byte aligned, whole
// groups of rows), completing on `bar`.
__device__ __forceinline__ void bulk_copy(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cta.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
                 "l"(__cvta_generic_to_global(src)), "r"(bytes), "r"(bar)
                 : "memory");
}

// A unit is a slice (one of `parts`) of the candidate tiles of an item (up to
// 128 consecutive query slots of one cell): slices give small joins and the
// sampling pass enough units for the whole chip and shorten the last wave.
//
// What bounds it: the two accumulators of a CTA (all of tensor memory at 2 CTAs
// an SM) alternate between the MMA and eight consumer warps that need them for
// different times, since only some warps of a tile meet an undecided pair (about
// 1 in 5 at 18 dims; such a warp takes some 1,000 cycles longer).  So a consumer
// warp reads its 64 columns at once and frees the accumulator before it looks at
// them, and the path of a warp with undecided pairs is kept short (one word of
// metadata says whether four groups are consecutive, which makes one record a
// query row; records go to a block that is never split).  A tile takes some 530
// cycles of an SM at K = 32 (the tensor pipe needs 128) and 650 at K = 96 (384).
// Measured (count stage of a join, the exact check included): 18-D 5M points 380 ->
// 145 ms (126 of it this kernel, 3 its sampling pass), 90-D 515k 121 -> 38 ms, 32-D
// 45k 2.0 -> 0.61 ms (both launches alone), against four warps staging rows one by
// one with cp.async and a compare per pair with a bound per 32 candidates (1,720
// cycles a tile).  Tried without gain: 16 consumer warps a CTA reading 16 columns
// at a time, an MMA warp per accumulator.
template <bool STAMP>
__global__ void __launch_bounds__(kSThreads, 2) k_tile_screen(const JoinArgs<float> a, const TileOut o,
                                                              const ScreenConst sc, uint32_t nrow, uint32_t stages,
                                                              uint32_t parts, uint32_t nunits) {
    extern __shared__ __align__(1024) unsigned char ssm[];
    const uint32_t n = a.n, npad = a.npad, k = a.g.k, kpad = sc.kpad, kch = kpad >> 3;
    const ScreenSmem L = screen_smem(kpad, nrow, stages);
    unsigned char* A = ssm + L.a;
    uint32_t* nb_start = reinterpret_cast<uint32_t*>(ssm + L.nbs);
    uint32_t* nb_end = reinterpret_cast<uint32_t*>(ssm + L.nbe);
    uint32_t* nb_grp = reinterpret_cast<uint32_t*>(ssm + L.nbg);
    uint32_t* m_base = reinterpret_cast<uint32_t*>(ssm + L.mbase);
    unsigned char* m_mask = ssm + L.mmask;
    uint32_t* misc = reinterpret_cast<uint32_t*>(ssm + L.misc);
    const unsigned FULL = 0xffffffffu;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const unsigned lt = lanemask_lt_s();
    const uint32_t sbo = kch * 128u;                          // bytes of a group
    const uint32_t stage_bytes = (uint32_t)kSC * kpad * 2u;
    const uint32_t a_addr = smem_u32(A), b_addr = smem_u32(ssm + L.b);
    const uint32_t full = smem_u32(misc + 20), empty = smem_u32(misc + 24);    // [2] each, 8 bytes apart
    const uint32_t landed = smem_u32(misc + 28), drained = smem_u32(misc + 44);  // [stages] each

    // ---- set-up: mbarriers, tensor memory (two accumulators)
    if (tid == 0) {
        misc[1] = 0u;
        for (uint32_t s = 0; s < 2u; s++) {
            bar_init(full + 8u * s, 2u);                  // the MMA's commit, the issuing thread
            bar_init(empty + 8u * s, kConsumers / 32u);   // a thread of every consumer warp
        }
        for (uint32_t b = 0; b < stages; b++) {
            bar_init(landed + 8u * b, 1u);   // the copying thread, and the bytes
            bar_init(drained + 8u * b, 1u);  // the MMA's commit
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(misc + 4)),
                     "r"(2u * kTmemCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tmem = misc[4];
    // tiles of earlier units: tile g uses buffer g % stages, accumulator g % 2 and
    // metadata entry g % kMeta, and its mbarriers' phases follow from g
    uint32_t g0 = 0;
    unsigned long long cand_total = 0;
    // consumer warps: the reserved block of records; undecided pairs and records
    // so far in shared memory
    uint4* blk = nullptr;
    uint32_t blk_used = kBlk, blk_room = 0;
    uint4* recs = reinterpret_cast<uint4*>(o.pairs);
    unsigned long long* n_und = reinterpret_cast<unsigned long long*>(misc + 64) + warp;
    unsigned long long* n_rec = n_und + kConsumers / 32;
    if (tid < kConsumers && lane == 0) *n_und = *n_rec = 0ull;

    for (;;) {
        __syncthreads();
        if (tid == 0) misc[0] = atomicAdd(a.work_counter, 1u);
        __syncthreads();
        const uint32_t unit = misc[0];
        if (unit >= nunits || misc[1]) break;
        const uint32_t vi = unit / parts, part = unit - vi * parts;
        const uint2 wi = a.items[(size_t)vi * o.stride];
        const uint32_t cell = wi.x;
        const uint32_t cs0 = a.cell_start[cell], ce = a.cell_start[cell + 1];
        const uint32_t q0 = cs0 + wi.y * (uint32_t)kSQ;
        const uint32_t qn = min((uint32_t)kSQ, ce - q0);

        // ---- neighbour rows in offset order (kernel.cu:180-303; stamploops.h)
        uint32_t own[kMaxK];
#pragma unroll
        for (int j = 0; j < kMaxK; j++)
            own[j] = (j < (int)k) ? FP<float>::to_uint_rz(FP<float>::div(
                                        FP<float>::sub(a.pts[(size_t)cs0 * npad + j], a.minv[j]), a.eps))
                                  : 0u;
        uint32_t nnb = 0;
        uint32_t lowmask, highmask, oddmask;
        cell_masks(own, a.g, lowmask, highmask, oddmask);
        const uint64_t own_lin = a.cell_key[cell];
        for (uint32_t base = 0; base < nrow; base += kSThreads) {
            const uint32_t r = base + (uint32_t)tid;
            uint32_t st = 0, cnt = 0;
            const bool found =
                row_range<float, STAMP>(a, r < nrow, r, own_lin, own[0], lowmask, highmask, oddmask, st, cnt);
            const unsigned m = __ballot_sync(FULL, found);
            if (lane == 0) misc[8 + warp] = __popc(m);
            __syncthreads();
            uint32_t before = 0, all = 0;
#pragma unroll
            for (int w = 0; w < kSThreads / 32; w++) {
                const uint32_t cw = misc[8 + w];
                before += (w < warp) ? cw : 0u;
                all += cw;
            }
            if (found) {
                const uint32_t pos = nnb + before + __popc(m & lt);
                nb_start[pos] = st;
                nb_end[pos] = st + cnt;
            }
            nnb += all;
            __syncthreads();
        }
        if (warp == kMmaWarp) {
            // exclusive prefix of the groups, and the candidates of a query
            uint32_t run = 0, cand = 0;
            for (uint32_t b0 = 0; b0 < nnb; b0 += 32) {
                const uint32_t i = b0 + lane;
                uint32_t v = 0;
                if (i < nnb) {
                    const uint32_t s = nb_start[i], e = nb_end[i];
                    v = (e + kGrp - 1u) / kGrp - s / kGrp;
                    cand += e - s;
                }
                uint32_t x = v;
#pragma unroll
                for (int s = 1; s < 32; s <<= 1) {
                    const uint32_t y = __shfl_up_sync(FULL, x, s);
                    if (lane >= s) x += y;
                }
                if (i < nnb) nb_grp[i] = run + x - v;
                run += __shfl_sync(FULL, x, 31);
            }
            cand = __reduce_add_sync(FULL, cand);
            if (lane == 0) {
                nb_grp[nnb] = run;
                misc[2] = run;
                misc[3] = cand;
            }
        } else {
            // ---- query tile [-2 q^, 1, 1, -G_hi, -G_lo] from the candidate rows; a row
            // past qn is 0 with -G = 2^100: never undecided
            const uint32_t nt = kSThreads - 32u;
            for (uint32_t e = tid; e < (uint32_t)kSQ * kch; e += nt) {
                const uint32_t kc = e / (uint32_t)kSQ, r = e - kc * (uint32_t)kSQ;
                uint4 v = make_uint4(0u, 0u, 0u, 0u);
                uint32_t g = 0x00007180u;  // BF16 (2^100, 0)
                if (r < qn) {
                    const uint32_t s = q0 + r;
                    v = sc.rows[((size_t)(s / kGrp) * kch + kc) * kGrp + s % kGrp];
                    g = sc.qg[s];
                }
                const uint16_t one = r < qn ? (uint16_t)0x3f80u : (uint16_t)0u;
                uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                for (int h = 0; h < 4; h++) {
                    uint32_t word = 0;
#pragma unroll
                    for (int x = 0; x < 2; x++) {
                        const uint32_t col = kc * 8u + 2u * (uint32_t)h + (uint32_t)x;
                        __nv_bfloat16_raw rb;
                        rb.x = (uint16_t)(w[h] >> (16 * x));
                        uint32_t bits;
                        if (col < n) {
                            // -2 q^ (exact)
                            const __nv_bfloat16_raw d =
                                __float2bfloat16_rn(-2.f * __bfloat162float(__nv_bfloat16(rb)));
                            bits = d.x;
                        } else if (col < n + 2u) {
                            bits = one;
                        } else if (col < n + 4u) {
                            bits = col == n + 2u ? (g & 0xffffu) : (g >> 16);
                        } else {
                            bits = 0u;
                        }
                        word |= bits << (16 * x);
                    }
                    w[h] = word;
                }
                *reinterpret_cast<uint4*>(A + core_off(r, kc, kpad)) = make_uint4(w[0], w[1], w[2], w[3]);
            }
        }
        fence_async_smem();
        __syncthreads();
        const uint32_t groups = misc[2];
        const uint32_t T = (groups + kTileGrps - 1u) / kTileGrps;
        const uint32_t t0 = (uint32_t)((uint64_t)T * part / parts), t1 = (uint32_t)((uint64_t)T * (part + 1u) / parts);
        if (part == 0u) cand_total += (unsigned long long)misc[3] * qn;

        if (warp == kCopyWarp) {
            // ================= candidate tiles: lanes 0-15 own the groups of tile t,
            // lanes 16-31 those of t + 1; a run of consecutive groups is one bulk copy
            const uint32_t sub = (uint32_t)lane / kTileGrps, half = (uint32_t)lane % kTileGrps;
            uint32_t e = 0;  // this lane's neighbour row (its group position grows by 32 per round)
            {
                uint32_t hi = nnb;
                const uint32_t f = t0 * kTileGrps + (uint32_t)lane;
                while (hi - e > 1u) {
                    const uint32_t mid = (e + hi) / 2u;
                    if (nb_grp[mid] <= f) e = mid;
                    else hi = mid;
                }
            }
            uint32_t g = g0, b = g0 % stages, ph = (g0 / stages) & 1u;
            bool ok = true;
            for (uint32_t t = t0; ok && t < t1; t += 2u) {
                const uint32_t f = t * kTileGrps + (uint32_t)lane;
                const bool mine = f < groups;
                uint32_t gid = 0;
                unsigned char mask = 0;
                if (mine) {
                    while (nb_grp[e + 1] <= f) e++;
                    const uint32_t s = nb_start[e], en = nb_end[e];
                    gid = s / kGrp + (f - nb_grp[e]);
                    const uint32_t b0 = gid * kGrp;
                    const uint32_t lo = s > b0 ? s - b0 : 0u, hi = min(kGrp, en - b0);
                    mask = (unsigned char)((0xffu << lo) & (0xffu >> (kGrp - hi)));
                }
                const uint32_t prev = __shfl_up_sync(FULL, gid, 1);
                const bool head = mine && (half == 0u || gid != prev + 1u);
                const unsigned heads = __ballot_sync(FULL, head);
                const unsigned breaks = heads | __ballot_sync(FULL, !mine);
                for (uint32_t u = 0; u < 2u && t + u < t1; u++) {
                    if (g >= stages) {
                        ok = warp_wait_bounded(drained + 8u * b, ph ^ 1u);
                        if (!ok) break;
                    }
                    const uint32_t ng = min(kTileGrps, groups - (t + u) * kTileGrps);
                    const uint32_t bar = landed + 8u * b;
                    if (sub == u) {
                        // bit 0: the four groups of the aligned quad are consecutive
                        m_base[(g % kMeta) * kTileGrps + half] = gid * kGrp | ((breaks >> (lane & ~3)) & 0xeu ? 0u : 1u);
                        m_mask[(g % kMeta) * kTileGrps + half] = mask;
                    }
                    __syncwarp();
                    if (lane == 0) bar_arrive_tx(bar, ng * sbo);
                    __syncwarp();
                    if (head && sub == u) {
                        const unsigned after = (heads >> lane >> 1) & (0xffffu >> (half + 1u));
                        const uint32_t len = after ? (uint32_t)__ffs(after) : ng - half;
                        bulk_copy(b_addr + b * stage_bytes + half * sbo, sc.rows + (size_t)gid * kch * kGrp, len * sbo,
                                  bar);
                    }
                    g++;
                    if (++b == stages) {
                        b = 0;
                        ph ^= 1u;
                    }
                }
            }
            if (!ok) {
                // give the copies in flight another bounded wait before the CTA stops
                misc[1] = 1u;
                for (uint32_t x = 0; x < stages && x < g; x++) {
                    if (b == 0u) {
                        b = stages;
                        ph ^= 1u;
                    }
                    b--;
                    warp_wait_bounded(landed + 8u * b, ph);
                }
            }
        } else if (warp == kMmaWarp) {
            // ================= a landed tile and a free accumulator -> MMA: the warp stays
            // converged (waits, descriptors), one elected lane issues
            bool ok = true;
            uint32_t b = g0 % stages, ph = (g0 / stages) & 1u;
            const uint64_t adesc = smem_desc(a_addr, 128u, sbo);
            const uint32_t ksteps = kpad >> 4;
            for (uint32_t t = t0, g = g0; t < t1; t++, g++) {
                // the first use of an accumulator waits for the phase before its first
                const uint32_t s = g & 1u;
                ok = warp_wait_bounded(landed + 8u * b, ph) && warp_wait_bounded(empty + 8u * s, ((g >> 1) & 1u) ^ 1u);
                if (!ok) break;
                fence_after();
                const uint64_t bdesc = smem_desc(b_addr + b * stage_bytes, 128u, sbo);
                const uint32_t acc = tmem + s * kTmemCols;
                if (elect_one()) {
                    // a K step is 2 core matrices of 128 bytes on (in units of 16 bytes)
                    mma_bf16(acc, adesc, bdesc, 0u);
                    for (uint32_t ks = 1; ks < ksteps; ks++)
                        mma_bf16(acc, adesc + 16u * ks, bdesc + 16u * ks, 1u);
                    mma_commit(full + 8u * s);
                    mma_commit(drained + 8u * b);
                    bar_arrive(full + 8u * s);
                }
                __syncwarp();
                if (++b == stages) {
                    b = 0;
                    ph ^= 1u;
                }
            }
            if (!ok) misc[1] = 1u;
            __syncwarp();
        } else {
            // ================= consumer warps: query row i = TMEM lane i; warps w and
            // w + 4 share lane quarter w % 4 and split the columns
            const uint32_t quarter = (uint32_t)warp & 3u, colbase = ((uint32_t)warp >> 2) * ((uint32_t)kSC / 2u);
            const uint32_t qslot = q0 + quarter * 32u + (uint32_t)lane;
            const bool idle = quarter * 32u >= qn;  // no query in the warp's 32 rows
            uint32_t und_count = 0, rec_count = 0;  // undecided pairs of the lane, records of the warp
            for (uint32_t t = t0, g = g0; t < t1; t++, g++) {
                const uint32_t s = g & 1u;
                if (!warp_wait_bounded(full + 8u * s, (g >> 1) & 1u)) {
                    misc[1] = 1u;
                    break;
                }
                fence_after();
                const uint32_t ta = tmem + s * kTmemCols + ((quarter * 32u) << 16) + colbase;
                if (idle) {
                    fence_before();
                    if (lane == 0) bar_arrive(empty + 8u * s);
                    continue;
                }
                // the accumulator is free as soon as the warp's 64 columns are in registers
                uint32_t v[64];
                tmem_ld32(ta, v);
                tmem_ld32(ta + 32u, v + 32);
                tmem_wait_ld(v);
                tmem_named(v + 32);
                fence_before();
                __syncwarp();
                if (lane == 0) bar_arrive(empty + 8u * s);
                // common case: every value has its sign bit clear (independent chains: one
                // chain of dependent operations would take several times the issue time)
                uint32_t x[8];
#pragma unroll
                for (int c = 0; c < 8; c++) {
                    x[c] = v[8 * c];
#pragma unroll
                    for (int j = 1; j < 8; j++) x[c] |= v[8 * c + j];
                }
                uint32_t signs[2] = {(x[0] | x[1]) | (x[2] | x[3]), (x[4] | x[5]) | (x[6] | x[7])};
                if (!__any_sync(FULL, (int)(signs[0] | signs[1]) < 0)) continue;
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    if (!__any_sync(FULL, (int)signs[h] < 0)) {
                        signs[h] = 0u;
                        continue;
                    }
                    signs[h] = 0u;
#pragma unroll
                    for (int c = 0; c < 4; c++) {
                        uint32_t y = 0;
#pragma unroll
                        for (int j = 7; j >= 0; j--) y = __funnelshift_l(v[32 * h + 8 * c + j], y, 1);
                        signs[h] |= y << (8 * c);
                    }
                }
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    const uint32_t mg = (g % kMeta) * kTileGrps + colbase / kGrp + 4u * (uint32_t)h;  // first group
                    const uint32_t und = signs[h] & *reinterpret_cast<const uint32_t*>(m_mask + mg);
                    const uint32_t base = m_base[mg];
                    unsigned have = __ballot_sync(FULL, und != 0u);
                    if (!have) continue;
                    und_count += (uint32_t)__popc(und);
                    // a record per run of consecutive groups (nearly always all four)
                    uint32_t mine = und, gs = base & ~1u, left = 0, next_grp = 4u;
                    if (!(base & 1u)) {
                        left = und & 0xffffff00u;
                        mine = und & 0xffu;
                        next_grp = 1u;
                        have = __ballot_sync(FULL, mine != 0u);
                    }
                    for (;;) {
                        // gs: the slot of column 0 (modulo 2^32) for the groups of `mine`
                        const uint32_t cnt = (uint32_t)__popc(have);
                        rec_count += cnt;
                        if (o.emit && cnt) {
                            if (blk_used + cnt > kBlk) {  // the rest of the block stays empty records
                                for (uint32_t e2 = blk_used + (uint32_t)lane; e2 < blk_room; e2 += 32u)
                                    blk[e2] = make_uint4(0u, 0u, 0u, 0u);
                                unsigned long long at = 0;
                                if (lane == 0) at = atomicAdd(o.cursor, (unsigned long long)kBlk);
                                at = __shfl_sync(FULL, at, 0);
                                blk = recs + at;
                                blk_room = at < o.cap ? (uint32_t)min((unsigned long long)kBlk, o.cap - at) : 0u;
                                blk_used = 0u;
                            }
                            const uint32_t p = blk_used + (uint32_t)__popc(have & lt);
                            if (mine && p < blk_room) {
                                uint32_t cross = 0;
                                if (STAMP) cross = outside_mask(gs, cs0, ce);
                                blk[p] = make_uint4(qslot, gs, mine, cross);
                            }
                            blk_used += cnt;
                        }
                        if (next_grp == 4u) break;
                        mine = (left >> (kGrp * next_grp) & 0xffu) << (kGrp * next_grp);
                        gs = (m_base[mg + next_grp] & ~1u) - kGrp * next_grp;
                        have = __ballot_sync(FULL, mine != 0u);
                        next_grp++;
                    }
                }
            }
            const uint32_t u0 = __reduce_add_sync(FULL, und_count & 0xffffu), u1 = __reduce_add_sync(FULL, und_count >> 16);
            if (lane == 0) {
                *n_und += u0 + ((unsigned long long)u1 << 16);
                *n_rec += rec_count;
            }
        }
        g0 += t1 - t0;
    }
    // ---- the consumer warps' last blocks and their counts
    if (tid < kConsumers) {
        for (uint32_t e2 = blk_used + (uint32_t)lane; e2 < blk_room; e2 += 32u) blk[e2] = make_uint4(0u, 0u, 0u, 0u);
        if (lane == 0 && *n_und) atomicAdd(o.rechecks, *n_und);
        if (lane == 0 && !o.emit && *n_rec) atomicAdd(o.cursor, *n_rec);
    }
    // ---- tear-down: every copy and MMA of this CTA has been waited for by its
    // consumers, unless a wait timed out
    if (misc[1] && tid == 0) *a.err_flag = 2u;
    fence_before();
    __syncthreads();
    fence_after();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(2u * kTmemCols)
                     : "memory");
    if (tid == 0 && cand_total) atomicAdd(a.cand_cnt, cand_total);
}

template <bool STAMP>
cudaError_t launch_screen_one(const JoinArgs<float>& a, const TileOut& o, const ScreenConst& sc, uint32_t nrow,
                              uint32_t nvisit, int num_sms, cudaStream_t st) {
    auto kern = k_tile_screen<STAMP>;
    // as many candidate tiles in flight as leave room for two CTAs on an SM
    const uint32_t two = (228u * 1024u) / 2u - 1024u;
    uint32_t stages = 2;
    while (stages < kMaxStages && screen_smem(sc.kpad, nrow, stages + 1u).total <= two) stages++;
    const ScreenSmem L = screen_smem(sc.kpad, nrow, stages);
    const uint32_t smem = L.total > kMinSmem ? L.total : kMinSmem;
    cudaError_t e = allow_smem((const void*)kern, smem);
    if (e != cudaSuccess) return e;
    // the whole unified L1/shared array as shared memory, so that the CTAs the
    // occupancy calculation counts on are resident together
    e = cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, (int)cudaSharedmemCarveoutMaxShared);
    if (e != cudaSuccess) return e;
    int per_sm = 0;
    e = blocks_per_sm((const void*)kern, kSThreads, smem, &per_sm);
    if (e != cudaSuccess) return e;
    if (per_sm < 1) return cudaErrorInvalidConfiguration;
    // tensor memory: 2 accumulators of 128 columns per CTA, 512 columns per SM
    if ((uint32_t)per_sm * 2u * kTmemCols > 512u) per_sm = (int)(512u / (2u * kTmemCols));
    if (a.shape_per_sm && (int)a.shape_per_sm < per_sm) per_sm = (int)a.shape_per_sm;
    uint64_t blocks = (uint64_t)num_sms * per_sm;
    // slices per item: 16 units per CTA, so that the last wave is short
    uint64_t parts = (blocks * kUnitsPerCta + nvisit - 1u) / nvisit;
    if (parts > kMaxParts) parts = kMaxParts;
    const uint64_t units = (uint64_t)nvisit * parts;
    if (units + blocks >= 0xffffffffull) return cudaErrorInvalidValue;
    if (blocks > units) blocks = units;
    kern<<<(unsigned)blocks, kSThreads, smem, st>>>(a, o, sc, nrow, stages, (uint32_t)parts, (uint32_t)units);
    return cudaGetLastError();
}

}  // namespace

// The exact check of the pairs the screen could not reject: the reference's
// arithmetic for the configured model (kernel.cu:307-365), s <= thr; a hit
// appends (query id, candidate id), and with the record's cross bit (unicomp,
// the candidate outside the query's cell) also the reverse pair.  A warp takes
// 32 records, lists their pairs in shared memory and checks 32 pairs at a time,
// so that records of one pair and of 32 keep the lanes equally busy.
// Bound by its instructions (0.75 issued a cycle and scheduler), the order of the
// model's roundings among them: which terms are fused is a bit mask per 16 dims,
// and a warp reserves output once for its 32 records.  18-D 5M points (524 M
// pairs) 23.0 -> 15.6 ms, 8-D 120k 211 -> 124 us, 90-D 515k 3.15 -> 2.96 ms.
template <int MODEL, bool STAMP>
__global__ void __launch_bounds__(256, 4) k_screen_recheck(const float* __restrict__ pts, const uint32_t* __restrict__ ids,
                                                        uint32_t n, uint32_t npad, uint32_t ilp, float thr,
                                                        uint32_t npoints, const uint4* __restrict__ recs,
                                                        unsigned long long nrec, const TileOut o) {
    __shared__ uint16_t list[8][1024];  // record lane << 5 | column
    __shared__ uint32_t fused[8];       // n <= 126
    if (MODEL == kIlpSc) {
        if (threadIdx.x < 8u) {
            uint32_t m = 0;
            for (uint32_t e = 0; e < 16u; e++) m |= (16u * threadIdx.x + e) % ilp == 0u ? 1u << e : 0u;
            fused[threadIdx.x] = m;
        }
        __syncthreads();
    }
    const unsigned FULL = 0xffffffffu;
    const unsigned lt = lanemask_lt_s();
    const uint32_t lane = threadIdx.x & 31u;
    uint16_t* wl = list[threadIdx.x >> 5];
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t i0 = (uint64_t)blockIdx.x * blockDim.x + (threadIdx.x & ~31u); i0 < nrec; i0 += stride) {
        const uint4 r = i0 + lane < nrec ? recs[i0 + lane] : make_uint4(0u, 0u, 0u, 0u);
        const uint32_t cnt = (uint32_t)__popc(r.z);
        uint32_t x = cnt;
#pragma unroll
        for (int s = 1; s < 32; s <<= 1) {
            const uint32_t y = __shfl_up_sync(FULL, x, s);
            if (lane >= (uint32_t)s) x += y;
        }
        const uint32_t total = __shfl_sync(FULL, x, 31);
        uint32_t pos = x - cnt;
        for (uint32_t m = r.z; m; m &= m - 1u) wl[pos++] = (uint16_t)((lane << 5) | ((uint32_t)__ffs(m) - 1u));
        __syncwarp();
        uint32_t nhit = 0, ncross = 0;
        for (uint32_t b = 0; b < total; b += 32u) {
            const bool valid = b + lane < total;
            const uint32_t e = valid ? wl[b + lane] : 0u;
            const uint32_t qs = __shfl_sync(FULL, r.x, (int)(e >> 5));
            const uint32_t cs = __shfl_sync(FULL, r.y, (int)(e >> 5)) + (e & 31u);
            const uint32_t crossm = STAMP ? __shfl_sync(FULL, r.w, (int)(e >> 5)) : 0u;
            bool hit = false;
            if (valid && qs < npoints && cs < npoints)
                hit = (MODEL == kIlp
                           ? exact_sqdist_ilp(pts + (size_t)qs * npad, pts + (size_t)cs * npad, n, ilp, thr)
                           : exact_sqdist4<MODEL>(pts + (size_t)qs * npad, pts + (size_t)cs * npad, n, fused, thr)) <= thr;
            // the hits move to the front of the list (behind the entries still to be read)
            const unsigned hb = __ballot_sync(FULL, hit);
            if (hit) wl[nhit + (uint32_t)__popc(hb & lt)] = (uint16_t)e;
            nhit += (uint32_t)__popc(hb);
            if (STAMP)
                ncross += (uint32_t)__popc(__ballot_sync(FULL, hit && ((crossm >> (e & 31u)) & 1u)));
            __syncwarp();
        }
        // one reservation for the warp's 32 records
        if (nhit) {
            unsigned long long base = 0;
            if (lane == 0u) base = atomicAdd(o.cursor, (unsigned long long)(nhit + ncross));
            base = __shfl_sync(FULL, base, 0);
            for (uint32_t b = 0; b < nhit; b += 32u) {
                const bool valid = b + lane < nhit;
                const uint32_t e = valid ? wl[b + lane] : 0u;
                const uint32_t qs = __shfl_sync(FULL, r.x, (int)(e >> 5));
                const uint32_t cs = __shfl_sync(FULL, r.y, (int)(e >> 5)) + (e & 31u);
                const uint32_t crossm = STAMP ? __shfl_sync(FULL, r.w, (int)(e >> 5)) : 0u;
                const bool cross = STAMP && valid && ((crossm >> (e & 31u)) & 1u);
                const unsigned cb = STAMP ? __ballot_sync(FULL, cross) : 0u;
                if (valid) {
                    unsigned long long p = base + lane + (unsigned)__popc(cb & lt);
                    const uint64_t qid = ids[qs], cid = ids[cs];
                    if (p < o.cap) o.pairs[p] = (qid << o.shift) | cid;
                    p++;
                    if (cross && p < o.cap) o.pairs[p] = (cid << o.shift) | qid;
                }
                base += 32u + (unsigned)__popc(cb);
            }
        }
        __syncwarp();
    }
}

template <int MODEL, bool STAMP>
cudaError_t launch_recheck_one(const JoinArgs<float>& a, const uint4* recs, unsigned long long nrec,
                               const TileOut& o, int num_sms, cudaStream_t st) {
    uint64_t blocks = (nrec + 255) / 256;
    const uint64_t cap = (uint64_t)num_sms * 16;
    if (blocks > cap) blocks = cap;
    k_screen_recheck<MODEL, STAMP><<<(unsigned)blocks, 256, 0, st>>>(a.pts, a.ids, a.n, a.npad, a.ilp, a.thr,
                                                                     a.n_points, recs, nrec, o);
    return cudaGetLastError();
}

// Per-block FP64 column sums and counts of the finite values over a fixed row
// range (deterministic): a thread keeps one column (the block's threads cover
// whole rows, so a row is read by consecutive threads), the threads of a
// column are added in order.  Non-finite coordinates are left out of the
// centre, so that only their own rows (and pairs) become inconclusive for the
// screen.
constexpr uint32_t kColThreads = 512;

__global__ void __launch_bounds__(kColThreads) k_col_partial(const float* __restrict__ pts, uint32_t N, uint32_t n,
                                                             uint32_t npad, double* __restrict__ partial) {
    __shared__ double s_acc[kColThreads], s_cnt[kColThreads];
    const uint32_t rpi = kColThreads / npad;  // rows per iteration (npad <= kTileMaxN)
    const uint32_t tr = threadIdx.x / npad, d = threadIdx.x - tr * npad;
    const uint32_t per = (N + gridDim.x - 1) / gridDim.x;
    const uint32_t r0 = min(N, blockIdx.x * per), r1 = min(N, r0 + per);
    double acc = 0.0, cnt = 0.0;
    if (tr < rpi && d < n) {
#pragma unroll 4
        for (uint32_t r = r0 + tr; r < r1; r += rpi) {
            const float v = pts[(size_t)r * npad + d];
            if (isfinite(v)) {
                acc += (double)v;
                cnt += 1.0;
            }
        }
    }
    s_acc[threadIdx.x] = acc;
    s_cnt[threadIdx.x] = cnt;
    __syncthreads();
    if (threadIdx.x < n) {
        for (uint32_t t = 1; t < rpi; t++) {
            acc += s_acc[t * npad + d];
            cnt += s_cnt[t * npad + d];
        }
        partial[((size_t)blockIdx.x * n + d) * 2] = acc;
        partial[((size_t)blockIdx.x * n + d) * 2 + 1] = cnt;
    }
}

// A warp per column: the blocks' sums, lane-strided, then a fixed tree.
__global__ void k_col_mean(const double* __restrict__ partial, uint32_t nblocks, uint32_t n,
                           float* __restrict__ centre) {
    const uint32_t d = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31u;
    if (d >= n) return;
    double acc = 0.0, cnt = 0.0;
    for (uint32_t b = lane; b < nblocks; b += 32u) {
        acc += partial[((size_t)b * n + d) * 2];
        cnt += partial[((size_t)b * n + d) * 2 + 1];
    }
    for (int s = 16; s > 0; s >>= 1) {
        acc += __shfl_xor_sync(0xffffffffu, acc, s);
        cnt += __shfl_xor_sync(0xffffffffu, cnt, s);
    }
    const double m = cnt > 0.0 ? acc / cnt : 0.0;
    if (lane == 0) centre[d] = isfinite(m) ? (float)m : 0.f;
}

// Row of slot s (see the head of this file): x' = fl(x - centre), c^ =
// bf16(x'), |c^|^2 between nlo and nhi, r bounded above by the exact residual
// x' - c^ and 2^-23 of the row's length for the centring.
__global__ void k_screen_rows(const float* __restrict__ pts, uint32_t N, uint32_t n, uint32_t npad,
                              const ScreenConst sc, const float* __restrict__ centre, uint4* __restrict__ rows,
                              uint32_t* __restrict__ qg) {
    const uint32_t kch = sc.kpad >> 3;
    const uint32_t s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= (N + kGrp - 1u) / kGrp * kGrp) return;
    uint4* row = rows + (size_t)(s / kGrp) * kch * kGrp + s % kGrp;  // chunk kc at row[kc * kGrp]
    if (s >= N) {  // the last group's unused rows
        for (uint32_t kc = 0; kc < kch; kc++) row[kc * kGrp] = make_uint4(0u, 0u, 0u, 0u);
        return;
    }
    const float* x = pts + (size_t)s * npad;
    float nlo = 0.f, nhi = 0.f, rsq = 0.f;
    uint32_t w[4];
    auto bits_of = [](__nv_bfloat16 b) { return (uint32_t)__bfloat16_as_ushort(b); };
    const uint32_t full = n >> 3;  // chunks of coordinates alone
    auto coord = [&](uint32_t l) -> uint32_t {
        const float xp = __fsub_rn(x[l], centre[l]);
        const __nv_bfloat16 b = __float2bfloat16_rn(xp);
        const float f = __bfloat162float(b), e = __fsub_rn(xp, f);
        nlo = __fmaf_rd(f, f, nlo);
        nhi = __fmaf_ru(f, f, nhi);
        rsq = __fmaf_ru(e, e, rsq);
        return bits_of(b);
    };
    for (uint32_t kc = 0; kc < full; kc++) {
#pragma unroll
        for (int h = 0; h < 4; h++) {
            const uint32_t lo = coord(kc * 8u + 2u * (uint32_t)h), hi = coord(kc * 8u + 2u * (uint32_t)h + 1u);
            w[h] = lo | (hi << 16);
        }
        row[kc * kGrp] = make_uint4(w[0], w[1], w[2], w[3]);
    }
    // the remaining coordinates (fewer than 8), then A_hi, A_lo, 1, 1 and zeros
    uint32_t tail[8];
#pragma unroll
    for (uint32_t i = 0; i < 8u; i++) tail[i] = full * 8u + i < n ? coord(full * 8u + i) : 0u;
    const float len = __fsqrt_ru(nhi);
    float r = __fsqrt_ru(rsq);
    r = __fmaf_ru(0x1p-23f, __fadd_ru(len, r), r);
    const float r2 = __fmul_ru(__fadd_ru(r, r), r), r0r = __fmul_ru(__fadd_ru(sc.r0, sc.r0), r);
    const float acc = __fmul_ru(sc.c1, nhi), r0sq = __fmul_ru(sc.r0, sc.r0);
    const bool far = !(nhi <= kFar) || !(rsq <= kFar);
    uint32_t ahi, alo, ghi, glo;
    if (far) {
        ahi = ghi = 0xfb80u;  // BF16 -2^120
        alo = glo = 0u;
    } else {
        const float A = __fsub_rd(__fsub_rd(__fsub_rd(nlo, r0r), r2), acc);
        const __nv_bfloat16 h = __float2bfloat16_rn(A);
        ahi = bits_of(h);
        alo = bits_of(__float2bfloat16_rd(__fsub_rn(A, __bfloat162float(h))));
        float G = __fadd_ru(__fadd_ru(__fadd_ru(r0sq, r0r), r2), acc);
        G = __fsub_ru(__fmaf_ru(sc.c0, r0sq, G), nlo);
        const __nv_bfloat16 gh = __float2bfloat16_rn(G);
        const __nv_bfloat16 gl = __float2bfloat16_ru(__fsub_rn(G, __bfloat162float(gh)));
        ghi = bits_of(gh) ^ 0x8000u;
        glo = bits_of(gl) ^ 0x8000u;
    }
    qg[s] = ghi | (glo << 16);
    if (far) {
        for (uint32_t kc = 0; kc < full; kc++) row[kc * kGrp] = make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
        for (int i = 0; i < 8; i++) tail[i] = 0u;
    }
    for (uint32_t kc = full; kc < kch; kc++) {
        uint32_t c[8];
#pragma unroll
        for (uint32_t i = 0; i < 8u; i++) {
            const uint32_t col = kc * 8u + i;
            c[i] = col < n        ? tail[i]
                   : col == n     ? ahi
                   : col == n + 1 ? alo
                   : col < n + 4u ? 0x3f80u
                                  : 0u;
        }
        row[kc * kGrp] = make_uint4(c[0] | (c[1] << 16), c[2] | (c[3] << 16), c[4] | (c[5] << 16), c[6] | (c[7] << 16));
    }
}

uint64_t screen_rows_count(uint64_t N, uint32_t kpad) { return (N + kGrp - 1u) / kGrp * kGrp * (kpad / 8u); }

cudaError_t launch_screen_prep(const float* pts, uint32_t N, uint32_t n, uint32_t npad, const ScreenConst& sc,
                               double* partial, float* centre, uint4* rows, uint32_t* qg, cudaStream_t st) {
    if (N == 0) return cudaSuccess;
    if (sc.kpad < n + 4u || (sc.kpad & 15u) || npad > kTileMaxN) return cudaErrorInvalidValue;
    k_col_partial<<<kScreenPrepBlocks, kColThreads, 0, st>>>(pts, N, n, npad, partial);
    k_col_mean<<<(n + 7u) / 8u, 256, 0, st>>>(partial, kScreenPrepBlocks, n, centre);
    k_screen_rows<<<(unsigned)(((uint64_t)N + 7u + 255u) / 256u), 256, 0, st>>>(pts, N, n, npad, sc, centre, rows, qg);
    return cudaGetLastError();
}

bool screen_supported(uint32_t n, uint32_t npad, uint32_t k, int model, uint32_t ilp, float thr) {
    // n + 4 columns: the dimensions, the candidate's and the query's bound terms
    return tile_supported(n, npad, k, model, ilp) && ((n + 4u + 15u) & ~15u) <= kMaxKpad && n + 2u <= kTileMaxN &&
           thr >= 1e-30f && thr <= 1e30f;
}

ScreenConst make_screen_const(uint32_t n, float thr) {
    ScreenConst sc{};
    sc.kpad = (n + 4u + 15u) & ~15u;
    // R0 >= sqrt(thr / (1 - (2n + 8) 2^-24)), plus room for the FP32 evaluation of A and G
    const double r0 = std::sqrt((double)thr) * (1.0 + (2.0 * n + 8.0) * 0x1p-24 + 0x1p-19);
    sc.r0 = std::nextafter((float)r0, INFINITY);
    // FP32 accumulation (K + 32 steps of 2^-20) of at most 2.1 (|q^|^2 + |c^|^2)
    // + 1.1 R0^2 in magnitude: 2 |q^.c^| <= |q^|^2 + |c^|^2, and |A| and |G| are
    // at most (1 + 2^-6)(|c^|^2 + 2^-8 R0^2) and (1 + 2^-6)(|q^|^2 + R0^2)
    // because r <= 2^-8 (1 + 2^-7) |c^| for finite points
    sc.c1 = 2.1f * (float)(sc.kpad + 32u) * 0x1p-20f;
    sc.c0 = 1.1f * (float)(sc.kpad + 32u) * 0x1p-20f;
    return sc;
}

cudaError_t launch_screen_recheck(const JoinArgs<float>& a, const uint4* recs, unsigned long long nrec,
                                  const TileOut& o, bool stamp, int model, int num_sms, cudaStream_t st) {
    if (nrec == 0) return cudaSuccess;
    if ((a.npad & 3u) || !recs) return cudaErrorInvalidValue;
    switch (model * 2 + (stamp ? 1 : 0)) {
        case kSeq * 2: return launch_recheck_one<kSeq, false>(a, recs, nrec, o, num_sms, st);
        case kSeq * 2 + 1: return launch_recheck_one<kSeq, true>(a, recs, nrec, o, num_sms, st);
        case kIlp * 2: return launch_recheck_one<kIlp, false>(a, recs, nrec, o, num_sms, st);
        case kIlp * 2 + 1: return launch_recheck_one<kIlp, true>(a, recs, nrec, o, num_sms, st);
        case kIlpSc * 2: return launch_recheck_one<kIlpSc, false>(a, recs, nrec, o, num_sms, st);
        case kIlpSc * 2 + 1: return launch_recheck_one<kIlpSc, true>(a, recs, nrec, o, num_sms, st);
        default: return cudaErrorInvalidValue;
    }
}

cudaError_t launch_tile_screen(const JoinArgs<float>& a, const TileOut& o, const ScreenConst& sc, bool stamp,
                               int model, uint32_t nvisit, int num_sms, cudaStream_t st) {
    if (!screen_supported(a.n, a.npad, a.g.k, model, a.ilp, a.thr) || o.stride == 0 || sc.kpad < a.n + 4u ||
        !sc.rows || !sc.qg || (sc.kpad & 15u) || sc.kpad > kMaxKpad)
        return cudaErrorInvalidValue;
    if (nvisit == 0) return cudaSuccess;
    if ((uint64_t)(nvisit - 1) * o.stride >= a.num_items) return cudaErrorInvalidValue;
    uint32_t nrow = 1;  // neighbour rows: 3^(k-1)
    for (uint32_t j = 1; j < a.g.k; j++) nrow *= 3u;
    return stamp ? launch_screen_one<true>(a, o, sc, nrow, nvisit, num_sms, st)
                 : launch_screen_one<false>(a, o, sc, nrow, nvisit, num_sms, st);
}

}  // namespace gsj
