// Stable LSD radix sort and run-length encoding (subsystems (a) and (d)).
//
// Replaces the library sorts of the index build: the reference builds its
// grid on the host with a std::set and per-cell vectors (main.cu:690-857) and
// sorts its result pairs with thrust::sort_by_key (GPU.cu:863-880).  Here the
// (cell id, point id) keys are sorted on the device by this sort, which orders
// points by cell with ties in ascending point id - the reference's per-cell
// order (main.cu:741-763).
//
// Each digit pass (8-bit digits, or 9-bit where that saves a pass) is a
// reduce-then-scan over tiles of kSortTile keys:
//   k_radix_hist     per-tile digit counts, written digit-major
//   scan_u32_u32     exclusive scan of the counts: the global offset of each
//                    (digit, tile) run; with few tiles (kFewTiles) every block
//                    of the scatter derives its offsets from the counts
//                    itself, and with one tile the counts are its own
//   k_radix_scatter  the tile is ranked stably in shared memory (per-warp
//                    match_any groups, in index order), then written out in
//                    sorted order, so each digit's run of the tile is stored
//                    by consecutive threads to consecutive addresses.
// Stability: keys are ranked by (warp, round, lane) = their index order within
// the tile, and tiles are laid out in order within each digit.
#include <cstdint>
#include <cuda_runtime.h>

#include "gsj_scan.cuh"
#include "gsj_scan.h"
#include "gsj_sort.h"

namespace gsj {

namespace {

constexpr int kSortThreads = 256;
constexpr int kSortWarps = kSortThreads / 32;
constexpr int kSortItems = 8;                           // keys per thread
constexpr int kSortTile = kSortThreads * kSortItems;    // keys per tile
constexpr int kWarpKeys = kSortTile / kSortWarps;       // keys per warp (8 rounds of 32)
constexpr int kMaxBins = 512;  // digits of 8 or 9 bits
// Tiles up to which a block of the scatter reads all the tiles' digit counts (64
// x 512 words at most, 1 to 2 us) instead of two more launches per pass (a scan
// of a few thousand counts takes 5 us and its gaps): up to 131,072 keys.
constexpr uint64_t kFewTiles = 64;
static_assert(kMaxBins % kSortThreads == 0, "whole digits per thread in the tile prefix");

__device__ __forceinline__ unsigned lanemask_lt_s() {
    unsigned m;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}

template <typename K, int BINS>
__device__ __forceinline__ uint32_t digit_of(K key, int shift) {
    return (uint32_t)(key >> shift) & (uint32_t)(BINS - 1);
}

template <typename K, int BINS>
__global__ void __launch_bounds__(kSortThreads) k_radix_hist(const K* __restrict__ keys, uint64_t n, int shift,
                                                             uint32_t* __restrict__ hist, uint32_t ntiles) {
    __shared__ uint32_t h[kSortWarps][BINS];
    for (int i = threadIdx.x; i < kSortWarps * BINS; i += kSortThreads) (&h[0][0])[i] = 0u;
    __syncthreads();
    const int warp = threadIdx.x >> 5;
    const uint64_t base = (uint64_t)blockIdx.x * kSortTile;
#pragma unroll 4
    for (int i = 0; i < kSortItems; i++) {
        const uint64_t e = base + (uint64_t)i * kSortThreads + threadIdx.x;
        if (e < n) atomicAdd(&h[warp][digit_of<K, BINS>(keys[e], shift)], 1u);
    }
    __syncthreads();
    for (int d = threadIdx.x; d < BINS; d += kSortThreads) {
        uint32_t s = 0;
#pragma unroll
        for (int w = 0; w < kSortWarps; w++) s += h[w][d];
        hist[(uint64_t)d * ntiles + blockIdx.x] = s;
    }
}

template <typename K, bool VALS, int BINS>
__global__ void __launch_bounds__(kSortThreads) k_radix_scatter(const K* __restrict__ kin,
                                                                const uint32_t* __restrict__ vin,
                                                                K* __restrict__ kout, uint32_t* __restrict__ vout,
                                                                uint64_t n, int shift,
                                                                const uint32_t* __restrict__ hist, bool scanned,
                                                                uint32_t ntiles) {
    extern __shared__ __align__(16) unsigned char sort_smem[];
    K* skeys = reinterpret_cast<K*>(sort_smem);
    uint32_t* svals = reinterpret_cast<uint32_t*>(sort_smem + sizeof(K) * kSortTile);
    constexpr int DPT = BINS / kSortThreads;       // digits per thread in the tile prefix
    __shared__ uint32_t wcnt[kSortWarps][BINS];    // per-warp digit counts, then their exclusive prefix
    __shared__ uint32_t tile_off[BINS];            // exclusive prefix of the tile's digit counts
    __shared__ uint32_t gbase[BINS];               // global offset of the digit's run minus tile_off
    __shared__ uint32_t wsum[kSortWarps];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned lt = lanemask_lt_s();
    for (int i = threadIdx.x; i < kSortWarps * BINS; i += kSortThreads) (&wcnt[0][0])[i] = 0u;
    __syncthreads();

    const uint64_t base = (uint64_t)blockIdx.x * kSortTile + (uint64_t)warp * kWarpKeys;
    K key[kSortItems];
    uint32_t val[kSortItems];
    uint32_t rank[kSortItems];  // digit << 16 | rank within the warp's keys of that digit
#pragma unroll
    for (int r = 0; r < kSortItems; r++) {
        const uint64_t e = base + (uint64_t)r * 32u + lane;
        const bool valid = e < n;
        key[r] = valid ? kin[e] : K(0);
        if (VALS) val[r] = valid ? vin[e] : 0u;
        const uint32_t d = valid ? digit_of<K, BINS>(key[r], shift) : (uint32_t)BINS;
        const unsigned peers = __match_any_sync(0xffffffffu, d);
        const int leader = __ffs(peers) - 1;
        uint32_t c = 0;
        if (lane == leader && valid) {
            c = wcnt[warp][d];
            wcnt[warp][d] = c + (uint32_t)__popc(peers);
        }
        c = __shfl_sync(0xffffffffu, c, leader);
        rank[r] = (d << 16) | (c + (uint32_t)__popc(peers & lt));
        __syncwarp();
    }
    __syncthreads();
    // per digit (DPT consecutive digits a thread): prefix over the warps, then
    // over the digits
    {
        const int d0 = threadIdx.x * DPT;
        uint32_t pd[DPT];
        uint32_t p = 0;
#pragma unroll
        for (int dd = 0; dd < DPT; dd++) {
            uint32_t q = 0;
#pragma unroll
            for (int w = 0; w < kSortWarps; w++) {
                const uint32_t t = wcnt[w][d0 + dd];
                wcnt[w][d0 + dd] = q;
                q += t;
            }
            pd[dd] = q;
            p += q;
        }
        uint32_t x = p;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) wsum[warp] = x;
        __syncthreads();
        uint32_t before = 0;
#pragma unroll
        for (int w = 0; w < kSortWarps; w++)
            if (w < warp) before += wsum[w];
        uint32_t ex = before + x - p;
        // global offset of each digit's run of this tile: from the scanned counts, or
        // the digit's start over all tiles plus its counts in the tiles before
        uint32_t run[DPT];
        if (scanned) {
#pragma unroll
            for (int dd = 0; dd < DPT; dd++) run[dd] = hist[(uint64_t)(d0 + dd) * ntiles + blockIdx.x];
        } else if (ntiles == 1u) {
            uint32_t e1 = ex;
#pragma unroll
            for (int dd = 0; dd < DPT; dd++) {
                run[dd] = e1;
                e1 += pd[dd];
            }
        } else {
            uint32_t all[DPT], sum = 0;
#pragma unroll
            for (int dd = 0; dd < DPT; dd++) {
                const uint32_t* h = hist + (uint64_t)(d0 + dd) * ntiles;
                uint32_t here = 0, t_all = 0;
                for (uint32_t t = 0; t < ntiles; t++) {
                    const uint32_t c = h[t];
                    here += t < blockIdx.x ? c : 0u;
                    t_all += c;
                }
                run[dd] = here;
                all[dd] = t_all;
                sum += t_all;
            }
            unsigned long long tot;
            uint32_t start = (uint32_t)block_excl_scan<kSortThreads>(sum, &tot);
#pragma unroll
            for (int dd = 0; dd < DPT; dd++) {
                run[dd] += start;
                start += all[dd];
            }
        }
#pragma unroll
        for (int dd = 0; dd < DPT; dd++) {
            const int d = d0 + dd;
            tile_off[d] = ex;
            gbase[d] = run[dd] - ex;  // modulo 2^32, re-added below
            ex += pd[dd];
        }
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < kSortItems; r++) {
        const uint32_t d = rank[r] >> 16;
        if (d < (uint32_t)BINS) {
            const uint32_t idx = tile_off[d] + wcnt[warp][d] + (rank[r] & 0xffffu);
            skeys[idx] = key[r];
            if (VALS) svals[idx] = val[r];
        }
    }
    __syncthreads();
    const uint64_t tbase = (uint64_t)blockIdx.x * kSortTile;
    const uint32_t cnt = (uint32_t)((n - tbase) < (uint64_t)kSortTile ? (n - tbase) : (uint64_t)kSortTile);
    for (uint32_t i = threadIdx.x; i < cnt; i += kSortThreads) {
        const K kk = skeys[i];
        const uint32_t g = gbase[digit_of<K, BINS>(kk, shift)] + i;
        kout[g] = kk;
        if (VALS) vout[g] = svals[i];
    }
}

// Runs of equal keys: a run begins where a key differs from the one before it.
// Run heads among elements [e0, e0 + kScanItems), bit i for e0 + i, with the
// keys in key[]; vec: keys is 16-byte aligned.
template <typename K>
__device__ __forceinline__ uint32_t run_heads(const K* __restrict__ keys, uint64_t e0, uint64_t n, bool vec,
                                              K (&key)[kScanItems]) {
    if (vec && e0 + kScanItems <= n) {
        const uint4* p = reinterpret_cast<const uint4*>(keys + e0);
#pragma unroll
        for (int q = 0; q < kScanItems * (int)sizeof(K) / 16; q++) {
            const uint4 x = p[q];
            if constexpr (sizeof(K) == 4) {
                key[4 * q] = x.x;
                key[4 * q + 1] = x.y;
                key[4 * q + 2] = x.z;
                key[4 * q + 3] = x.w;
            } else {
                key[2 * q] = ((K)x.y << 32) | x.x;
                key[2 * q + 1] = ((K)x.w << 32) | x.z;
            }
        }
    } else {
#pragma unroll
        for (int i = 0; i < kScanItems; i++) key[i] = e0 + (uint64_t)i < n ? keys[e0 + i] : K(0);
    }
    uint32_t heads = 0;
    if (e0 < n) heads = e0 == 0 || keys[e0 - 1] != key[0] ? 1u : 0u;
#pragma unroll
    for (int i = 1; i < kScanItems; i++) heads |= (e0 + (uint64_t)i < n && key[i] != key[i - 1] ? 1u : 0u) << i;
    return heads;
}

template <typename K>
__global__ void __launch_bounds__(kScanThreads) k_run_sums(const K* __restrict__ keys, uint64_t n, bool vec,
                                                           unsigned long long* __restrict__ tsum) {
    const uint64_t e0 = blockIdx.x * kScanTile + (uint64_t)threadIdx.x * kScanItems;
    K key[kScanItems];
    const uint32_t heads = run_heads(keys, e0, n, vec, key);
    unsigned long long tot;
    block_excl_scan<kScanThreads>((unsigned long long)__popc(heads), &tot);
    if (threadIdx.x == 0) tsum[blockIdx.x] = tot;
}

// run_key, run_start and (optionally) elem_run[i] = run of element i, in one pass
// over the keys once the tiles' run counts are known (see k_tile_scan for
// `scanned`).
template <typename K>
__global__ void __launch_bounds__(kScanThreads) k_run_write(const K* __restrict__ keys, uint64_t n, bool vec,
                                                            const unsigned long long* __restrict__ tsum, bool scanned,
                                                            uint64_t* __restrict__ run_key,
                                                            uint32_t* __restrict__ run_start,
                                                            uint32_t* __restrict__ elem_run, bool vout,
                                                            uint32_t* __restrict__ nruns) {
    const uint64_t e0 = blockIdx.x * kScanTile + (uint64_t)threadIdx.x * kScanItems;
    K key[kScanItems];
    const uint32_t heads = run_heads(keys, e0, n, vec, key);
    const unsigned long long before = scanned ? tsum[blockIdx.x] : tile_prefix(tsum, blockIdx.x);
    unsigned long long tot;
    uint32_t run = (uint32_t)(before + block_excl_scan<kScanThreads>((unsigned long long)__popc(heads), &tot));
    uint32_t er[kScanItems];
#pragma unroll
    for (int i = 0; i < kScanItems; i++) {
        if ((heads >> i) & 1u) {
            run_key[run] = (uint64_t)key[i];
            run_start[run] = (uint32_t)(e0 + (uint64_t)i);
            run++;
        }
        er[i] = run - 1u;
    }
    if (elem_run) {
        if (vout && e0 + kScanItems <= n) {
            uint4* p = reinterpret_cast<uint4*>(elem_run + e0);
#pragma unroll
            for (int q = 0; q < kScanItems / 4; q++)
                p[q] = make_uint4(er[4 * q], er[4 * q + 1], er[4 * q + 2], er[4 * q + 3]);
        } else {
#pragma unroll
            for (int i = 0; i < kScanItems; i++)
                if (e0 + (uint64_t)i < n) elem_run[e0 + i] = er[i];
        }
    }
    if (blockIdx.x == gridDim.x - 1u && threadIdx.x == 0) {
        run_start[before + tot] = (uint32_t)n;
        *nruns = (uint32_t)(before + tot);
    }
}

inline unsigned blocks_for(uint64_t n, unsigned t) { return (unsigned)((n + t - 1) / t); }

inline uint64_t tiles_of(uint64_t n) { return (n + kSortTile - 1) / kSortTile; }

}  // namespace

size_t radix_sort_temp_bytes(uint64_t n) {
    const uint64_t nt = tiles_of(n);
    const size_t hist = (size_t)kMaxBins * nt * sizeof(uint32_t);
    const size_t hist_al = (2 * hist + sizeof(uint32_t) + 255) / 256 * 256;
    return hist_al + scan_u32_u64_temp_bytes((uint64_t)kMaxBins * nt) + 256;
}

template <typename K>
cudaError_t radix_sort(K* keys, K* keys_alt, uint32_t* vals, uint32_t* vals_alt, uint64_t n, int begin_bit,
                       int end_bit, void* temp, bool* in_alt, int* launches, cudaStream_t st) {
    *in_alt = false;
    if (n <= 1 || begin_bit >= end_bit) return cudaSuccess;
    if (n >= (1ull << 32)) return cudaErrorInvalidValue;
    const uint64_t nt = tiles_of(n);
    const size_t hist_bytes = (size_t)kMaxBins * nt * sizeof(uint32_t);
    uint32_t* hist = static_cast<uint32_t*>(temp);
    uint32_t* scan = reinterpret_cast<uint32_t*>(static_cast<unsigned char*>(temp) + hist_bytes);
    void* stemp = static_cast<unsigned char*>(temp) + (2 * hist_bytes + sizeof(uint32_t) + 255) / 256 * 256;
    const size_t smem = sizeof(K) * kSortTile + (vals ? sizeof(uint32_t) * kSortTile : 0);
    cudaError_t e;
    // 24 KiB at most: no opt-in needed
    // digits of 8 bits, or of 9 where that saves a pass (25 key bits: 9 + 8 + 8)
    const int B = end_bit - begin_bit;
    const int p8 = (B + 7) / 8, p9 = (B + 8) / 9;
    const int passes = p9 < p8 ? p9 : p8;
    const int nine = p9 < p8 ? B - 8 * passes : 0;  // passes with 9-bit digits
    K *ki = keys, *ko = keys_alt;
    uint32_t *vi = vals, *vo = vals_alt;
    bool alt = false;
    int shift = begin_bit;
    for (int pass = 0; pass < passes; pass++) {
        const bool wide = pass < nine;
        const uint32_t bins = wide ? 512u : 256u;
        const bool scanned = nt > kFewTiles;
        const uint32_t* offs = hist;
        int nl = 1;
        if (nt > 1) {
            if (wide) k_radix_hist<K, 512><<<(unsigned)nt, kSortThreads, 0, st>>>(ki, n, shift, hist, (uint32_t)nt);
            else k_radix_hist<K, 256><<<(unsigned)nt, kSortThreads, 0, st>>>(ki, n, shift, hist, (uint32_t)nt);
            nl++;
        }
        if (scanned) {
            e = scan_u32_u32(hist, scan, (uint64_t)bins * nt, stemp, st);
            if (e != cudaSuccess) return e;
            nl += scan_launches((uint64_t)bins * nt);
            offs = scan;
        }
        if (wide) {
            if (vals) k_radix_scatter<K, true, 512><<<(unsigned)nt, kSortThreads, smem, st>>>(ki, vi, ko, vo, n, shift, offs, scanned, (uint32_t)nt);
            else k_radix_scatter<K, false, 512><<<(unsigned)nt, kSortThreads, smem, st>>>(ki, nullptr, ko, nullptr, n, shift, offs, scanned, (uint32_t)nt);
        } else {
            if (vals) k_radix_scatter<K, true, 256><<<(unsigned)nt, kSortThreads, smem, st>>>(ki, vi, ko, vo, n, shift, offs, scanned, (uint32_t)nt);
            else k_radix_scatter<K, false, 256><<<(unsigned)nt, kSortThreads, smem, st>>>(ki, nullptr, ko, nullptr, n, shift, offs, scanned, (uint32_t)nt);
        }
        e = cudaGetLastError();
        if (e != cudaSuccess) return e;
        if (launches) *launches += nl;
        shift += wide ? 9 : 8;
        K* tk = ki;
        ki = ko;
        ko = tk;
        uint32_t* tv = vi;
        vi = vo;
        vo = tv;
        alt = !alt;
    }
    *in_alt = alt;
    return cudaSuccess;
}

template cudaError_t radix_sort<uint32_t>(uint32_t*, uint32_t*, uint32_t*, uint32_t*, uint64_t, int, int, void*,
                                          bool*, int*, cudaStream_t);
template cudaError_t radix_sort<uint64_t>(uint64_t*, uint64_t*, uint32_t*, uint32_t*, uint64_t, int, int, void*,
                                          bool*, int*, cudaStream_t);

size_t runs_temp_bytes(uint64_t n) { return scan_u32_u64_temp_bytes(n); }

template <typename K>
cudaError_t run_length(const K* keys, uint64_t n, uint64_t* run_key, uint32_t* run_start, uint32_t* elem_run,
                       uint32_t* d_nruns, void* temp, int* launches, cudaStream_t st) {
    if (n == 0) return cudaMemsetAsync(d_nruns, 0, sizeof(uint32_t), st);
    unsigned long long* tsum = static_cast<unsigned long long*>(temp);
    const uint64_t nt = (n + kScanTile - 1) / kScanTile;
    const bool scanned = nt > kDirectTiles;
    const bool vec = (reinterpret_cast<uintptr_t>(keys) & 15u) == 0;
    const bool vout = (reinterpret_cast<uintptr_t>(elem_run) & 15u) == 0;
    if (nt > 1) k_run_sums<K><<<(unsigned)nt, kScanThreads, 0, st>>>(keys, n, vec, tsum);
    if (scanned) {
        const cudaError_t e = scan_tile_sums(tsum, nt, st);
        if (e != cudaSuccess) return e;
    }
    k_run_write<K><<<(unsigned)nt, kScanThreads, 0, st>>>(keys, n, vec, tsum, scanned, run_key, run_start, elem_run,
                                                          vout, d_nruns);
    if (launches) *launches += scan_launches(n);
    return cudaGetLastError();
}

template cudaError_t run_length<uint32_t>(const uint32_t*, uint64_t, uint64_t*, uint32_t*, uint32_t*, uint32_t*, void*,
                                          int*, cudaStream_t);
template cudaError_t run_length<uint64_t>(const uint64_t*, uint64_t, uint64_t*, uint32_t*, uint32_t*, uint32_t*, void*,
                                          int*, cudaStream_t);

}  // namespace gsj
