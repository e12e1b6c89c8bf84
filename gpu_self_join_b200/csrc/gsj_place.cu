// Pair keys -> neighbour table (subsystem (d)).
//
// The reference sorts its (query id, neighbour id) result pairs by key with
// thrust::sort_by_key and finds the list boundaries with kernelUniqueKeys and
// a second sort (GPU.cu:863-980, kernel.cu:79-105).  Here the warp, tile and
// screen paths emit packed keys (query id << shift | neighbour id) in an
// arbitrary order, and the table is built without a global sort:
//   k_pair_count   list lengths: one atomic per run of equal queries in a warp
//   scan           list offsets
//   k_pair_place   each neighbour id goes to its query's list (a per-query
//                  cursor, one atomic per run of equal queries in a warp)
//   list sort      every list ascending, which also makes the table
//                  independent of the emission order: a warp per list held in
//                  registers (bitonic network) up to kWarpSortMax entries, a
//                  CTA per list (a run per warp by the same network, then
//                  merged in shared memory) up to kCtaSortMax, above that a CTA
//                  per list of LSD radix passes through a scratch copy.
// The sorts are bound by their instructions: a network with consecutive entries
// in a lane's registers has 15 stages of shuffles whatever its size, and three
// merging levels replace the long network of a CTA (28 stages through shared
// memory for 4,096 entries).  18-D 5M points (524 M entries, most in lists of
// 513 to 4,096): 13.4 -> 5.9 ms; 6-D 5M: 5.2 -> 3.3 ms; 32-D 45k: 145 -> 93 us.
// 512 entries is where a warp's network still fits its registers (80 at 16 per
// lane).
#include <cstdint>
#include <cuda_runtime.h>

#include "gsj_kernels.h"
#include "gsj_place.h"
#include "gsj_scan.h"

namespace gsj {

namespace {

constexpr unsigned long long kPadKey = ~0ull;  // unused entries of reserved blocks
constexpr uint32_t kWarpSortMax = 512;         // 16 entries per lane
constexpr int kCtaSortThreads = 256;
constexpr uint32_t kCtaSortMax = 4096;         // 16 entries per thread
constexpr int kBlockSortThreads = 256;

__device__ __forceinline__ unsigned lanemask_lt_p() {
    unsigned m;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}

// Both passes over the keys wait for memory (a key, an atomic, in the placement also
// the list's offsets and a scattered store): a thread keeps kKeys of them in flight.
// 6-D 5M points 7.4 -> 6.8 ms, 8-D 142k 53 -> 36 us, 18-D 5M unchanged (11.2 to 11.6 ms).
constexpr int kKeys = 4;

__global__ void __launch_bounds__(256) k_pair_count(const unsigned long long* __restrict__ keys, uint64_t nkeys,
                                                    uint32_t shift, uint32_t* __restrict__ counts) {
    const uint64_t stride = (uint64_t)gridDim.x * 256u * kKeys;
    for (uint64_t i0 = (uint64_t)blockIdx.x * 256u * kKeys; i0 < nkeys; i0 += stride) {
        unsigned long long kk[kKeys];
#pragma unroll
        for (int u = 0; u < kKeys; u++) {
            const uint64_t i = i0 + (uint32_t)u * 256u + threadIdx.x;
            kk[u] = i < nkeys ? keys[i] : kPadKey;
        }
#pragma unroll
        for (int u = 0; u < kKeys; u++) {
            const bool v = kk[u] != kPadKey;
            const uint32_t q = v ? (uint32_t)(kk[u] >> shift) : 0xffffffffu;
            const unsigned peers = __match_any_sync(0xffffffffu, q);
            if (v && (threadIdx.x & 31) == (unsigned)(__ffs(peers) - 1)) atomicAdd(&counts[q], (uint32_t)__popc(peers));
        }
    }
}

__global__ void __launch_bounds__(256) k_pair_place(const unsigned long long* __restrict__ keys, uint64_t nkeys,
                                                    uint32_t shift, const uint64_t* __restrict__ offsets,
                                                    uint32_t* __restrict__ cursor, uint32_t* __restrict__ table,
                                                    uint64_t cap, uint32_t* __restrict__ err) {
    const uint64_t mask = (1ull << shift) - 1ull;
    const unsigned lt = lanemask_lt_p();
    const int lane = threadIdx.x & 31;
    const uint64_t stride = (uint64_t)gridDim.x * 256u * kKeys;
    for (uint64_t i0 = (uint64_t)blockIdx.x * 256u * kKeys; i0 < nkeys; i0 += stride) {
        unsigned long long kk[kKeys];
        uint64_t begin[kKeys], end[kKeys];
        uint32_t base[kKeys];
        unsigned peers[kKeys];
#pragma unroll
        for (int u = 0; u < kKeys; u++) {
            const uint64_t i = i0 + (uint32_t)u * 256u + threadIdx.x;
            kk[u] = i < nkeys ? keys[i] : kPadKey;
        }
#pragma unroll
        for (int u = 0; u < kKeys; u++) {
            const bool v = kk[u] != kPadKey;
            const uint32_t q = v ? (uint32_t)(kk[u] >> shift) : 0xffffffffu;
            peers[u] = __match_any_sync(0xffffffffu, q);
            begin[u] = end[u] = 0;
            base[u] = 0;
            if (v) {
                if (lane == __ffs(peers[u]) - 1) base[u] = atomicAdd(&cursor[q], (uint32_t)__popc(peers[u]));
                begin[u] = offsets[q];
                end[u] = offsets[q + 1];
            }
        }
#pragma unroll
        for (int u = 0; u < kKeys; u++) {
            const uint32_t at = __shfl_sync(0xffffffffu, base[u], __ffs(peers[u]) - 1);
            if (kk[u] != kPadKey) {
                const uint64_t pos = begin[u] + at + (uint32_t)__popc(peers[u] & lt);
                if (pos < end[u] && pos < cap) table[pos] = (uint32_t)(kk[u] & mask);
                else *err = 1u;
            }
        }
    }
}

// Where entry i of a list lies in shared memory: one word in 33 is left out, so
// that a lane's consecutive entries (any power of two up to 32 of them) and the
// lanes' consecutive entries are both free of bank conflicts.
__device__ __forceinline__ uint32_t spread(uint32_t i) { return i + (i >> 5); }

// Ascending bitonic sort of 32*E entries held as E registers per lane; the result
// has entry lane*E + r in register r.  Of the log2(P)(log2(P)+1)/2 stages only 15
// exchange between lanes (for any E), the others are within a lane's registers.  A phase k
// runs ascending throughout: where it is to be descending the values are
// complemented for its duration.
template <int E>
__device__ __forceinline__ void warp_sort(uint32_t (&v)[E], int lane) {
    const unsigned FULL = 0xffffffffu;
    uint32_t flip = 0;
#pragma unroll
    for (int k = 2; k <= 32 * E; k <<= 1) {
        if (k >= E) {
            const uint32_t f = (lane & (k / E)) ? 0xffffffffu : 0u, d = f ^ flip;
            flip = f;
#pragma unroll
            for (int r = 0; r < E; r++) v[r] ^= d;
        }
#pragma unroll
        for (int j = k >> 1; j > 0; j >>= 1) {
            if (j >= E) {
                const bool lower = (lane & (j / E)) == 0;
#pragma unroll
                for (int r = 0; r < E; r++) {
                    const uint32_t o = __shfl_xor_sync(FULL, v[r], j / E);
                    v[r] = lower ? min(v[r], o) : max(v[r], o);
                }
            } else {
#pragma unroll
                for (int r = 0; r < E; r++) {
                    if (r & j) continue;
                    const bool up = k >= E || (r & k) == 0;
                    const uint32_t x = min(v[r], v[r | j]), y = max(v[r], v[r | j]);
                    v[r] = up ? x : y;
                    v[r | j] = up ? y : x;
                }
            }
        }
    }
}

// One list of n <= 32*E entries sorted by a warp; buf: its 33*E words of shared memory.
template <int E>
__device__ __forceinline__ void warp_sort_list(uint32_t* __restrict__ list, uint32_t n, int lane,
                                               uint32_t* __restrict__ buf) {
    uint32_t v[E];
#pragma unroll
    for (int r = 0; r < E; r++) {
        const uint32_t i = (uint32_t)r * 32u + (uint32_t)lane;
        v[r] = i < n ? list[i] : 0xffffffffu;
    }
    warp_sort<E>(v, lane);
    if (E > 1) {
        __syncwarp();
#pragma unroll
        for (int r = 0; r < E; r++) buf[spread((uint32_t)(lane * E + r))] = v[r];
        __syncwarp();
#pragma unroll
        for (int r = 0; r < E; r++) v[r] = buf[33 * r + lane];
    }
#pragma unroll
    for (int r = 0; r < E; r++) {
        const uint32_t i = (uint32_t)r * 32u + (uint32_t)lane;
        if (i < n) list[i] = v[r];
    }
}

// Every list of 2..kWarpSortMax entries sorted by one warp (the
// network sized to the list: 32, 64, ... 512 entries); lists above
// kWarpSortMax are gathered into long_lists (*nlong, warp-aggregated), those
// above kCtaSortMax counted in *nvery.  List l: table[offsets[l] ..
// offsets[l+1]).
template <typename OffT>
__global__ void __launch_bounds__(256) k_list_sort_short(uint32_t* __restrict__ table,
                                                         const OffT* __restrict__ offsets, uint32_t nlists,
                                                         uint32_t* __restrict__ long_lists,
                                                         uint32_t* __restrict__ nlong) {
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const unsigned lt = lanemask_lt_p();
    __shared__ uint32_t s_buf[8][33 * (kWarpSortMax / 32)];
    uint32_t* const buf = s_buf[threadIdx.x >> 5];
    const uint32_t gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint32_t nw = (gridDim.x * blockDim.x) >> 5;
    for (uint32_t l0 = gw * 32u; l0 < nlists; l0 += nw * 32u) {
        // the lengths of 32 consecutive lists, then the short ones one by one
        const uint32_t li = l0 + (uint32_t)lane;
        uint64_t b = 0, e = 0;
        if (li < nlists) {
            b = (uint64_t)offsets[li];
            e = (uint64_t)offsets[li + 1];
        }
        const uint64_t len = e - b;
        const unsigned lng = __ballot_sync(FULL, len > kWarpSortMax);
        if (lng) {
            uint32_t at = 0;
            if (lane == 0) at = atomicAdd(nlong, (uint32_t)__popc(lng));
            at = __shfl_sync(FULL, at, 0);
            if ((lng >> lane) & 1u) long_lists[at + (uint32_t)__popc(lng & lt)] = li;
            const unsigned vl = __ballot_sync(FULL, len > kCtaSortMax);
            if (vl && lane == 0) atomicAdd(nlong + 1, (uint32_t)__popc(vl));
        }
        unsigned mine = __ballot_sync(FULL, len > 1u && len <= kWarpSortMax);
        while (mine) {
            const int j = __ffs(mine) - 1;
            mine &= mine - 1u;
            uint32_t* list = table + __shfl_sync(FULL, b, j);
            const uint32_t n = (uint32_t)__shfl_sync(FULL, len, j);
            if (n <= 32u) warp_sort_list<1>(list, n, lane, buf);
            else if (n <= 64u) warp_sort_list<2>(list, n, lane, buf);
            else if (n <= 128u) warp_sort_list<4>(list, n, lane, buf);
            else if (n <= 256u) warp_sort_list<8>(list, n, lane, buf);
            else warp_sort_list<16>(list, n, lane, buf);
        }
    }
}

// One list of n <= 256*E entries sorted by the whole CTA: each warp sorts a run
// of 32*E entries in registers, then three levels of merging double the runs to
// the list's size.  A thread finds by bisection where its E outputs start in
// the two runs and merges them one by one; the outputs replace the runs in the
// same buffer after a barrier.
template <int E>
__device__ __forceinline__ void cta_sort_list(uint32_t* __restrict__ list, uint32_t n, uint32_t* __restrict__ buf) {
    constexpr uint32_t kTop = (uint32_t)kCtaSortThreads * E;
    const uint32_t t = threadIdx.x, lane = t & 31u, run0 = (t >> 5) * 32u * E;
    uint32_t v[E];
#pragma unroll
    for (int r = 0; r < E; r++) {
        const uint32_t i = run0 + (uint32_t)r * 32u + lane;
        v[r] = i < n ? list[i] : 0xffffffffu;
    }
    if (run0 < n) warp_sort<E>(v, (int)lane);
    __syncthreads();  // the buffer's last reads, by the list before
#pragma unroll
    for (int r = 0; r < E; r++) buf[spread(t * E + (uint32_t)r)] = v[r];
    __syncthreads();
#pragma unroll 1
    for (uint32_t L = 32u * E; L < kTop; L <<= 1) {
        const uint32_t a0 = (t * E) & ~(2u * L - 1u), b0 = a0 + L, diag = t * E - a0;
        if (b0 < n) {  // else the second run is empty: nothing moves
            uint32_t lo = diag > L ? diag - L : 0u, hi = min(diag, L);
            while (lo < hi) {
                const uint32_t mid = (lo + hi) >> 1;
                if (buf[spread(a0 + mid)] <= buf[spread(b0 + diag - 1u - mid)]) lo = mid + 1u;
                else hi = mid;
            }
            uint32_t ia = lo, ib = diag - lo;
            uint32_t x = ia < L ? buf[spread(a0 + ia)] : 0xffffffffu, y = ib < L ? buf[spread(b0 + ib)] : 0xffffffffu;
#pragma unroll
            for (int r = 0; r < E; r++) {
                const bool first = x <= y;
                v[r] = first ? x : y;
                ia += first ? 1u : 0u;
                ib += first ? 0u : 1u;
                const uint32_t at = first ? ia : ib;
                const uint32_t z = at < L ? buf[spread((first ? a0 : b0) + at)] : 0xffffffffu;
                x = first ? z : x;
                y = first ? y : z;
            }
        } else {
#pragma unroll
            for (int r = 0; r < E; r++) v[r] = buf[spread(t * E + (uint32_t)r)];
        }
        __syncthreads();
#pragma unroll
        for (int r = 0; r < E; r++) buf[spread(t * E + (uint32_t)r)] = v[r];
        __syncthreads();
    }
    for (uint32_t i = t; i < n; i += kCtaSortThreads) list[i] = buf[spread(i)];
}

// A CTA per list of kWarpSortMax+1 .. kCtaSortMax entries (longer lists are
// left to k_list_sort_block).
template <typename OffT>
__global__ void __launch_bounds__(kCtaSortThreads) k_list_sort_cta(uint32_t* __restrict__ table,
                                                                   const OffT* __restrict__ offsets,
                                                                   const uint32_t* __restrict__ long_lists,
                                                                   const uint32_t* __restrict__ d_nlong) {
    __shared__ uint32_t buf[kCtaSortMax + kCtaSortMax / 32];
    const uint32_t nlong = *d_nlong;
    for (uint32_t li = blockIdx.x; li < nlong; li += gridDim.x) {
        const uint32_t l = long_lists[li];
        const uint64_t b = (uint64_t)offsets[l];
        const uint32_t n = (uint32_t)((uint64_t)offsets[l + 1] - b);
        if (n > kCtaSortMax) continue;
        if (n <= 1024u) cta_sort_list<4>(table + b, n, buf);
        else if (n <= 2048u) cta_sort_list<8>(table + b, n, buf);
        else cta_sort_list<16>(table + b, n, buf);
    }
}

// One CTA per list longer than kCtaSortMax: LSD radix passes of 8 bits over
// the list's entries (ids below 2^bits), alternating between the table and
// the same range of `scratch`; the pass count is even, so the sorted list ends
// in the table.  Each pass: a digit histogram of the whole list, then its
// tiles in order, each ranked stably (per-warp match_any groups in index
// order) and written at the running offset of its digit.
template <typename OffT>
__global__ void __launch_bounds__(kBlockSortThreads) k_list_sort_block(uint32_t* __restrict__ table,
                                                                       uint32_t* __restrict__ scratch,
                                                                       const OffT* __restrict__ offsets,
                                                                       const uint32_t* __restrict__ long_lists,
                                                                       uint32_t nlong, int passes) {
    __shared__ uint32_t hist[256];
    __shared__ uint32_t run[256];
    __shared__ uint32_t wcnt[kBlockSortThreads / 32][256];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned lt = lanemask_lt_p();
    for (uint32_t li = blockIdx.x; li < nlong; li += gridDim.x) {
        const uint32_t l = long_lists[li];
        const uint64_t b = (uint64_t)offsets[l];
        const uint32_t n = (uint32_t)((uint64_t)offsets[l + 1] - b);
        if (n <= kCtaSortMax) continue;  // block-uniform: sorted by k_list_sort_cta
        uint32_t* src = table + b;
        uint32_t* dst = scratch + b;
        for (int p = 0; p < passes; p++) {
            const int shift = 8 * p;
            hist[threadIdx.x] = 0u;
            __syncthreads();
            for (uint32_t i = threadIdx.x; i < n; i += kBlockSortThreads) atomicAdd(&hist[(src[i] >> shift) & 255u], 1u);
            __syncthreads();
            if (threadIdx.x == 0) {
                uint32_t acc = 0;
                for (int d = 0; d < 256; d++) {
                    run[d] = acc;
                    acc += hist[d];
                }
            }
            __syncthreads();
            for (uint32_t t0 = 0; t0 < n; t0 += kBlockSortThreads) {
                for (int d = threadIdx.x; d < (kBlockSortThreads / 32) * 256; d += kBlockSortThreads)
                    (&wcnt[0][0])[d] = 0u;
                __syncthreads();
                const uint32_t i = t0 + threadIdx.x;
                const bool v = i < n;
                const uint32_t x = v ? src[i] : 0u;
                const uint32_t dg = v ? ((x >> shift) & 255u) : 256u;
                const unsigned peers = __match_any_sync(0xffffffffu, dg);
                const uint32_t rk = (uint32_t)__popc(peers & lt);
                if (v && lane == __ffs(peers) - 1) wcnt[warp][dg] = (uint32_t)__popc(peers);
                __syncthreads();
                uint32_t before = 0;
                if (v)
                    for (int w = 0; w < warp; w++) before += wcnt[w][dg];
                if (v) dst[run[dg] + before + rk] = x;
                __syncthreads();
                {
                    uint32_t tot = 0;
#pragma unroll
                    for (int w = 0; w < kBlockSortThreads / 32; w++) tot += wcnt[w][threadIdx.x];
                    run[threadIdx.x] += tot;
                }
                __syncthreads();
            }
            uint32_t* t = src;
            src = dst;
            dst = t;
        }
    }
}

inline unsigned grid_for(uint64_t n, unsigned t, uint64_t cap) {
    uint64_t b = (n + t - 1) / t;
    if (b > cap) b = cap;
    return (unsigned)(b ? b : 1);
}

}  // namespace

size_t place_temp_bytes(uint64_t nlists) {
    return (nlists + 64) * sizeof(uint32_t) + scan_u32_u64_temp_bytes(nlists) + 256;
}

template <typename OffT>
cudaError_t sort_lists(uint32_t* table, const OffT* offsets, uint32_t nlists, void* temp, uint32_t* d_nlong,
                       int num_sms, int* launches, cudaStream_t st) {
    if (nlists == 0) return cudaSuccess;
    uint32_t* ll = static_cast<uint32_t*>(temp);
    const unsigned g = grid_for((uint64_t)nlists, 256, (uint64_t)num_sms * 64);
    k_list_sort_short<OffT><<<g, 256, 0, st>>>(table, offsets, nlists, ll, d_nlong);
    // the longer lists' number stays on the device: a CTA that finds none ends at once
    k_list_sort_cta<OffT><<<grid_for(nlists, 1, (uint64_t)num_sms * 6), kCtaSortThreads, 0, st>>>(table, offsets, ll,
                                                                                                 d_nlong);
    if (launches) *launches += 2;
    return cudaGetLastError();
}

template <typename OffT>
cudaError_t sort_very_long_lists(uint32_t* table, uint32_t* scratch, const OffT* offsets, const void* temp,
                                 uint32_t nlong, uint32_t nvery, uint32_t id_bits, int num_sms, int* launches,
                                 cudaStream_t st) {
    if (nvery == 0) return cudaSuccess;
    if (!scratch) return cudaErrorInvalidValue;
    int passes = (int)((id_bits + 7u) / 8u);
    passes += passes & 1;  // even: the sorted list ends in the table
    k_list_sort_block<OffT><<<grid_for(nvery, 1, (uint64_t)num_sms * 8), kBlockSortThreads, 0, st>>>(
        table, scratch, offsets, static_cast<const uint32_t*>(temp), nlong, passes);
    if (launches) *launches += 1;
    return cudaGetLastError();
}

template cudaError_t sort_lists<uint64_t>(uint32_t*, const uint64_t*, uint32_t, void*, uint32_t*, int, int*,
                                          cudaStream_t);
template cudaError_t sort_very_long_lists<uint64_t>(uint32_t*, uint32_t*, const uint64_t*, const void*, uint32_t,
                                                    uint32_t, uint32_t, int, int*, cudaStream_t);

cudaError_t place_pairs(const unsigned long long* keys, uint64_t nkeys, uint32_t shift, uint32_t nlists,
                        uint32_t* counts, uint64_t* offsets, uint32_t* table, uint64_t cap, uint32_t* cursor,
                        uint32_t* err, void* temp, int num_sms, int* launches, cudaStream_t st) {
    cudaError_t e = cudaMemsetAsync(counts, 0, ((size_t)nlists + 1) * sizeof(uint32_t), st);
    if (e != cudaSuccess) return e;
    e = cudaMemsetAsync(cursor, 0, (size_t)nlists * sizeof(uint32_t), st);
    if (e != cudaSuccess) return e;
    const unsigned g = grid_for(nkeys, 256u * kKeys, (uint64_t)num_sms * 32);
    if (nkeys) k_pair_count<<<g, 256, 0, st>>>(keys, nkeys, shift, counts);
    e = scan_u32_u64(counts, offsets, nlists, temp, st);
    if (e != cudaSuccess) return e;
    if (nkeys) k_pair_place<<<g, 256, 0, st>>>(keys, nkeys, shift, offsets, cursor, table, cap, err);
    if (launches) *launches += (nkeys ? 2 : 0) + scan_launches(nlists);
    return cudaGetLastError();
}

}  // namespace gsj
