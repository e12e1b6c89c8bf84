// Device parts shared by the scans and the run-length encoding.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace gsj {

constexpr int kScanThreads = 256;
constexpr int kScanItems = 16;
constexpr uint64_t kScanTile = (uint64_t)kScanThreads * kScanItems;

__device__ __forceinline__ unsigned long long warp_incl_scan(unsigned long long x, int lane) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    return x;
}

// Block-wide exclusive scan of one value per thread (THREADS threads);
// returns the exclusive prefix and writes the block total to *total.
template <int THREADS>
__device__ __forceinline__ unsigned long long block_excl_scan(unsigned long long v, unsigned long long* total) {
    __shared__ unsigned long long wsum[THREADS / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned long long inc = warp_incl_scan(v, lane);
    if (lane == 31) wsum[warp] = inc;
    __syncthreads();
    if (warp == 0) {
        unsigned long long w = lane < THREADS / 32 ? wsum[lane] : 0ull;
        w = warp_incl_scan(w, lane);
        if (lane < THREADS / 32) wsum[lane] = w;
    }
    __syncthreads();
    const unsigned long long before = warp ? wsum[warp - 1] : 0ull;
    *total = wsum[THREADS / 32 - 1];
    __syncthreads();
    return before + inc - v;
}

// Elements [e0, e0 + kScanItems) (zero past n); vec: in is 16-byte aligned.
__device__ __forceinline__ void load_items(const uint32_t* __restrict__ in, uint64_t e0, uint64_t n, bool vec,
                                           uint32_t (&v)[kScanItems]) {
    if (vec && e0 + kScanItems <= n) {
        const uint4* p = reinterpret_cast<const uint4*>(in + e0);
#pragma unroll
        for (int q = 0; q < kScanItems / 4; q++) {
            const uint4 x = p[q];
            v[4 * q] = x.x;
            v[4 * q + 1] = x.y;
            v[4 * q + 2] = x.z;
            v[4 * q + 3] = x.w;
        }
    } else {
#pragma unroll
        for (int i = 0; i < kScanItems; i++) v[i] = e0 + (uint64_t)i < n ? in[e0 + i] : 0u;
    }
}

// Sum of tsum[0 .. tile) for the whole block.
__device__ __forceinline__ unsigned long long tile_prefix(const unsigned long long* __restrict__ tsum, uint64_t tile) {
    unsigned long long s = 0, tot;
    for (uint64_t i = threadIdx.x; i < tile; i += kScanThreads) s += tsum[i];
    block_excl_scan<kScanThreads>(s, &tot);
    return tot;
}

// Up to this many tiles every block of a scan adds up the sums of the tiles
// before its own (at most 8 loads a thread) instead of waiting for a launch of
// one block that scans them.
constexpr uint64_t kDirectTiles = 2048;

// tsum[i] becomes the exclusive prefix of the tile sums, tsum[ntiles] the total (one block).
cudaError_t scan_tile_sums(unsigned long long* tsum, uint64_t ntiles, cudaStream_t st);

}  // namespace gsj
