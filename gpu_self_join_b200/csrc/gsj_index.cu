// Grid index construction on the device (subsystem (a)).
//
// Replaces the reference's host-side index build, which is restated here with
// the same arithmetic so that every point lands in the same cell:
//   ReorderByDimension        main.cu:981-1075   (variance statistic: k_variance)
//   generateNDGridDimensions  main.cu:891-948    (k_minmax_*; the scalar tail runs on the host)
//   populateNDGridIndexAndLookupArray + getLinearID_nDimensions
//                             main.cu:690-883    (k_cell_keys -> radix sort -> runs -> lookup)
//   computeWorkDifficulty     GPU.cu:1491-1525   (k_item_* work items, heavy cells first)
#include <cstdint>
#include <cuda_runtime.h>
#include <type_traits>

#include "gsj_common.cuh"
#include "gsj_fp.cuh"
#include "gsj_kernels.h"
#include "gsj_scan.cuh"

namespace gsj {

// ------------------------------------------------------------ REORDER statistic
// Every dimension's sampled values (rows 0, 100, 200, ...) are added one after
// another in the reference's order, unfused, in T: a chain of dependent additions
// per dimension, twice (mean, then squared deviations).  A block takes 8
// dimensions (a 32-byte sector of a row in FP32); its warps 1.. stage the next
// chunk of samples, in the second pass already as squared deviations, while the
// first 8 lanes of warp 0 add the current one from shared memory, 16 values read
// ahead of the chain.
// Bound by the additions' latency (4 cycles) and the staging of one block.  Against
// one block that staged and added in turn: 18-D 5M points 1.38 -> 0.48 ms, 90-D
// 515k 460 -> 66 us, 8-D 120k 26 -> 16 us.
constexpr uint32_t kVarDims = 8, kVarThreads = 1024, kVarUnroll = 16;
template <typename T>
constexpr uint32_t kVarChunk = 992u * 4u / sizeof(T);  // samples: 8 (FP32) or 4 loads a thread
template <typename T>
constexpr size_t kVarSmem = 2u * kVarChunk<T> * kVarDims * sizeof(T);

template <typename T>
__global__ void __launch_bounds__(kVarThreads, 1) k_variance(const T* __restrict__ in, uint64_t N, uint32_t n, T denom,
                                                          T* __restrict__ var_out) {
    extern __shared__ unsigned char smem_raw[];
    T* const stage = reinterpret_cast<T*>(smem_raw);
    __shared__ T s_avg[kVarDims];
    constexpr uint32_t C = kVarChunk<T>, E = C * kVarDims;
    const uint32_t d0 = blockIdx.x * kVarDims, nd = min(kVarDims, n - d0);
    const uint64_t nsamp = (N + 99) / 100;
    const uint64_t nchunk = (nsamp + C - 1) / C;
    T avg = 0;
    // elements t, t + nt, ... of chunk c into its buffer
    auto fill = [&](uint64_t c, int pass, uint32_t t, uint32_t nt) {
        T* const dst = stage + (c & 1u) * E;
        const uint64_t s0 = c * C;
        const uint32_t cnt = (uint32_t)min((uint64_t)C, nsamp - s0) * kVarDims;
        const T a = pass ? s_avg[t & (kVarDims - 1u)] : T(0);  // nt is a multiple of kVarDims
#pragma unroll 4
        for (uint32_t e = t; e < cnt; e += nt) {
            const uint32_t d = e & (kVarDims - 1u);
            T v = d < nd ? in[(s0 + e / kVarDims) * 100ull * n + d0 + d] : T(0);
            if (pass) {
                const T dv = FP<T>::sub(v, a);
                v = FP<T>::mul(dv, dv);
            }
            dst[e] = v;
        }
    };
    for (int pass = 0; pass < 2; pass++) {
        T sum = 0;
        fill(0, pass, threadIdx.x, kVarThreads);
        __syncthreads();
        for (uint64_t c = 0; c < nchunk; c++) {
            if (threadIdx.x < 32u) {
                if (threadIdx.x < nd) {
                    const T* const p = stage + (c & 1u) * E + threadIdx.x;
                    const uint32_t cs = (uint32_t)min((uint64_t)C, nsamp - c * C);
                    uint32_t s = 0;
                    for (; s + kVarUnroll <= cs; s += kVarUnroll) {
                        T v[kVarUnroll];
#pragma unroll
                        for (uint32_t u = 0; u < kVarUnroll; u++) v[u] = p[(s + u) * kVarDims];
#pragma unroll
                        for (uint32_t u = 0; u < kVarUnroll; u++) sum = FP<T>::add(sum, v[u]);
                    }
                    for (; s < cs; s++) sum = FP<T>::add(sum, p[s * kVarDims]);
                }
            } else if (c + 1 < nchunk) {
                fill(c + 1, pass, threadIdx.x - 32u, kVarThreads - 32u);
            }
            __syncthreads();
        }
        if (threadIdx.x < nd) {
            avg = FP<T>::div(sum, denom);
            if (pass == 0) s_avg[threadIdx.x] = avg;
            else var_out[d0 + threadIdx.x] = avg;
        }
        __syncthreads();
    }
}

// ------------------------------------------------------------ grid extents
// Per indexed dim j (input column perm[j]): min/max with the reference's
// sequential semantics (start from point 0, replace on strict < / >), so NaN
// values other than point 0's are skipped exactly as main.cu:906-916 skips them.
template <typename T>
__global__ void k_minmax_partial(const T* __restrict__ in, uint64_t N, uint32_t n, uint32_t k,
                                 const uint32_t* __restrict__ perm, T* __restrict__ part) {
    __shared__ T smin[kMaxK][32], smax[kMaxK][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    T mn[kMaxK], mx[kMaxK];
    uint32_t col[kMaxK];
#pragma unroll
    for (int j = 0; j < kMaxK; j++)
        if (j < (int)k) {
            col[j] = perm ? perm[j] : (uint32_t)j;
            mn[j] = mx[j] = in[col[j]];
        }
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    // four points per round, their loads issued together
    for (; i + 3u * stride < N; i += 4u * stride) {
#pragma unroll
        for (int j = 0; j < kMaxK; j++)
            if (j < (int)k) {
                T v[4];
#pragma unroll
                for (int u = 0; u < 4; u++) v[u] = in[(i + (uint64_t)u * stride) * n + col[j]];
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    if (v[u] < mn[j]) mn[j] = v[u];
                    if (v[u] > mx[j]) mx[j] = v[u];
                }
            }
    }
    for (; i < N; i += stride) {
#pragma unroll
        for (int j = 0; j < kMaxK; j++)
            if (j < (int)k) {
                const T v = in[i * n + col[j]];
                if (v < mn[j]) mn[j] = v;
                if (v > mx[j]) mx[j] = v;
            }
    }
#pragma unroll
    for (int j = 0; j < kMaxK; j++)
        if (j < (int)k) {
            for (int o = 16; o > 0; o >>= 1) {
                const T a = __shfl_down_sync(0xffffffffu, mn[j], o);
                const T b = __shfl_down_sync(0xffffffffu, mx[j], o);
                if (a < mn[j]) mn[j] = a;
                if (b > mx[j]) mx[j] = b;
            }
            if (lane == 0) { smin[j][warp] = mn[j]; smax[j][warp] = mx[j]; }
        }
    __syncthreads();
    if (warp == 0) {
        const int nw = blockDim.x >> 5;
        for (int j = 0; j < (int)k; j++) {
            T a = lane < nw ? smin[j][lane] : smin[j][0];
            T b = lane < nw ? smax[j][lane] : smax[j][0];
            for (int o = 16; o > 0; o >>= 1) {
                const T a2 = __shfl_down_sync(0xffffffffu, a, o);
                const T b2 = __shfl_down_sync(0xffffffffu, b, o);
                if (a2 < a) a = a2;
                if (b2 > b) b = b2;
            }
            if (lane == 0) {
                part[(size_t)blockIdx.x * 2 * k + j] = a;
                part[(size_t)blockIdx.x * 2 * k + k + j] = b;
            }
        }
    }
}

// Warp j reduces dim j's partials (every partial starts from point 0's value,
// so the strict comparisons keep the sequential semantics in any order).
template <typename T>
__global__ void k_minmax_final(const T* __restrict__ part, uint32_t nparts, uint32_t k,
                               T* __restrict__ out) {
    const uint32_t j = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    if (j >= k) return;
    T a = part[j], b = part[k + j];
    for (uint32_t p = lane; p < nparts; p += 32u) {
        const T a2 = part[(size_t)p * 2 * k + j], b2 = part[(size_t)p * 2 * k + k + j];
        if (a2 < a) a = a2;
        if (b2 > b) b = b2;
    }
    for (int o = 16; o > 0; o >>= 1) {
        const T a2 = __shfl_down_sync(0xffffffffu, a, o);
        const T b2 = __shfl_down_sync(0xffffffffu, b, o);
        if (a2 < a) a = a2;
        if (b2 > b) b = b2;
    }
    if (lane == 0) {
        out[j] = a;
        out[k + j] = b;
    }
}

// ------------------------------------------------------------ cell keys
// Cell coordinate (x - minArr)/eps truncated to unsigned (main.cu:713,744 and
// kernel.cu:184 compute it identically), linear id with dim 0 fastest.
// Linear cell id of point i (dim 0 fastest); a coordinate whose index
// reaches the grid's extent (eps below the data's resolution, so that the
// rounded max + eps equals max) raises *bad and counts as cell 0.
template <typename T>
__device__ __forceinline__ uint64_t cell_key_of(const T* __restrict__ in, uint64_t i, uint32_t n,
                                                const uint32_t* __restrict__ perm, const GridGeom& g,
                                                const MinVals<T>& minArr, T eps, uint32_t* bad) {
    uint64_t key = 0;
    bool out = false;
#pragma unroll
    for (int j = 0; j < kMaxK; j++)
        if (j < (int)g.k) {
            const T x = in[i * n + (perm ? perm[j] : (uint32_t)j)];
            const uint32_t c = FP<T>::to_uint_rz(FP<T>::div(FP<T>::sub(x, minArr.v[j]), eps));
            out |= c >= g.ncells[j];
            key += (uint64_t)c * g.mult[j];
        }
    if (out) {
        *bad = 1u;
        key = 0;
    }
    return key;
}

template <typename T, typename K>
__global__ void k_cell_keys(const T* __restrict__ in, uint64_t N, uint32_t n, const uint32_t* __restrict__ perm,
                            GridGeom g, MinVals<T> minArr, T eps,
                            K* __restrict__ keys, uint32_t* __restrict__ vals, uint32_t* __restrict__ bad) {
    const uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    if (i >= N) return;
    keys[i] = (K)cell_key_of<T>(in, i, n, perm, g, minArr, eps, bad);
    vals[i] = (uint32_t)i;
}

// Points in cell order with reordered, zero-padded columns: pts[s][j] = in[ids[s]][perm[j]].
template <typename T>
__global__ void k_gather_points(const T* __restrict__ in, uint64_t N, uint32_t n, uint32_t npad,
                                const uint32_t* __restrict__ perm, const uint32_t* __restrict__ ids,
                                T* __restrict__ pts) {
    const uint64_t e = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    if (e >= N * npad) return;
    const uint64_t s = e / npad;
    const uint32_t j = (uint32_t)(e - s * npad);
    pts[e] = j < n ? in[(uint64_t)ids[s] * n + (perm ? perm[j] : j)] : T(0);
}

// The same for rows of npad = NP <= 4 entries: a thread per point, one id
// load and the row stored as one vector.
template <typename T, int NP>
__global__ void k_gather_rows(const T* __restrict__ in, uint64_t N, uint32_t n, const uint32_t* __restrict__ perm,
                              const uint32_t* __restrict__ ids, T* __restrict__ pts) {
    const uint64_t s = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    if (s >= N) return;
    const T* src = in + (uint64_t)ids[s] * n;
    T v[NP];
#pragma unroll
    for (int j = 0; j < NP; j++) v[j] = (uint32_t)j < n ? src[perm ? perm[j] : (uint32_t)j] : T(0);
    T* dst = pts + s * NP;
    if constexpr (std::is_same<T, float>::value && NP == 2) {
        *reinterpret_cast<float2*>(dst) = make_float2(v[0], v[1]);
    } else if constexpr (std::is_same<T, float>::value && NP == 4) {
        *reinterpret_cast<float4*>(dst) = make_float4(v[0], v[1], v[2], v[3]);
    } else if constexpr (std::is_same<T, double>::value && NP >= 2) {
#pragma unroll
        for (int j = 0; j < NP; j += 2) *reinterpret_cast<double2*>(dst + j) = make_double2(v[j], v[j + 1]);
    } else {
#pragma unroll
        for (int j = 0; j < NP; j++) dst[j] = v[j];
    }
}

// ------------------------------------------------------------ cell lookup
// First index of sorted keys[0 .. M) at or past `v`, found by a warp: 32 probes
// cut the range to a 33rd at a time.
__device__ __forceinline__ uint32_t warp_lower_bound(const uint64_t* __restrict__ keys, uint32_t M, uint64_t v) {
    const uint32_t lane = threadIdx.x & 31u;
    uint32_t lo = 0, hi = M;
    while (lo < hi) {
        const uint32_t step = (hi - lo) / 33u + 1u;
        const uint32_t at = (uint32_t)min((uint64_t)hi - 1u, (uint64_t)lo + (uint64_t)(lane + 1u) * step - 1u);
        const uint32_t below = (uint32_t)__popc(__ballot_sync(0xffffffffu, keys[at] < v));  // a prefix of the lanes
        // keys[probe of lane below - 1] < v <= keys[probe of lane below]
        const uint64_t nlo = below ? min((uint64_t)hi, (uint64_t)lo + (uint64_t)below * step) : lo;
        const uint64_t nhi = below < 32u ? min((uint64_t)hi - 1u, (uint64_t)lo + (uint64_t)(below + 1u) * step - 1u) : hi;
        lo = (uint32_t)nlo;
        hi = (uint32_t)(nhi < nlo ? nlo : nhi);
    }
    return lo;
}

// Slot-prefix table of a dense grid: ds[L] = points in cells below L, for L in
// [0, total] (cell L holds slots [ds[L], ds[L+1])).  A block owns kScanTile
// linear ids: it finds its cells in the sorted list, marks their places, and
// the rank of every place leads to the first slot of the next cell.  (Before:
// a cleared count array, a scatter of the cells' sizes and a scan of the
// whole grid, three more passes over it.)
__global__ void __launch_bounds__(kScanThreads) k_dense_slots(const uint64_t* __restrict__ cell_key,
                                                              const uint32_t* __restrict__ cell_start, uint32_t M,
                                                              uint64_t total, uint32_t* __restrict__ ds) {
    __shared__ uint32_t mark[kScanTile / 32];
    __shared__ uint32_t starts[kScanTile + 1];
    __shared__ uint32_t range[2];
    const uint64_t l0 = blockIdx.x * kScanTile;
    if (threadIdx.x < kScanTile / 32) mark[threadIdx.x] = 0u;
    if (threadIdx.x < 64u) {
        const uint32_t w = threadIdx.x >> 5;
        const uint32_t r = warp_lower_bound(cell_key, M, l0 + w * kScanTile);
        if ((threadIdx.x & 31u) == 0u) range[w] = r;
    }
    __syncthreads();
    const uint32_t c0 = range[0], n = range[1] - c0;
    for (uint32_t i = threadIdx.x; i <= n; i += kScanThreads) {
        starts[i] = cell_start[c0 + i];
        if (i < n) {
            const uint32_t at = (uint32_t)(cell_key[c0 + i] - l0);
            atomicOr(&mark[at >> 5], 1u << (at & 31u));
        }
    }
    __syncthreads();
    const uint32_t bits = (mark[threadIdx.x >> 1] >> (16u * (threadIdx.x & 1u))) & 0xffffu;
    unsigned long long tot;
    uint32_t rank = (uint32_t)block_excl_scan<kScanThreads>((unsigned long long)__popc(bits), &tot);
    const uint64_t e0 = l0 + (uint64_t)threadIdx.x * kScanItems;
    uint32_t o[kScanItems];
#pragma unroll
    for (int i = 0; i < kScanItems; i++) {
        o[i] = starts[rank];
        rank += (bits >> i) & 1u;
    }
    if (e0 + kScanItems <= total + 1u) {
        uint4* p = reinterpret_cast<uint4*>(ds + e0);
#pragma unroll
        for (int q = 0; q < kScanItems / 4; q++) p[q] = make_uint4(o[4 * q], o[4 * q + 1], o[4 * q + 2], o[4 * q + 3]);
    } else {
#pragma unroll
        for (int i = 0; i < kScanItems; i++)
            if (e0 + (uint64_t)i <= total) ds[e0 + i] = o[i];
    }
}

// Entries {linear id of the row's cell 0, first cell, cells} of the grid rows
// that hold a cell; n0: cells of dim 0.  The first cell of a row finds the row's
// end by a galloping search.
__global__ void k_row_insert(const uint64_t* __restrict__ cell_key, uint32_t M, uint32_t n0, uint4* htab,
                             uint64_t hmask) {
    const uint32_t c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= M) return;
    const unsigned long long key = cell_key[c];
    const unsigned long long base = key - key % n0;
    if (c > 0u && cell_key[c - 1u] >= base) return;
    // cells [c, lo) are in the row, hi (if below M) is not
    uint32_t lo = c + 1u, hi = M;
    for (uint32_t step = 1u; lo < M; step <<= 1) {
        const uint32_t probe = step < M - lo ? lo + step - 1u : M - 1u;
        if (cell_key[probe] - base >= n0) {
            hi = probe;
            break;
        }
        lo = probe + 1u;
    }
    while (lo < hi) {
        const uint32_t m = lo + (hi - lo) / 2u;
        if (cell_key[m] - base < n0) lo = m + 1u;
        else hi = m;
    }
    const uint64_t h = mix64(base);
    for (uint64_t probe = 0; probe <= hmask; probe++) {
        uint4* e = htab + ((h + probe) & hmask);
        const unsigned long long prev =
            atomicCAS(reinterpret_cast<unsigned long long*>(e), (unsigned long long)kEmptyKey, base);
        if (prev == kEmptyKey) {
            e->z = c;
            e->w = lo - c;
            return;
        }
    }
}

// Cell plan of dense low-dimensional grids (k <= 3): for every non-empty
// cell and each of its 3^(k-1) neighbour rows, the slot range of the row's
// cells x-1..x+1, clipped to the grid (kernel.cu:180-188 clamp the same way).
// These cells have consecutive linear ids (dim 0 is fastest), so the range is
// [ds[row + xlo], ds[row + xhi + 1]).
__global__ void k_cell_plan(const uint64_t* __restrict__ cell_key, uint32_t M, GridGeom g,
                            const uint32_t* __restrict__ ds, uint2* __restrict__ plan) {
    const uint32_t c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= M) return;
    const uint32_t k = g.k;
    const uint32_t key = (uint32_t)cell_key[c];
    const uint32_t n0 = g.ncells[0];
    const uint32_t o0 = key % n0, rest = key / n0;
    const uint32_t o1 = k >= 2 ? rest % g.ncells[1] : 0u;
    const uint32_t o2 = k >= 3 ? rest / g.ncells[1] : 0u;
    const uint32_t nrows = k == 1 ? 1u : (k == 2 ? 3u : 9u);
    const uint32_t xlo = o0 > 0 ? o0 - 1u : 0u;
    const uint32_t xhi = o0 + 1u < n0 ? o0 + 1u : n0 - 1u;
    for (uint32_t r = 0; r < nrows; r++) {
        const long long r1 = (long long)o1 + (k >= 2 ? (long long)(r % 3) - 1 : 0);
        const long long r2 = (long long)o2 + (k >= 3 ? (long long)(r / 3) - 1 : 0);
        uint2 e = make_uint2(0u, 0u);
        const bool ok = (k < 2 || (r1 >= 0 && r1 < (long long)g.ncells[1])) &&
                        (k < 3 || (r2 >= 0 && r2 < (long long)g.ncells[2]));
        if (ok) {
            const uint32_t rowbase = (uint32_t)r1 * n0 + (k >= 3 ? (uint32_t)r2 * (uint32_t)g.mult[2] : 0u);
            const uint32_t lo = ds[rowbase + xlo];
            e = make_uint2(lo, ds[rowbase + xhi + 1u] - lo);
        }
        plan[(size_t)c * nrows + r] = e;
    }
}

// Row plan of the warp join on hashed grids with k <= 3.  A warp of the join has at
// most 9 rows to look up, so most of its lanes would idle through the dependent
// loads (entry, a search among the row's cells, keys and slots) that a thread each
// does here for 128 neighbouring cells at a time, whose searches share their
// lines.  Count stage, lookups in the join / plan (the plan's launch included),
// with the earlier hash of single cells before: 2-D double 1M points 1.35, 1.90 /
// 0.97 ms, 1-D double 1M 1.12, 1.50 / 0.75, 3-D double 3M 4.86, 5.59 / 3.20, 2-D
// float 4M 4.15, 4.47 / 2.87.
constexpr uint32_t kPlanCells = 128, kPlanRows = 9;

template <typename T, bool STAMP>
__global__ void __launch_bounds__(kPlanCells) k_row_plan(const JoinArgs<T> a, uint32_t nrow, uint2* __restrict__ plan) {
    __shared__ uint2 out[kPlanCells * kPlanRows];
    const uint32_t c0 = blockIdx.x * kPlanCells, c = c0 + threadIdx.x;
    if (c < a.num_cells) {
        const uint64_t key = a.cell_key[c];
        uint32_t own[kMaxK] = {};
        uint64_t t = key;
#pragma unroll
        for (int j = 0; j < 3; j++)
            if (j < (int)a.g.k) {
                own[j] = (uint32_t)(t % a.g.ncells[j]);
                t /= a.g.ncells[j];
            }
        uint32_t lowmask, highmask, oddmask;
        cell_masks(own, a.g, lowmask, highmask, oddmask);
        for (uint32_t r = 0; r < nrow; r++) {
            uint32_t start, cnt;
            row_range<T, STAMP>(a, true, r, key, own[0], lowmask, highmask, oddmask, start, cnt);
            out[threadIdx.x * nrow + r] = make_uint2(start, cnt);
        }
    }
    __syncthreads();
    const uint32_t n = min(kPlanCells, a.num_cells - c0) * nrow;
    for (uint32_t i = threadIdx.x; i < n; i += kPlanCells) plan[(size_t)c0 * nrow + i] = out[i];
}

// ------------------------------------------------------------ work items
// A work item is one chunk of up to `qchunk` consecutive query slots of one cell.
__global__ void k_item_counts(const uint32_t* __restrict__ cell_start, const uint32_t* __restrict__ order,
                              uint32_t M, uint32_t qchunk, uint32_t* __restrict__ nchunks,
                              uint32_t* __restrict__ sizes) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= M) return;
    const uint32_t c = order ? order[i] : i;
    const uint32_t sz = cell_start[c + 1] - cell_start[c];
    nchunks[i] = (sz + qchunk - 1) / qchunk;
    if (sizes) sizes[i] = ~sz;  // complemented: an ascending sort gives the descending order
}

__global__ void k_make_items(const uint32_t* __restrict__ order, const uint32_t* __restrict__ nchunks,
                             const uint32_t* __restrict__ item_off, uint32_t M, uint2* __restrict__ items) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= M) return;
    const uint32_t c = order ? order[i] : i;
    const uint32_t off = item_off[i], nc = nchunks[i];
    for (uint32_t q = 0; q < nc; q++) items[off + q] = make_uint2(c, q);
}

// Neighbour offsets in the kernels' order (digit j of o is dim j's step + 1):
// linear-id delta (x lo, y hi), moved-down dims | moved-up dims << 16, highest
// moved dim (0xff: none).
__global__ void k_neighbour_table(GridGeom g, uint32_t noff, uint4* __restrict__ tab) {
    const uint32_t o = blockIdx.x * blockDim.x + threadIdx.x;
    if (o >= noff) return;
    uint64_t delta = 0;
    uint32_t down = 0, up = 0, hd = 0xffu, t = o;
    for (uint32_t j = 0; j < g.k; j++) {
        const uint32_t d = t % 3u;
        t /= 3u;
        if (d == 0u) {
            delta -= g.mult[j];
            down |= 1u << j;
        } else if (d == 2u) {
            delta += g.mult[j];
            up |= 1u << j;
        }
        if (d != 1u) hd = j;
    }
    tab[o] = make_uint4((uint32_t)delta, (uint32_t)(delta >> 32), down | (up << 16), hd);
}

__global__ void k_iota(uint32_t* __restrict__ out, uint32_t M) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < M) out[i] = i;
}



// ------------------------------------------------------------ launchers
static inline unsigned blocks_for(uint64_t n, unsigned t) { return (unsigned)((n + t - 1) / t); }

template <typename T>
cudaError_t launch_variance(const T* in, uint64_t N, uint32_t n, T denom, T* var_out, cudaStream_t st) {
    const int smem = (int)kVarSmem<T>;
    cudaError_t e = cudaFuncSetAttribute(k_variance<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    k_variance<T><<<(n + kVarDims - 1u) / kVarDims, kVarThreads, smem, st>>>(in, N, n, denom, var_out);
    return cudaGetLastError();
}

template <typename T>
cudaError_t launch_minmax(const T* in, uint64_t N, uint32_t n, uint32_t k, const uint32_t* perm, T* part,
                          uint32_t nparts, T* out, cudaStream_t st) {
    k_minmax_partial<T><<<nparts, 256, 0, st>>>(in, N, n, k, perm, part);
    k_minmax_final<T><<<1, 32u * k, 0, st>>>(part, nparts, k, out);
    return cudaGetLastError();
}

template <typename T, typename K>
cudaError_t launch_cell_keys(const T* in, uint64_t N, uint32_t n, const uint32_t* perm, const GridGeom& g,
                             const MinVals<T>& minArr, T eps, K* keys, uint32_t* vals, uint32_t* bad,
                             cudaStream_t st) {
    k_cell_keys<T, K><<<blocks_for(N, 256), 256, 0, st>>>(in, N, n, perm, g, minArr, eps, keys, vals, bad);
    return cudaGetLastError();
}

template <typename T>
cudaError_t launch_gather_points(const T* in, uint64_t N, uint32_t n, uint32_t npad, const uint32_t* perm,
                                 const uint32_t* ids, T* pts, cudaStream_t st) {
    if (npad == 1) k_gather_rows<T, 1><<<blocks_for(N, 256), 256, 0, st>>>(in, N, n, perm, ids, pts);
    else if (npad == 2) k_gather_rows<T, 2><<<blocks_for(N, 256), 256, 0, st>>>(in, N, n, perm, ids, pts);
    else if (npad == 4) k_gather_rows<T, 4><<<blocks_for(N, 256), 256, 0, st>>>(in, N, n, perm, ids, pts);
    else k_gather_points<T><<<blocks_for(N * npad, 256), 256, 0, st>>>(in, N, n, npad, perm, ids, pts);
    return cudaGetLastError();
}


cudaError_t launch_dense_slots(const uint64_t* cell_key, const uint32_t* cell_start, uint32_t M, uint64_t total,
                               uint32_t* ds, cudaStream_t st) {
    if (reinterpret_cast<uintptr_t>(ds) & 15u) return cudaErrorInvalidValue;
    k_dense_slots<<<(unsigned)((total + 1u + kScanTile - 1u) / kScanTile), kScanThreads, 0, st>>>(cell_key, cell_start,
                                                                                                  M, total, ds);
    return cudaGetLastError();
}

cudaError_t launch_row_table(const uint64_t* cell_key, uint32_t M, uint32_t n0, uint4* htab, uint64_t hmask,
                             cudaStream_t st) {
    k_row_insert<<<blocks_for(M, 256), 256, 0, st>>>(cell_key, M, n0, htab, hmask);
    return cudaGetLastError();
}

cudaError_t launch_cell_plan(const uint64_t* cell_key, uint32_t M, const GridGeom& g, const uint32_t* ds,
                             uint2* plan, cudaStream_t st) {
    k_cell_plan<<<blocks_for(M, 256), 256, 0, st>>>(cell_key, M, g, ds, plan);
    return cudaGetLastError();
}

template <typename T>
cudaError_t launch_row_plan(const JoinArgs<T>& a, bool stamp, uint2* plan, cudaStream_t st) {
    if (a.g.k < 1 || a.g.k > 3 || !a.nbtab || a.num_cells == 0) return cudaErrorInvalidValue;
    const uint32_t nrow = a.g.k == 1 ? 1u : (a.g.k == 2 ? 3u : 9u);
    const unsigned blocks = blocks_for(a.num_cells, kPlanCells);
    if (stamp) k_row_plan<T, true><<<blocks, kPlanCells, 0, st>>>(a, nrow, plan);
    else k_row_plan<T, false><<<blocks, kPlanCells, 0, st>>>(a, nrow, plan);
    return cudaGetLastError();
}

cudaError_t launch_item_counts(const uint32_t* cell_start, const uint32_t* order, uint32_t M, uint32_t qchunk,
                               uint32_t* nchunks, uint32_t* sizes, cudaStream_t st) {
    k_item_counts<<<blocks_for(M, 256), 256, 0, st>>>(cell_start, order, M, qchunk, nchunks, sizes);
    return cudaGetLastError();
}

cudaError_t launch_make_items(const uint32_t* order, const uint32_t* nchunks, const uint32_t* item_off,
                              uint32_t M, uint2* items, cudaStream_t st) {
    k_make_items<<<blocks_for(M, 256), 256, 0, st>>>(order, nchunks, item_off, M, items);
    return cudaGetLastError();
}

cudaError_t launch_neighbour_table(const GridGeom& g, uint32_t noff, uint4* tab, cudaStream_t st) {
    k_neighbour_table<<<blocks_for(noff, 256), 256, 0, st>>>(g, noff, tab);
    return cudaGetLastError();
}

cudaError_t launch_iota(uint32_t* out, uint32_t M, cudaStream_t st) {
    k_iota<<<blocks_for(M, 256), 256, 0, st>>>(out, M);
    return cudaGetLastError();
}


#define GSJ_INST_INDEX(T)                                                                                  \
    template cudaError_t launch_variance<T>(const T*, uint64_t, uint32_t, T, T*, cudaStream_t);           \
    template cudaError_t launch_minmax<T>(const T*, uint64_t, uint32_t, uint32_t, const uint32_t*, T*,     \
                                          uint32_t, T*, cudaStream_t);                                     \
    template cudaError_t launch_cell_keys<T, uint64_t>(const T*, uint64_t, uint32_t, const uint32_t*,      \
                                                       const GridGeom&, const MinVals<T>&, T, uint64_t*, uint32_t*, \
                                                       uint32_t*, cudaStream_t);                           \
    template cudaError_t launch_cell_keys<T, uint32_t>(const T*, uint64_t, uint32_t, const uint32_t*,      \
                                                       const GridGeom&, const MinVals<T>&, T, uint32_t*, uint32_t*, \
                                                       uint32_t*, cudaStream_t);                           \
    template cudaError_t launch_row_plan<T>(const JoinArgs<T>&, bool, uint2*, cudaStream_t);               \
    template cudaError_t launch_gather_points<T>(const T*, uint64_t, uint32_t, uint32_t, const uint32_t*,  \
                                                 const uint32_t*, T*, cudaStream_t);
GSJ_INST_INDEX(float)
GSJ_INST_INDEX(double)

}  // namespace gsj
