// Shared definitions of the B200 epsilon-grid self-join kernels.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace gsj {

constexpr int kMaxK = 10;        // indexed dimensions supported (3^10 neighbour offsets)
constexpr int kMaxIlp = 64;      // ILP register blocks supported
constexpr int kQChunk = 32;      // queries per work item (one per lane)
constexpr uint64_t kEmptyKey = ~0ull;        // hash table empty slot

// Arithmetic order of the squared-distance sum, i.e. the reference's
// ILP/SHORTCIRCUIT switches (kernel.cu:307-377):
//   kSeq    ILP==0                  s = fma(d, d, s) over l = 0..n-1
//   kIlp    ILP>0,  SHORTCIRCUIT=0  r_j = fma(d, d, r_j) for l = j (mod ILP); s = r_0 + r_1 + ...
//   kIlpSc  ILP>0,  SHORTCIRCUIT=1  per ILP block: s = fma(d_l, d_l, s); s += d_{l+j}^2 (j >= 1)
enum Model : int { kSeq = 0, kIlp = 1, kIlpSc = 2 };

// Grid geometry (k <= kMaxK indexed dims).
struct GridGeom {
    uint32_t k;
    uint32_t ncells[kMaxK];
    uint64_t mult[kMaxK];  // linear id stride of dim j (dim 0 fastest, main.cu:867-883)
};

template <typename T>
struct JoinArgs {
    const T* pts;                 // [N][npad] points in cell order, columns reordered
    const uint32_t* ids;          // [N] slot -> original point id
    const uint32_t* cell_start;   // [M+1]
    const uint64_t* cell_key;     // [M]
    const uint32_t* ds;           // [totalCells+1] slot prefix over all linear ids (dense grids), or null
    const uint2* plan;            // [M][3^(k-1)] (slot start, count) of each neighbour row, or null: the ROWS
                                  // path's (whole rows), the warp join's on hashed grids of k <= 3 (rows as
                                  // its traversal takes them)
    const uint4* htab;            // [hcap] hash table of the grid rows that hold a cell {linear id of the row's
                                  // cell 0 (lo, hi; kEmptyKey = empty), first cell, cells}, or null
    uint64_t hmask;               // hcap - 1
    const uint2* items;           // [num_items] (cell, chunk)
    const uint4* nbtab;           // [3^k] neighbour offsets: linear-id delta (x lo, y hi), z = moved-down dims
                                  // | moved-up dims << 16, w = highest moved dim (0xff: none)
    uint32_t num_items;
    uint32_t* work_counter;       // dynamic work distribution
    uint32_t n, npad, ilp;
    uint32_t n_points;            // N
    uint32_t num_cells;           // non-empty cells
    GridGeom g;
    T thr;                        // s <= thr  <=>  sqrt(s) <= eps
    T eps;                        // epsilon in T (cell formula)
    T minv[kMaxK];                // minArr (grid origin per indexed dim)
    unsigned long long* cand_cnt; // candidate evaluations
    // fill pass (ROWS path)
    const uint64_t* offsets;      // [N+1] by original id
    uint32_t* table;              // [R]
    unsigned long long table_cap; // R: writes at or beyond it are dropped and flagged
    uint32_t* err_flag;           // set to 1 when a write would leave the table
    // launch shape of this join (0 = the launcher's default), from the tuning table
    uint32_t shape_threads;       // ROWS count / fill CTA size (64..256, a multiple of 32)
    uint32_t shape_warps;         // WARP join: warps per CTA (1..8)
    uint32_t shape_per_sm;        // WARP, TILE, SCREEN joins: CTAs per SM at most
};

__host__ __device__ inline uint64_t mix64(uint64_t x) {
    // splitmix64 finaliser: hash of a linear cell id
    x ^= x >> 30;
    x *= 0xbf58476d1ce4e5b9ull;
    x ^= x >> 27;
    x *= 0x94d049bb133111ebull;
    x ^= x >> 31;
    return x;
}

// Neighbour offset `o` of a cell: usable when it stays inside the grid (no
// moved-down dim at the cell's low edge, no moved-up dim at its high edge) and,
// with unicomp, when the highest moved dim has an odd own coordinate
// (stamploops.h: `nDCellIDs[d] & 1`; the cell itself is always visited).
// Returns the neighbour's linear id in `lin`.
template <typename T, bool STAMP>
__device__ __forceinline__ bool nb_offset(const JoinArgs<T>& a, uint32_t o, uint64_t own_lin, uint32_t lowmask,
                                          uint32_t highmask, uint32_t oddmask, uint64_t& lin) {
    const uint4 e = a.nbtab[o];
    if ((e.z & 0xffffu) & lowmask) return false;
    if ((e.z >> 16) & highmask) return false;
    if (STAMP && e.w != 0xffu && !((oddmask >> e.w) & 1u)) return false;
    lin = own_lin + (((uint64_t)e.y << 32) | e.x);
    return true;
}

// Edge and parity masks of a cell's coordinates for nb_offset.
__device__ __forceinline__ void cell_masks(const uint32_t (&own)[kMaxK], const GridGeom& g, uint32_t& lowmask,
                                           uint32_t& highmask, uint32_t& oddmask) {
    lowmask = highmask = oddmask = 0u;
#pragma unroll
    for (int j = 0; j < kMaxK; j++)
        if (j < (int)g.k) {
            lowmask |= (own[j] == 0u ? 1u : 0u) << j;
            highmask |= (own[j] + 1u >= g.ncells[j] ? 1u : 0u) << j;
            oddmask |= (own[j] & 1u) << j;
        }
}

__device__ __forceinline__ uint64_t entry_key(const uint4& e) { return ((uint64_t)e.y << 32) | e.x; }

// Cells of the grid row whose cell 0 has linear id `base`: indices [first,
// first + n) of the sorted cell list (n = 0: none).  e: the table entry at the
// row's own position.
template <typename T>
__device__ __forceinline__ void row_entry(const JoinArgs<T>& a, uint64_t base, uint4 e, uint32_t& first, uint32_t& n) {
    for (uint64_t p = 1; entry_key(e) != base; p++) {
        if (entry_key(e) == kEmptyKey || p > a.hmask) {
            n = 0u;
            return;
        }
        e = a.htab[(mix64(base) + p) & a.hmask];
    }
    first = e.z;
    n = e.w;
}

// Slot range [start, start + cnt) of the cells xlo..xhi (at most three) of the
// grid row whose cell 0 has linear id `base`.  These cells are consecutive in
// cell order (dim 0 is fastest), so the range is contiguous whichever of them
// are non-empty.
//
// row_probe issues the first loads of a row, so that a thread can have the next
// row's in flight: on dense grids the slot-prefix table's entries, which are all
// it takes, else the row's table entry.  row_slots finishes: a hashed row needs
// one more step, its cells' ids and slots together (rows of more than four
// cells are bisected first).
struct RowProbe {
    bool ok;
    uint64_t base;
    uint32_t xlo, xhi;
    uint4 e;  // the row's entry, or (dense) first slot of cell xlo and of cell xhi + 1
};

template <typename T>
__device__ __forceinline__ void row_probe(const JoinArgs<T>& a, bool ok, uint64_t base, uint32_t xlo, uint32_t xhi,
                                          RowProbe& p) {
    p.ok = ok;
    p.base = base;
    p.xlo = xlo;
    p.xhi = xhi;
    if (!ok) return;
    if (a.ds) {
        p.e.x = a.ds[base + xlo];
        p.e.y = a.ds[base + xhi + 1u];
    } else {
        p.e = a.htab[mix64(base) & a.hmask];
    }
}

template <typename T>
__device__ __forceinline__ void row_slots(const JoinArgs<T>& a, const RowProbe& p, uint32_t& start, uint32_t& cnt) {
    start = cnt = 0u;
    if (!p.ok) return;
    if (a.ds) {
        start = p.e.x;
        cnt = p.e.y - start;
        return;
    }
    const uint64_t klo = p.base + p.xlo, khi = p.base + p.xhi;
    uint32_t first = 0, n = 0;
    row_entry(a, p.base, p.e, first, n);
    if (n > 4u) {
        // the row's first cell at or past xlo; at most three cells follow up to xhi
        uint32_t l = first, h = first + n;
        while (l < h) {
            const uint32_t m = l + (h - l) / 2u;
            if (a.cell_key[m] < klo) l = m + 1u;
            else h = m;
        }
        n -= l - first;
        first = l;
    }
    if (n == 0u) return;
    uint64_t key[4];
    uint32_t slot[5];
#pragma unroll
    for (uint32_t i = 0; i < 4u; i++) key[i] = i < n ? a.cell_key[first + i] : kEmptyKey;
#pragma unroll
    for (uint32_t i = 0; i < 5u; i++) slot[i] = a.cell_start[first + min(i, n)];
    uint32_t end = 0;
    start = 0xffffffffu;
#pragma unroll
    for (uint32_t i = 0; i < 4u; i++)
        if (key[i] >= klo && key[i] <= khi) {
            start = min(start, slot[i]);
            end = slot[i + 1u];
        }
    if (end) cnt = end - start;
}

// Slot range of the cell with linear id `lin`.
template <typename T>
__device__ __forceinline__ bool lookup_range(const JoinArgs<T>& a, uint64_t lin, uint32_t& start, uint32_t& cnt) {
    const uint32_t x = a.ds ? 0u : (uint32_t)(lin % a.g.ncells[0]);
    RowProbe p;
    row_probe(a, true, lin - x, x, x, p);
    row_slots(a, p, start, cnt);
    return cnt != 0u;
}

// A neighbour row of the cell with linear id own_lin and dim-0 coordinate x: the
// cells x-1..x+1 of the grid row that offset r (digit j of r is dim j+1's step +
// 1) leads to.  With unicomp the own row (r's centre) adds its dim-0 neighbours
// only when x is odd, every other row comes whole or not at all (the highest
// moved dim is the same for its three cells).
template <typename T, bool STAMP>
__device__ __forceinline__ void neighbour_row(const JoinArgs<T>& a, bool valid, uint32_t r, uint64_t own_lin,
                                              uint32_t x, uint32_t lowmask, uint32_t highmask, uint32_t oddmask,
                                              RowProbe& p) {
    uint64_t lin = 0;
    const bool ok = valid && nb_offset<T, STAMP>(a, 3u * r + 1u, own_lin, lowmask, highmask, oddmask, lin);
    const bool side = !STAMP || lin != own_lin || (oddmask & 1u);
    row_probe(a, ok, lin - x, x - (side && !(lowmask & 1u) ? 1u : 0u), x + (side && !(highmask & 1u) ? 1u : 0u), p);
}

template <typename T, bool STAMP>
__device__ __forceinline__ bool row_range(const JoinArgs<T>& a, bool valid, uint32_t r, uint64_t own_lin, uint32_t x,
                                          uint32_t lowmask, uint32_t highmask, uint32_t oddmask, uint32_t& start,
                                          uint32_t& cnt) {
    RowProbe p;
    neighbour_row<T, STAMP>(a, valid, r, own_lin, x, lowmask, highmask, oddmask, p);
    row_slots(a, p, start, cnt);
    return cnt != 0u;
}

}  // namespace gsj
