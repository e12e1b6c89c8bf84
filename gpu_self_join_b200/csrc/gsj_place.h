// Pair keys -> neighbour table without a global sort, and per-list sorting
// (gsj_place.cu).
#pragma once
#include <cstddef>
#include <cstdint>
#include <cuda_runtime.h>

namespace gsj {

// Temporary bytes of place_pairs, sort_lists and sort_very_long_lists for nlists lists.
size_t place_temp_bytes(uint64_t nlists);

// Lists of the packed keys (query id << shift | neighbour id; entries equal
// to ~0 are skipped): counts[q] (nlists + 1 entries), offsets (exclusive
// prefix, nlists + 1 entries), and each neighbour id at a free place of its
// query's list in table (capacity cap).  cursor: nlists scratch counters.
// *err (device, zeroed by the caller) is set when a key falls outside its
// list.  The order within a list is arbitrary until the lists are sorted.
cudaError_t place_pairs(const unsigned long long* keys, uint64_t nkeys, uint32_t shift, uint32_t nlists,
                        uint32_t* counts, uint64_t* offsets, uint32_t* table, uint64_t cap, uint32_t* cursor,
                        uint32_t* err, void* temp, int num_sms, int* launches, cudaStream_t st);

// Sorts every list of up to 4096 entries ascending (a warp per list up to 512
// entries, a CTA above) and gathers the indices of the lists above 512 into
// temp.  List l is table[offsets[l] .. offsets[l+1]).  d_nlong: two device
// words, zeroed by the caller, which receive the number of lists above 512 and
// above 4096 entries.
template <typename OffT>
cudaError_t sort_lists(uint32_t* table, const OffT* offsets, uint32_t nlists, void* temp, uint32_t* d_nlong,
                       int num_sms, int* launches, cudaStream_t st);
// Sorts the gathered lists above 4096 entries (ids below 2^id_bits): LSD radix
// passes using the same ranges of `scratch` (as large as the table) as a second
// buffer.
template <typename OffT>
cudaError_t sort_very_long_lists(uint32_t* table, uint32_t* scratch, const OffT* offsets, const void* temp,
                                 uint32_t nlong, uint32_t nvery, uint32_t id_bits, int num_sms, int* launches,
                                 cudaStream_t st);

}  // namespace gsj
