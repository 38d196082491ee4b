// Device-wide primitives shared across libpyg sources (host-callable).
#pragma once

#include "pyg_internal.cuh"

namespace pyg {

// Exclusive prefix sum of n 64-bit counts (in and out may alias).
// Writes the total to *total_dev if not null.
int exclusive_scan_u64(pyg_ctx* ctx, const unsigned long long* in, unsigned long long* out, int64_t n,
                       unsigned long long* total_dev);

// Stable LSD radix sorts (sort.cu) of 16-byte elements by 64-bit word
// `field` (0 or 1), and of bare 64-bit keys.  Each reads the key range back
// (one stream synchronisation) beyond 4096 elements.  After the caller's
// next synchronisation of the stream, sort_status reports a pass whose
// bounded device-side wait gave up; the result is then undefined, and a
// kernel that takes row numbers from it must look at the error word first.
//
// Into out (may not alias in).
int radix_sort16_to(pyg_ctx* ctx, const ulonglong2* in, ulonglong2* out, int64_t n, int field, bool is_signed);
// Two relations of (signed key, value) elements by the key, with one
// synchronisation for both key ranges.
int radix_sort16_two(pyg_ctx* ctx, const ulonglong2* const in[2], ulonglong2* const out[2], const int64_t n[2]);
int radix_sort8_to(pyg_ctx* ctx, const uint64_t* in, uint64_t* out, int64_t n, bool is_signed);
// Unsigned order, both buffers overwritten; *result is the one holding the
// sorted elements.
int radix_sort16_swap(pyg_ctx* ctx, ulonglong2* a, ulonglong2* b, int64_t n, int field, ulonglong2** result);
int sort_status(pyg_ctx* ctx);
// The counter word that such a wait sets (zero since the context was made)
// and its pinned copy, which sort_status reads and clears.
constexpr int SORT_ERR_WORD = 36;
constexpr int SORT_ERR_PINNED = 1000;

// Order-preserving map of a signed 64-bit value to an unsigned one.
__host__ __device__ __forceinline__ uint64_t to_sortable(int64_t v)
{
    return (uint64_t)v ^ 0x8000000000000000ULL;
}
__host__ __device__ __forceinline__ int64_t from_sortable(uint64_t u)
{
    return (int64_t)(u ^ 0x8000000000000000ULL);
}

// Sortable form of a packed key word (KeySpec): signed order of the single
// column, or lexicographic signed order of an (int32, int32) pair.
__host__ __device__ __forceinline__ uint64_t packed_to_sortable(uint64_t k, int nkeys)
{
    return nkeys == 2 ? (k ^ 0x8000000080000000ULL) : (k ^ 0x8000000000000000ULL);
}

// Distinct-key estimate for n tuples (device, tb bytes each) from the
// packed keys of a sample of CDF_ESTIMATE_SAMPLE tuples: the GEE
// estimate carried by the learned CDF model trained on that sample
// (cdf.cu).  Sizes hash tables when a caller gives no group estimate.
constexpr int64_t CDF_ESTIMATE_SAMPLE = (int64_t)1 << 18;
// Largest key sample the MPSM join draws for its learned splitters.
constexpr int64_t CDF_MPSM_SAMPLE = (int64_t)1 << 21;
int estimate_distinct_keys(pyg_ctx* ctx, const uint8_t* base, int64_t n, int32_t tb, const KeySpec& ks,
                           int64_t* out);

// Gather rows: out[i] = in[items[i].y] for tuples of tb bytes.  Nothing is
// read when the sort of the items gave up.
int gather_rows(pyg_ctx* ctx, const uint8_t* in, const ulonglong2* items, int64_t n, int32_t tb, uint8_t* out);

}  // namespace pyg
