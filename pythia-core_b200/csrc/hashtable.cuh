// The device hash table shared by the hash join entry points.
#pragma once

#include "pyg_internal.cuh"
#include "radixpart.cuh"

// Open-addressing table of cap slots, W 64-bit words per slot: word 0 is
// the packed key (kEmptyKey marks a free slot), words 1..W-1 hold the
// stored build columns (MATERIALIZE: one slot per build tuple) or their
// wrapped per-key sums (AGGREGATE: one slot per distinct key).  Build
// tuples whose key word equals kEmptyKey live in a small side list.
struct pyg_hashtable {
    int32_t mode;
    int32_t nkeys;
    pyg::KeySpec ks;
    int32_t npay;
    int32_t pay_cols[PYG_MAX_COLS];
    int32_t pay_types[PYG_MAX_COLS];
    int32_t W;
    uint64_t cap;
    uint64_t* slots = nullptr;
    uint64_t* side = nullptr;
    int64_t nside = 0;
    unsigned long long* counts = nullptr;  // AGGREGATE with duplicate keys
    int32_t has_dups = 0;
    int64_t entries = 0;
};

namespace pyg {

// Home slot of packed key k in a table of cap slots: the radix operators'
// hash (rj_hash), whose top bits spread a dense key range evenly, scaled by a
// 32-bit multiply-high where 32 hash bits resolve the slots finely enough.
// A random hash at half load gives a warp of 32 x 4 lookups a longest chain of
// about ten dependent reads; consecutive keys here hardly meet: build of 1 M
// keys 67 -> 19 us, materialising probe of 8 M 163 -> 88 us (against mix64).
// Random keys keep their chains: build, probe and sort of the joined rows take
// 487 us with keys 1..n, 625 us with random 31- or 64-bit keys.
__device__ __forceinline__ uint64_t ht_slot(uint64_t k, uint64_t cap)
{
    const uint64_t h = rj_hash(k);
    return cap <= ((uint64_t)1 << 28) ? (uint64_t)__umulhi((unsigned)(h >> 32), (unsigned)cap) : reduce_range(h, cap);
}

}  // namespace pyg
