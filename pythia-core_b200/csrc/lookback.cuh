// Decoupled look-back (Merrill and Garland, "Single-pass Parallel Prefix Scan
// with Decoupled Look-back", 2016): tiles of one kernel learn what precedes
// them from their predecessors' status words.  A tile's word is a single
// 64-bit store that carries a flag and a value, so relaxed accesses suffice.
// Tiles are numbered by a ticket that running CTAs draw: a tile waits only for
// tiles whose CTAs are already running and never wait for it, so every wait
// ends; the waits are bounded all the same and report an error.
#pragma once
#include <stdint.h>

#include "bulk.cuh"

namespace pyg {

constexpr unsigned long long kLookBackWaitNs = 2000000000ULL;  // 2 s

__device__ __forceinline__ unsigned long long lb_load(const unsigned long long* p)
{
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}

__device__ __forceinline__ void lb_store(unsigned long long* p, unsigned long long v)
{
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

// One value per tile (status words zeroed before the kernel: value << 2 |
// flag, flag 1 the tile's own value, 2 the sum up to and with it).  Called by
// one whole warp: publishes `own` and returns the sum of the tiles before
// `tile` in `before`; false when a wait gave up (*err is set).
__device__ __forceinline__ bool lb_prefix(unsigned long long* status, int64_t tile, unsigned long long own,
                                          unsigned* err, unsigned long long& before)
{
    const int lane = threadIdx.x & 31;
    before = 0;
    if (lane == 0) lb_store(status + tile, own << 2 | (tile == 0 ? 2 : 1));
    if (tile == 0) return true;
    unsigned long long sum = 0, t0 = 0;
    for (int64_t j = tile - 1;;) {
        const unsigned long long v = j - lane >= 0 ? lb_load(status + (j - lane)) : 2ULL;
        const unsigned ready = __ballot_sync(0xffffffffu, (v & 3) != 0);
        const unsigned incl = __ballot_sync(0xffffffffu, (v & 3) == 2);
        // Lanes up to the nearest inclusive word (all of them if none).
        const unsigned need = incl ? (incl & (0u - incl)) | ((incl & (0u - incl)) - 1u) : 0xffffffffu;
        if ((ready & need) == need) {
            unsigned long long x = (need >> lane) & 1 ? v >> 2 : 0;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
            sum += x;
            if (incl) break;
            j -= 32;
            t0 = 0;
            continue;
        }
        const unsigned long long now = bulk_now_ns();
        bool stop = false;
        if (t0 == 0) t0 = now;
        else stop = now - t0 > kLookBackWaitNs || *(volatile unsigned*)err;
        if (__any_sync(0xffffffffu, stop)) {
            if (lane == 0) atomicOr(err, 1u);
            return false;
        }
    }
    before = sum;
    if (lane == 0) lb_store(status + tile, (sum + own) << 2 | 2);
    return true;
}

}  // namespace pyg
