// Group-by (sum and/or count) of 16-byte device tuples, aggregated in shared
// memory: (int64 key, int64 value), or (int32, int32, int64) with the pair as
// the key.
//
// Same result table as the generic group-by kernel (groupby.cu): 32-byte
// slots {key, sum, count, -} in HBM plus the flags {full, groups, sum and
// count of the INT64_MIN key}; compaction and ordering by key are shared.
// What differs is how the table is filled:
//
//   very few     (expected <= GBR_TINY_GROUPS) every warp folds into its own
//                128-slot table.
//   few groups   (expected <= GBR_DIRECT_GROUPS) every CTA folds its slice
//                of the input into a 160 KB shared-memory table and flushes
//                it once: one HBM read of the input, G atomics per CTA.
//   many groups  the input is hash-partitioned (radixpart.cu), to 8-byte
//                words where the key and value ranges allow, into partitions
//                of at most about GBR_PART_GROUPS distinct keys; a persistent
//                CTA folds each partition into its shared table and flushes
//                it.  Traffic: the partition passes plus one read.
//
// A key that does not fit a full shared table goes straight to the HBM
// table, so the result never depends on the group estimate being right.
//
// Sums are kept as two 32-bit halves: a 64-bit atomic add in shared memory
// is a compare-and-swap loop (20-40 clocks per warp and SM, measured, against
// 2.6-4 for a 32-bit one); the low half's old value tells the carry, and the
// high half is touched only when there is something to add.  Each warp also
// keeps the sum and count of one frequent key of its work item in its lanes'
// registers, so that skewed keys do not meet on one shared slot.
//
// Measured (sum and count per group, sorted; before: 64-bit shared atomics,
// leader rounds of shuffles for repeated keys, 16-byte partitions from an
// exact histogram): 2^28 tuples, G = 16: 1284 -> 848 us (5.3 TB/s in the
// fold); 2^27 Zipf(1.0) ids, G = 2^16: 5074 -> 1340 us; 40 M (int32, int32)
// keys, G = 2^16, which took the generic kernel: 3441 -> 694 us.
#include <cuda_runtime.h>
#include <stdint.h>
#include <string.h>

#include <algorithm>
#include <type_traits>
#include <vector>

#include "gbradix.cuh"
#include "lookback.cuh"
#include "radixpart.cuh"

namespace pyg {

constexpr int GBR_THREADS = 1024;               // few-groups kernels: one CTA per SM
constexpr unsigned GBR_SLOTS = 8192;            // their shared table: 20 bytes per slot
constexpr int GBR_SMEM = GBR_SLOTS * 20;        // 160 KB
constexpr int GBR_TINY_SLOTS = 128;             // very few groups: slots per warp
constexpr int64_t GBR_TINY_GROUPS = 64;
constexpr int64_t GBR_DIRECT_GROUPS = 3072;     // fold without partitioning up to this many groups
constexpr int GBR_PT_THREADS = 512;             // partitioned: two CTAs per SM, one folds while the other flushes
constexpr unsigned GBR_PT_SLOTS = 5120;         // their tables (16 or 20 bytes per slot: at most 100 KB)
constexpr int64_t GBR_PART_GROUPS = 2048;       // distinct keys per partition when partitioned
// At least 2^7 partitions of a large input, so that most are one work item
// and flushed once.  2^27 Zipf(1.0) ids, G = 2^16, partition pass + fold:
// 603 + 545 us with 2^6, 623 + 496 with 2^7, 822 + 465 with 2^8.
constexpr int GBR_PART_BITS = 7;
constexpr unsigned GBR_PROBES = 128;            // shared table probes, then the HBM table
constexpr uint64_t GBR_PROBE_LIMIT = 4096;      // HBM table probe limit (then "full")
constexpr int64_t GBR_CHUNK = (int64_t)1 << 22; // tuples per work item (at most)

struct GbrArgs {
    const void* in;              // direct modes: the input; partitioned: the partitions
    int64_t n;                   // direct modes: tuples
    const unsigned long long* item_start;  // partitioned: first tuple of each item
    const unsigned* item_len;              // partitioned: tuples of each item
    long long nitems;
    unsigned* next;              // work queue head (partitioned)
    int fine_bits;               // slot bits below the partition bits (0 in direct modes)
    int want_sum;
    unsigned long long kbase, pbase;  // frame of packed words
    ulonglong4* table;           // HBM result table
    uint64_t cap;
    unsigned long long* flags;   // [0] full, [1] groups, [2] INT64_MIN sum, [3] INT64_MIN count
};

// What a thread carries to the end of its kernel.
struct GbrTail {
    uint64_t sent_sum = 0, sent_cnt = 0;  // the INT64_MIN key's
    unsigned long long fresh = 0;         // new groups in the HBM table
    bool full = false;
};

// Adds (sum, cnt) for key k to the HBM table.  Once the table is full the
// result is discarded and the host redoes the call with a larger one, so
// nothing more is looked up: without this, 2^25 tuples of 2^23 random keys
// (no estimate given) spent 245 ms walking full tables.
__device__ __forceinline__ void gbr_global_add(const GbrArgs& a, uint64_t k, uint64_t sum, uint64_t cnt, GbrTail& z)
{
    if (k == kEmptyKey) {
        z.sent_sum += sum;
        z.sent_cnt += cnt;
        return;
    }
    if (z.full) return;
    uint64_t s = reduce_range(mix64(k), a.cap);
    for (uint64_t steps = 0; steps < GBR_PROBE_LIMIT && steps < a.cap; ++steps) {
        if ((steps & 63) == 63 && lb_load(a.flags)) break;
        unsigned long long* slot = (unsigned long long*)&a.table[s];
        unsigned long long prev = slot[0];
        if (prev == kEmptyKey) {
            prev = atomicCAS(slot, kEmptyKey, k);
            if (prev == kEmptyKey) ++z.fresh;
        }
        if (prev == kEmptyKey || prev == k) {
            if (a.want_sum) atomicAdd(slot + 1, (unsigned long long)sum);
            atomicAdd(slot + 2, (unsigned long long)cnt);
            return;
        }
        s = (s + 1 == a.cap) ? 0 : s + 1;
    }
    z.full = true;
    // One store per group of lanes that end together: one per thread, all to
    // this address, took a millisecond (2^25 tuples, 1000 groups, 250
    // expected: 1434 us, now 824; walking full tables to the end 738).
    if ((threadIdx.x & 31) == (unsigned)__ffs(__activemask()) - 1 && !lb_load(a.flags)) lb_store(a.flags, 1);
}

// How the kernels read a tuple: 16-byte (key, value); the same with the two
// int32 key columns, whose key word has the first column on top; packed
// words of a partition, whose 32-bit key offsets are the table's keys.
enum GbrFormat { GBR_PAIR = 0, GBR_PAIR32 = 1, GBR_PACKED = 2 };

template <int FMT>
struct GbrFmt {
    using In = typename std::conditional<FMT == GBR_PACKED, unsigned long long, longlong2>::type;
    using Key = typename std::conditional<FMT == GBR_PACKED, unsigned, unsigned long long>::type;
    static constexpr Key EMPTY = FMT == GBR_PACKED ? (Key)0xFFFFFFFFu : (Key)kEmptyKey;
    static __device__ __forceinline__ Key key(const In& e)
    {
        if constexpr (FMT == GBR_PACKED) return (unsigned)e;
        else if constexpr (FMT == GBR_PAIR32) return ((unsigned long long)e.x << 32) | ((unsigned long long)e.x >> 32);
        else return (unsigned long long)e.x;
    }
    static __device__ __forceinline__ uint64_t val(const In& e)
    {
        if constexpr (FMT == GBR_PACKED) return e >> 32;
        else return (uint64_t)e.y;
    }
    // Table slot of a key among `slots`.  Packed: the MurmurHash3 32-bit
    // finaliser of the offset, independent of the partition bits.
    static __device__ __forceinline__ unsigned slot(Key k, int fb, unsigned slots)
    {
        if constexpr (FMT == GBR_PACKED) {
            unsigned h = k;
            h ^= h >> 16;
            h *= 0x85ebca6bu;
            h ^= h >> 13;
            h *= 0xc2b2ae35u;
            h ^= h >> 16;
            return __umulhi(h, slots);
        } else if constexpr (FMT == GBR_PAIR32) {
            // The partition bits are those of the word as stored.
            return rj_slot((k << 32) | (k >> 32), fb, slots);
        } else {
            return rj_slot(k, fb, slots);
        }
    }
    // A table entry as (key, sum) of the HBM table.
    static __device__ __forceinline__ uint64_t full_key(const GbrArgs& a, Key k)
    {
        if constexpr (FMT == GBR_PACKED) return a.kbase + k;
        else return k;
    }
    static __device__ __forceinline__ uint64_t full_sum(const GbrArgs& a, uint64_t sum, uint64_t cnt)
    {
        if constexpr (FMT == GBR_PACKED) return sum + cnt * a.pbase;
        else return sum;
    }
};

template <int FMT, unsigned SLOTS>
struct GbrTable {
    using Key = typename GbrFmt<FMT>::Key;
    Key* key;
    unsigned *lo, *hi, *cnt;  // sum halves, count
    static constexpr size_t BYTES = (size_t)SLOTS * (sizeof(Key) + 12);
    __device__ explicit GbrTable(unsigned char* p)
        : key(reinterpret_cast<Key*>(p)), lo(reinterpret_cast<unsigned*>(p + (size_t)SLOTS * sizeof(Key))),
          hi(lo + SLOTS), cnt(hi + SLOTS)
    {
    }
    __device__ __forceinline__ void clear(unsigned first, unsigned step)
    {
        for (unsigned s = first; s < SLOTS; s += step) {
            key[s] = GbrFmt<FMT>::EMPTY;
            lo[s] = 0;
            hi[s] = 0;
            cnt[s] = 0;
        }
    }
    // Adds (sum, c) for key k; false if no slot was found.
    __device__ __forceinline__ bool add(Key k, uint64_t sum, unsigned c, int want_sum, int fb)
    {
        unsigned pos = GbrFmt<FMT>::slot(k, fb, SLOTS);
        for (unsigned steps = 0; steps < (SLOTS < GBR_PROBES ? SLOTS : GBR_PROBES); ++steps) {
            Key prev = key[pos];
            if (prev == GbrFmt<FMT>::EMPTY) prev = atomicCAS(&key[pos], GbrFmt<FMT>::EMPTY, k);
            if (prev == GbrFmt<FMT>::EMPTY || prev == k) {
                atomicAdd(&cnt[pos], c);
                if (want_sum) {
                    const unsigned l = (unsigned)sum;
                    const unsigned old = atomicAdd(&lo[pos], l);
                    const unsigned h = (unsigned)(sum >> 32) + (old + l < old ? 1u : 0u);
                    if (h) atomicAdd(&hi[pos], h);
                }
                return true;
            }
            pos = pos + 1 == SLOTS ? 0 : pos + 1;
        }
        return false;
    }
    __device__ __forceinline__ void flush(const GbrArgs& a, unsigned first, unsigned step, GbrTail& z)
    {
        for (unsigned s = first; s < SLOTS; s += step) {
            const Key k = key[s];
            if (k == GbrFmt<FMT>::EMPTY) continue;
            const uint64_t c = cnt[s];
            gbr_global_add(a, GbrFmt<FMT>::full_key(a, k),
                           GbrFmt<FMT>::full_sum(a, ((uint64_t)hi[s] << 32) | lo[s], c), c, z);
        }
    }
};

// Folds tuples [0, n) of p into table t; the calling threads are `threads`
// whole warps, thread `at` of them this one.
template <int FMT, unsigned SLOTS>
__device__ void gbr_fold_range(const GbrArgs& a, GbrTable<FMT, SLOTS>& t, const typename GbrFmt<FMT>::In* __restrict__ p,
                               int64_t n, int64_t at, int64_t threads, GbrTail& z)
{
    using F = GbrFmt<FMT>;
    using Key = typename F::Key;
    constexpr int U = FMT == GBR_PACKED ? 8 : 4;
    const int lane = threadIdx.x & 31;
    // The warp's frequent key: the commonest of its first 32 tuples, if any
    // repeats.  Every lane adds its own tuples of that key in registers.
    Key hot = F::EMPTY;
    uint64_t hot_s = 0;
    unsigned hot_c = 0;
    const int64_t w0 = at - lane;
    if (w0 + 31 < n) {
        const Key k = F::key(p[w0 + lane]);
        const unsigned c = __popc(__match_any_sync(0xffffffffu, k));
        const unsigned top = __reduce_max_sync(0xffffffffu, (c << 5) | (unsigned)lane);
        hot = __shfl_sync(0xffffffffu, k, (int)(top & 31));
        if (top >> 5 < 3) hot = F::EMPTY;
    }
    auto one = [&](const typename F::In& e) {
        const Key k = F::key(e);
        const uint64_t v = F::val(e);
        if (k == hot) {  // the empty marker too, when no key is frequent
            hot_s += v;
            ++hot_c;
        } else if (FMT != GBR_PACKED && k == F::EMPTY) {
            z.sent_sum += v;
            z.sent_cnt += 1;
        } else if (!t.add(k, v, 1u, a.want_sum, a.fine_bits)) {
            gbr_global_add(a, F::full_key(a, k), F::full_sum(a, v, 1), 1, z);
        }
    };
    int64_t i = at;
    for (; i + (int64_t)(U - 1) * threads < n; i += (int64_t)U * threads) {
        typename F::In x[U];
#pragma unroll
        for (int u = 0; u < U; ++u) x[u] = __ldcs(&p[i + (int64_t)u * threads]);
#pragma unroll
        for (int u = 0; u < U; ++u) one(x[u]);
    }
    for (; i < n; i += threads) one(__ldcs(&p[i]));
    // The frequent key's lanes are added up and folded once per warp.
    hot_s = warp_sum_u64(hot_s);
    hot_c = __reduce_add_sync(0xffffffffu, hot_c);
    if (lane == 0 && hot_c) {
        if (FMT != GBR_PACKED && hot == F::EMPTY) {
            z.sent_sum += hot_s;
            z.sent_cnt += hot_c;
        } else if (!t.add(hot, hot_s, hot_c, a.want_sum, a.fine_bits)) {
            gbr_global_add(a, F::full_key(a, hot), F::full_sum(a, hot_s, hot_c), hot_c, z);
        }
    }
}

__device__ void gbr_finish(const GbrArgs& a, const GbrTail& z)
{
    const uint64_t sent_sum = warp_sum_u64(z.sent_sum), sent_cnt = warp_sum_u64(z.sent_cnt);
    const unsigned long long fresh = warp_sum_u64(z.fresh);
    const bool anyfull = __any_sync(0xffffffffu, z.full);
    if ((threadIdx.x & 31) == 0) {
        if (sent_cnt) {
            atomicAdd(&a.flags[2], (unsigned long long)sent_sum);
            atomicAdd(&a.flags[3], (unsigned long long)sent_cnt);
        }
        if (fresh) atomicAdd(&a.flags[1], fresh);
        if (anyfull) a.flags[0] = 1;
    }
}

// Few groups: CTA b folds the b-th slice of the input, then flushes once.
template <int FMT>
__global__ void __launch_bounds__(GBR_THREADS, 1) gbr_direct_kernel(GbrArgs a)
{
    extern __shared__ __align__(16) unsigned char gbr_smem[];
    GbrTable<FMT, GBR_SLOTS> t(gbr_smem);
    t.clear(threadIdx.x, GBR_THREADS);
    __syncthreads();
    GbrTail z;
    const int64_t per = (a.n + gridDim.x - 1) / gridDim.x;
    const int64_t b0 = (int64_t)blockIdx.x * per, b1 = min(a.n, b0 + per);
    if (b0 < b1)
        gbr_fold_range<FMT, GBR_SLOTS>(a, t, reinterpret_cast<const longlong2*>(a.in) + b0, b1 - b0, threadIdx.x,
                                       GBR_THREADS, z);
    __syncthreads();
    t.flush(a, threadIdx.x, GBR_THREADS, z);
    gbr_finish(a, z);
}

// Very few groups: every warp folds into its own 128-slot table, so the
// shared atomics of different warps never meet on one address.
template <int FMT>
__global__ void __launch_bounds__(GBR_THREADS, 1) gbr_tiny_kernel(GbrArgs a)
{
    extern __shared__ __align__(16) unsigned char gbr_smem[];
    using Table = GbrTable<FMT, GBR_TINY_SLOTS>;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    Table t(gbr_smem + (size_t)w * Table::BYTES);
    t.clear(lane, 32);
    __syncwarp();
    GbrTail z;
    const int64_t per = (a.n + gridDim.x - 1) / gridDim.x;
    const int64_t b0 = (int64_t)blockIdx.x * per, b1 = min(a.n, b0 + per);
    if (b0 < b1)
        gbr_fold_range<FMT, GBR_TINY_SLOTS>(a, t, reinterpret_cast<const longlong2*>(a.in) + b0, b1 - b0, threadIdx.x,
                                            GBR_THREADS, z);
    __syncwarp();
    t.flush(a, lane, 32, z);
    gbr_finish(a, z);
}

// Many groups: persistent CTAs claim (partition chunk) items.
template <int FMT>
__global__ void __launch_bounds__(GBR_PT_THREADS, 2) gbr_part_kernel(GbrArgs a)
{
    extern __shared__ __align__(16) unsigned char gbr_smem[];
    GbrTable<FMT, GBR_PT_SLOTS> t(gbr_smem);
    __shared__ long long item;
    GbrTail z;
    for (;;) {
        if (threadIdx.x == 0)
            item = *(volatile unsigned long long*)a.flags ? a.nitems : (long long)atomicAdd(a.next, 1u);
        t.clear(threadIdx.x, GBR_PT_THREADS);
        __syncthreads();
        const long long it = item;
        if (it >= a.nitems) break;
        gbr_fold_range<FMT, GBR_PT_SLOTS>(a, t, reinterpret_cast<const typename GbrFmt<FMT>::In*>(a.in) + a.item_start[it],
                                          (int64_t)a.item_len[it], threadIdx.x, GBR_PT_THREADS, z);
        __syncthreads();
        t.flush(a, threadIdx.x, GBR_PT_THREADS, z);
        __syncthreads();
    }
    gbr_finish(a, z);
}

bool groupby16_eligible(int64_t expected_groups) { return expected_groups > 0; }

namespace {

template <typename Fn>
int launch_fold(pyg_ctx* ctx, Fn* fn, unsigned grid, int threads, size_t smem, const GbrArgs& a)
{
    PYG_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    fn<<<grid, threads, smem, ctx->stream>>>(a);
    PYG_LAUNCHED(ctx);
    return PYG_OK;
}

}  // namespace

int groupby16_fill(pyg_ctx* ctx, const void* in, int64_t n, bool pair32, int want_sum, int64_t expected_groups,
                   ulonglong4* table, uint64_t cap, unsigned long long* flags)
{
    GbrArgs a;
    memset(&a, 0, sizeof(a));
    a.want_sum = want_sum;
    a.table = table;
    a.cap = cap;
    a.flags = flags;
    if (n <= 0) return PYG_OK;
    if (expected_groups <= GBR_DIRECT_GROUPS) {
        a.in = in;
        a.n = n;
        const int64_t want = (n + 64 * GBR_THREADS - 1) / (64 * GBR_THREADS);
        const unsigned grid = (unsigned)std::max<int64_t>(1, std::min<int64_t>(want, ctx->sm_count));
        if (expected_groups <= GBR_TINY_GROUPS) {
            const size_t smem = (GBR_THREADS / 32) * GbrTable<GBR_PAIR, GBR_TINY_SLOTS>::BYTES;
            return pair32 ? launch_fold(ctx, gbr_tiny_kernel<GBR_PAIR32>, grid, GBR_THREADS, smem, a)
                          : launch_fold(ctx, gbr_tiny_kernel<GBR_PAIR>, grid, GBR_THREADS, smem, a);
        }
        return pair32 ? launch_fold(ctx, gbr_direct_kernel<GBR_PAIR32>, grid, GBR_THREADS, GBR_SMEM, a)
                      : launch_fold(ctx, gbr_direct_kernel<GBR_PAIR>, grid, GBR_THREADS, GBR_SMEM, a);
    }
    // Partition so that each partition holds at most about GBR_PART_GROUPS
    // keys, and into at least 2^GBR_PART_BITS partitions, so that most are
    // folded and flushed once, by one CTA (2.9 M tuples, 3817 groups: 330 us
    // in two partitions of 23 chunks each).
    int FB = n >= ((int64_t)1 << 17) ? GBR_PART_BITS : 1;
    while (FB < RJ_MAX_FINE_BITS && (double)expected_groups / (double)(1 << FB) > (double)GBR_PART_GROUPS) ++FB;
    const bool two = FB > RJ_MAX_LOCAL_BITS;
    const int F = 1 << FB;
    RPSide side;
    side.in = (const longlong2*)in;
    side.n = n;
    side.allow_pack = !pair32;
    unsigned* pflags = (unsigned*)(ctx->dcounters + 204);
    unsigned* hflags = (unsigned*)ctx->pinned + 64;
    unsigned long long* dstart = nullptr;
    int rc = rp_partition_sides(ctx, &side, 1, FB, two, pflags, hflags, nullptr);
    if (rc) return rc;
    const RJLayout& L = side.L;
    do {
        // Work items: whole partitions, or chunks of a large one, small
        // enough for about four items per SM.
        const unsigned long long chunk = (unsigned long long)std::max<int64_t>(
            (int64_t)1 << 14, std::min<int64_t>(GBR_CHUNK, n / (4 * (int64_t)ctx->sm_count) + 1));
        std::vector<unsigned long long> istart;
        std::vector<unsigned> ilen;
        for (int f = 0; f < F; ++f)
            for (unsigned long long o = 0; o < L.count[f]; o += chunk) {
                istart.push_back(L.fstart[f] + o);
                ilen.push_back((unsigned)std::min<unsigned long long>(chunk, L.count[f] - o));
            }
        if (istart.empty()) break;
        const size_t ni = istart.size();
        if ((rc = dalloc(ctx, (void**)&dstart, ni * 12 + 16))) break;
        unsigned* dlen = (unsigned*)(dstart + ni);
        if ((rc = stage_h2d(ctx, dstart, istart.data(), ni * 8)) || (rc = stage_h2d(ctx, dlen, ilen.data(), ni * 4))) break;
        unsigned* next = (unsigned*)(ctx->dcounters + 206);
        PYG_CUDA(cudaMemsetAsync(next, 0, 8, ctx->stream));
        a.in = two ? side.P2 : side.P1;
        a.item_start = dstart;
        a.item_len = dlen;
        a.nitems = (long long)ni;
        a.next = next;
        a.fine_bits = FB;
        a.kbase = L.kbase;
        a.pbase = L.pbase;
        const unsigned grid = (unsigned)std::min<long long>(2LL * ctx->sm_count, (long long)ni);
        const size_t wide = GbrTable<GBR_PAIR, GBR_PT_SLOTS>::BYTES, packed = GbrTable<GBR_PACKED, GBR_PT_SLOTS>::BYTES;
        rc = L.packed ? launch_fold(ctx, gbr_part_kernel<GBR_PACKED>, grid, GBR_PT_THREADS, packed, a)
             : pair32 ? launch_fold(ctx, gbr_part_kernel<GBR_PAIR32>, grid, GBR_PT_THREADS, wide, a)
                      : launch_fold(ctx, gbr_part_kernel<GBR_PAIR>, grid, GBR_PT_THREADS, wide, a);
    } while (0);
    // Stream-ordered frees: the kernels above finish before the memory is reused.
    dfree(ctx, dstart);
    dfree(ctx, side.P1);
    dfree(ctx, side.P2);
    return rc;
}

}  // namespace pyg
