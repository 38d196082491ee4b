// Scan, stable LSD radix sort, gather, and the sort / lower-bound entry
// points (reference SortOp and TupleBuffer::sort / findsmallest).
#include <string.h>

#include "lookback.cuh"
#include "primitives.cuh"

namespace pyg {

// ---------------------------------------------------------------------------
// Exclusive scan (three phases: block reduce, scan of block totals, scan).

constexpr int SCAN_THREADS = 1024;

__device__ __forceinline__ unsigned long long block_incl_scan(unsigned long long v, unsigned long long* warp_tot)
{
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        unsigned long long t = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += t;
    }
    if (lane == 31) warp_tot[w] = v;
    __syncthreads();
    if (w == 0) {
        int nw = blockDim.x >> 5;
        unsigned long long x = lane < nw ? warp_tot[lane] : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            unsigned long long t = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += t;
        }
        if (lane < nw) warp_tot[lane] = x;
    }
    __syncthreads();
    unsigned long long r = v + (w > 0 ? warp_tot[w - 1] : 0);
    __syncthreads();
    return r;
}

__global__ void scan_reduce_kernel(const unsigned long long* __restrict__ in, int64_t n, int64_t chunk,
                                   unsigned long long* __restrict__ partial)
{
    __shared__ unsigned long long red[32];
    int64_t lo = blockIdx.x * chunk, hi = min(n, lo + chunk);
    unsigned long long s = 0;
    for (int64_t i = lo + threadIdx.x; i < hi; i += blockDim.x) s += in[i];
    s = warp_sum_u64(s);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x < 32) {
        unsigned long long x = threadIdx.x < (blockDim.x >> 5) ? red[threadIdx.x] : 0;
        x = warp_sum_u64(x);
        if (threadIdx.x == 0) partial[blockIdx.x] = x;
    }
}

// Exclusive scan of `partial` (nb entries, one block), total to *total.
__global__ void scan_partials_kernel(unsigned long long* partial, int nb, unsigned long long* total)
{
    __shared__ unsigned long long warp_tot[32];
    unsigned long long carry = 0;
    for (int base = 0; base < nb; base += blockDim.x) {
        int i = base + threadIdx.x;
        unsigned long long v = i < nb ? partial[i] : 0;
        unsigned long long incl = block_incl_scan(v, warp_tot);
        if (i < nb) partial[i] = carry + incl - v;
        __shared__ unsigned long long last;
        if (threadIdx.x == blockDim.x - 1) last = incl;
        __syncthreads();
        carry += last;
        __syncthreads();
    }
    if (threadIdx.x == 0 && total) *total = carry;
}

__global__ void scan_apply_kernel(const unsigned long long* in, unsigned long long* out, int64_t n, int64_t chunk,
                                  const unsigned long long* __restrict__ partial)
{
    __shared__ unsigned long long warp_tot[32];
    __shared__ unsigned long long last;
    int64_t lo = blockIdx.x * chunk, hi = min(n, lo + chunk);
    unsigned long long carry = partial[blockIdx.x];
    for (int64_t base = lo; base < hi; base += blockDim.x) {
        int64_t i = base + threadIdx.x;
        unsigned long long v = i < hi ? in[i] : 0;
        unsigned long long incl = block_incl_scan(v, warp_tot);
        if (threadIdx.x == blockDim.x - 1) last = incl;
        if (i < hi) out[i] = carry + incl - v;
        __syncthreads();
        carry += last;
        __syncthreads();
    }
}

int exclusive_scan_u64(pyg_ctx* ctx, const unsigned long long* in, unsigned long long* out, int64_t n,
                       unsigned long long* total_dev)
{
    if (n <= 0) {
        if (total_dev) PYG_CUDA(cudaMemsetAsync(total_dev, 0, 8, ctx->stream));
        return PYG_OK;
    }
    int nb = (int)((n + 65535) / 65536);
    if (nb > 4096) nb = 4096;
    int64_t chunk = (n + nb - 1) / nb;
    nb = (int)((n + chunk - 1) / chunk);
    unsigned long long* partial;
    int rc = dalloc(ctx, (void**)&partial, nb * sizeof(unsigned long long));
    if (rc) return rc;
    scan_reduce_kernel<<<nb, SCAN_THREADS, 0, ctx->stream>>>(in, n, chunk, partial);
    PYG_LAUNCHED(ctx);
    scan_partials_kernel<<<1, SCAN_THREADS, 0, ctx->stream>>>(partial, nb, total_dev);
    PYG_LAUNCHED(ctx);
    scan_apply_kernel<<<nb, SCAN_THREADS, 0, ctx->stream>>>(in, out, n, chunk, partial);
    PYG_LAUNCHED(ctx);
    dfree(ctx, partial);
    return PYG_OK;
}

// ---------------------------------------------------------------------------
// Stable LSD radix sort in one sweep per 8-bit digit, the published Onesweep
// scheme (Adinets and Merrill, "Onesweep: A Faster Least Significant Digit
// Radix Sort for GPUs", 2022).
//
//   range   one read takes the smallest and largest key and the low bits that
//           all keys share; digits are those of key - smallest above these, so
//           only the bits the keys span are sorted (a signed 40-bit range
//           takes 5 passes, not 8; 256 multiples of 2^56 take one).
//   hist    one read counts every pass's digits (shared-memory counters).
//   pass    each CTA takes a tile by ticket, ranks it by digit, learns how
//           many elements of each digit precede the tile from its
//           predecessors' status words (decoupled look-back), groups the
//           tile by digit in shared memory and writes each digit's run
//           contiguously: one read and one write of the data per digit.
//
// Bound: 32 bytes per 16-byte tuple and pass (98 us at 20 M tuples and the
// copy bandwidth); a pass takes 191 us there: 148 thread instructions per
// tuple (44% issue active), barriers between the phases of a tile and the
// 16-byte shared-memory scatter.  Measured, 20 M tuples of 40-bit signed
// keys: 1114 us, against 4636 us with a histogram, a scan and an unstaged
// scatter per digit over separate key and value arrays, eight digits (the
// sign's copies counted as key bits) and a split and a merge of the tuples.
// CTA shapes measured for the whole sort (threads x elements, CTAs per SM):
// 512 x 8, 2: 1144 us; 384 x 12, 2: 1139; 256 x 16, 2: 1147; 512 x 12, 1:
// 1234; 512 x 6, 2: 1243; 256 x 16, 3 and 512 x 12, 2 spill registers
// (1311, 1283).
//
// The waits of the look-back are bounded (lookback.cuh).  A wait that gives up
// sets the context's sort error word, and nothing that was queued behind it
// touches the unfinished order: passes, gathers and merges look at the word
// first.

constexpr int OS_BINS = 256;
constexpr int OS_MAX_PASSES = 8;

// Elements: 16-byte {x, y} sorted by word FIELD, or bare 8-byte keys.
template <typename Item, int FIELD>
__device__ __forceinline__ uint64_t os_key(const Item& t)
{
    if constexpr (sizeof(Item) == 8) return t;
    else return FIELD ? t.y : t.x;
}

// Threads and elements per thread of a pass's CTA.
template <typename Item>
struct OsShape {
    static constexpr int THREADS = 512;
    static constexpr int PER = sizeof(Item) == 16 ? 8 : 12;
    static constexpr int MINB = 2;
    static constexpr int TILE = THREADS * PER;
    static constexpr int WARPS = THREADS / 32;
    static constexpr size_t COUNTERS = (size_t)WARPS * OS_BINS * 4;
    static constexpr size_t STAGE = (size_t)TILE * sizeof(Item);
    static constexpr size_t SMEM = STAGE > COUNTERS ? STAGE : COUNTERS;  // the counters are consumed before staging
};

// Smallest and largest key, each as an atomicMin (words start at all ones):
// words[0] the smallest order-preserving image, words[1] the complement of
// the largest; words[2] the bits in which all keys are equal.
template <typename Item, int FIELD>
__global__ void __launch_bounds__(512) os_range_kernel(const Item* __restrict__ in, int64_t n, uint64_t flip,
                                                       unsigned long long* __restrict__ words)
{
    unsigned long long lo = ~0ULL, hi = ~0ULL, diff = 0;
    const unsigned long long first = os_key<Item, FIELD>(in[0]) ^ flip;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    auto take = [&](const Item& t) {
        const unsigned long long k = os_key<Item, FIELD>(t) ^ flip;
        lo = min(lo, k);
        hi = min(hi, ~k);
        diff |= k ^ first;
    };
    constexpr int U = 4;
    for (; i + (U - 1) * stride < n; i += U * stride) {
        Item t[U];
#pragma unroll
        for (int u = 0; u < U; ++u) t[u] = in[i + u * stride];
#pragma unroll
        for (int u = 0; u < U; ++u) take(t[u]);
    }
    for (; i < n; i += stride) take(in[i]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        lo = min(lo, __shfl_xor_sync(0xffffffffu, lo, o));
        hi = min(hi, __shfl_xor_sync(0xffffffffu, hi, o));
        diff |= __shfl_xor_sync(0xffffffffu, diff, o);
    }
    __shared__ unsigned long long red[3][16];
    if ((threadIdx.x & 31) == 0) {
        red[0][threadIdx.x >> 5] = lo;
        red[1][threadIdx.x >> 5] = hi;
        red[2][threadIdx.x >> 5] = ~diff;
    }
    __syncthreads();
    if (threadIdx.x < 3) {
        unsigned long long m = ~0ULL;
        for (int w = 0; w < 16; ++w) m = threadIdx.x < 2 ? min(m, red[threadIdx.x][w]) : m & red[2][w];
        if (threadIdx.x < 2) atomicMin(&words[threadIdx.x], m);
        else atomicAnd(&words[2], m);
    }
}

// Scratch of one sort, zeroed before use: digit counts (then their
// exclusive prefixes) per pass, tickets, and one status word per (tile,
// digit).  A status word holds a count above its 8-bit tag; pass p tags
// the tile's own count 2 p + 1 and the count of all tiles up to it 2 p + 2,
// so the words need no reset between passes.
struct OsScratch {
    unsigned long long hist[OS_MAX_PASSES][OS_BINS];
    unsigned ticket[OS_MAX_PASSES + 1];  // [OS_MAX_PASSES]: histogram CTAs done
    unsigned pad[7];
};

// Digit counts of all passes in one read.  Each digit has HREP copies of
// its counter, chosen by lane, so that narrow digits (few distinct values)
// do not serialise a warp on one address; the last CTA to finish turns the
// totals into exclusive prefixes.
constexpr int OS_HREP = 4;
template <typename Item, int FIELD>
__global__ void __launch_bounds__(512) os_hist_kernel(const Item* __restrict__ in, int64_t n, uint64_t base, int low, int passes,
                                                      OsScratch* __restrict__ sc)
{
    extern __shared__ unsigned os_h[];  // [pass][digit][copy]
    __shared__ bool last;
    const int words = passes * OS_BINS * OS_HREP;
    for (int b = threadIdx.x; b < words; b += blockDim.x) os_h[b] = 0;
    __syncthreads();
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    unsigned* mine = os_h + (threadIdx.x & (OS_HREP - 1));
    auto count = [&](const Item& t) {
        uint64_t k = (os_key<Item, FIELD>(t) - base) >> low;
        for (int p = 0; p < passes; ++p, k >>= 8) atomicAdd(&mine[(p * OS_BINS + (int)(k & 255)) * OS_HREP], 1u);
    };
    constexpr int U = 4;
    for (; i + (U - 1) * stride < n; i += U * stride) {
        Item t[U];
#pragma unroll
        for (int u = 0; u < U; ++u) t[u] = in[i + u * stride];
#pragma unroll
        for (int u = 0; u < U; ++u) count(t[u]);
    }
    for (; i < n; i += stride) count(in[i]);
    __syncthreads();
    for (int b = threadIdx.x; b < passes * OS_BINS; b += blockDim.x) {
        unsigned c = 0;
        for (int r = 0; r < OS_HREP; ++r) c += os_h[b * OS_HREP + r];
        if (c) atomicAdd(&sc->hist[0][b], (unsigned long long)c);
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(&sc->ticket[OS_MAX_PASSES], 1u) == gridDim.x - 1;
    __syncthreads();
    if (!last) return;
    __threadfence();
    // Warp p scans pass p's 256 counts, 8 per lane.
    const int p = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (p >= passes) return;
    unsigned long long c[8], sum = 0;
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        c[q] = __ldcg(&sc->hist[p][lane * 8 + q]);
        sum += c[q];
    }
    unsigned long long incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += v;
    }
    unsigned long long run = incl - sum;
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        sc->hist[p][lane * 8 + q] = run;
        run += c[q];
    }
}

// Elements of digit `d` in the tiles before `tile`: walks the predecessors'
// status words back to the nearest inclusive count, LOOK words in flight
// per step.  false when the wait gave up.
__device__ bool os_look_back(const unsigned long long* status, int64_t tile, int d, unsigned agg_tag, unsigned* err,
                             unsigned long long& before)
{
    constexpr int LOOK = 8;
    unsigned long long sum = 0, t0 = 0;
    int64_t j = tile - 1;
    for (;;) {
        unsigned long long v[LOOK];
#pragma unroll
        for (int q = 0; q < LOOK; ++q) v[q] = j - q >= 0 ? lb_load(status + (j - q) * OS_BINS + d) : 0ULL;
        int used = 0;
        bool open = true;
#pragma unroll
        for (int q = 0; q < LOOK; ++q) {
            if (!open) continue;
            const unsigned tag = (unsigned)(v[q] & 255);
            if (tag == agg_tag + 1) {
                before = sum + (v[q] >> 8);
                return true;
            }
            if (tag == agg_tag) {
                sum += v[q] >> 8;
                ++used;
            } else {
                open = false;
            }
        }
        j -= used;
        if (used == 0) {
            const unsigned long long now = bulk_now_ns();
            if (t0 == 0) t0 = now;
            else if (now - t0 > kLookBackWaitNs || *(volatile unsigned*)err) {
                atomicOr(err, 1u);
                return false;
            }
        } else {
            t0 = 0;
        }
    }
}

template <typename Item, int FIELD>
__global__ void __launch_bounds__(OsShape<Item>::THREADS, OsShape<Item>::MINB)
    os_pass_kernel(const Item* __restrict__ in, Item* __restrict__ out, int64_t n, uint64_t base, int shift, int pass,
                   OsScratch* __restrict__ sc, unsigned long long* __restrict__ status,
                   unsigned* __restrict__ err, int64_t mute)
{
    using S = OsShape<Item>;
    constexpr int PER = S::PER, TILE = S::TILE, WARPS = S::WARPS;
    extern __shared__ __align__(16) unsigned char os_smem[];
    Item* stage = reinterpret_cast<Item*>(os_smem);
    unsigned(*wcnt)[OS_BINS] = reinterpret_cast<unsigned(*)[OS_BINS]>(os_smem);  // before staging
    __shared__ unsigned long long gbase[OS_BINS];  // output position of staged slot i = gbase[digit] + i
    __shared__ unsigned warp_tot[OS_BINS / 32];
    __shared__ unsigned ticket;
    __shared__ int ok;
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const unsigned agg_tag = 2u * (unsigned)pass + 1u;
    if (tid == 0) {
        ticket = atomicAdd(&sc->ticket[pass], 1u);
        ok = *(volatile unsigned*)err == 0;
    }
    for (int b = tid; b < WARPS * OS_BINS; b += S::THREADS) (&wcnt[0][0])[b] = 0;
    __syncthreads();
    // A pass that gave up left tiles unwritten: what is read here is then no
    // permutation of what was counted, and its digits have no bound.
    if (!ok) return;
    const int64_t tile = ticket;
    const int64_t first = tile * TILE;
    const int count = n - first < TILE ? (int)(n - first) : TILE;
    // (1) Load: warp w owns a contiguous run of 32 x PER elements, so the
    // order (warp, row, lane) is the input order and the ranks are stable.
    Item t[PER];
    const int e0 = w * (32 * PER) + lane;
    if (count == TILE) {
#pragma unroll
        for (int j = 0; j < PER; ++j) t[j] = in[first + e0 + j * 32];
    } else {
#pragma unroll
        for (int j = 0; j < PER; ++j)
            if (e0 + j * 32 < count) t[j] = in[first + e0 + j * 32];
    }
    // (2) Rank within the warp: lanes of one digit find one another with
    // eight ballots; the warp's counter of the digit gives the rank's base.
    // Slots past the end count as digit 255: they rank after every element.
    unsigned short rank[PER];
    unsigned char dig[PER];
    const unsigned below = (1u << lane) - 1u;
#pragma unroll
    for (int j = 0; j < PER; ++j) {
        const bool valid = e0 + j * 32 < count;
        const unsigned d = valid ? (unsigned)((os_key<Item, FIELD>(t[j]) - base) >> shift) & 255u : 255u;
        unsigned m = 0xffffffffu;
#pragma unroll
        for (int b = 0; b < 8; ++b) {
            const unsigned bit = (d >> b) & 1u;
            m &= __ballot_sync(0xffffffffu, bit) ^ (bit - 1u);
        }
        const unsigned old = wcnt[w][d];
        __syncwarp();
        if ((m & below) == 0) wcnt[w][d] = old + __popc(m);
        __syncwarp();
        rank[j] = (unsigned short)(old + __popc(m & below));
        dig[j] = (unsigned char)d;
    }
    __syncthreads();
    // (3) Digit totals of the tile, published at once; then their prefix.
    unsigned long long* st = status + tile * OS_BINS;
    unsigned c = 0, incl = 0;
    if (tid < OS_BINS) {
        for (int v = 0; v < WARPS; ++v) c += wcnt[v][tid];
        const unsigned real = tid == OS_BINS - 1 ? c - (unsigned)(TILE - count) : c;
        if (tile != mute) lb_store(st + tid, ((unsigned long long)real << 8) | (tile == 0 ? agg_tag + 1 : agg_tag));
        incl = c;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned v = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += v;
        }
        if (lane == 31) warp_tot[w] = incl;
    }
    __syncthreads();
    unsigned start = 0;
    if (tid < OS_BINS) {
        start = incl - c;
        for (int v = 0; v < w; ++v) start += warp_tot[v];
        unsigned run = start;
        for (int v = 0; v < WARPS; ++v) {
            const unsigned x = wcnt[v][tid];
            wcnt[v][tid] = run;
            run += x;
        }
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < PER; ++j) rank[j] = (unsigned short)(rank[j] + wcnt[w][dig[j]]);
    __syncthreads();  // the counters' memory becomes the stage
    // (4) Group the tile by digit; meanwhile the look-back.
#pragma unroll
    for (int j = 0; j < PER; ++j) stage[rank[j]] = t[j];
    if (tid < OS_BINS) {
        unsigned long long before = 0;
        if (tile > 0) {
            const unsigned real = tid == OS_BINS - 1 ? c - (unsigned)(TILE - count) : c;
            if (os_look_back(status, tile, tid, agg_tag, err, before))
                lb_store(st + tid, ((before + real) << 8) | (agg_tag + 1));
            else
                ok = 0;
        }
        gbase[tid] = sc->hist[pass][tid] + before - start;
    }
    __syncthreads();
    if (!ok) return;
    // (5) Write each digit's run.
#pragma unroll
    for (int j = 0; j < PER; ++j) {
        const int i = j * S::THREADS + tid;
        if (i < count) {
            const Item x = stage[i];
            out[gbase[(unsigned)((os_key<Item, FIELD>(x) - base) >> shift) & 255u] + i] = x;
        }
    }
}

// Up to OS_SMALL elements: one CTA sorts (key, input position) with a
// bitonic network in shared memory and gathers the elements; one launch, no
// host round trip.  At these sizes the digit passes are launches and a
// round trip (a group-by of 16 groups: 1284 us with this kernel, 1320 us
// with the key range's round trip and digit passes).
constexpr int OS_SMALL = 4096;
constexpr int OS_SMALL_SMEM = OS_SMALL * 8 + OS_SMALL * 2;

template <typename Item, int FIELD>
__global__ void __launch_bounds__(1024) os_small_kernel(const Item* __restrict__ in, int n, uint64_t flip,
                                                        Item* __restrict__ out)
{
    extern __shared__ __align__(16) unsigned char os_smem[];
    uint64_t* key = reinterpret_cast<uint64_t*>(os_smem);
    unsigned short* idx = reinterpret_cast<unsigned short*>(key + OS_SMALL);
    int m = 64;
    while (m < n) m <<= 1;
    for (int i = threadIdx.x; i < m; i += blockDim.x) {
        key[i] = i < n ? os_key<Item, FIELD>(in[i]) ^ flip : ~0ULL;
        idx[i] = (unsigned short)i;  // padding: the largest key, the largest positions
    }
    // Keys in order already (equal ones among them) need no network: 4000
    // equal keys took 58 us with it.
    __syncthreads();
    bool disorder = false;
    for (int i = threadIdx.x; i + 1 < n; i += blockDim.x) disorder |= key[i] > key[i + 1];
    if (!__syncthreads_or(disorder)) m = 0;
    // Pairs at stride j <= 32 stay inside the warp's own 64-element blocks:
    // those stages need only a warp barrier.
    bool wide = true;
    for (int k = 2; k <= m; k <<= 1) {
        for (int j = k >> 1; j > 0; j >>= 1) {
            if (wide || j >= 64) __syncthreads();
            else __syncwarp();
            wide = j >= 64;
            for (int p = threadIdx.x; p < m / 2; p += blockDim.x) {
                const int a = 2 * p - (p & (j - 1)), b = a + j;
                const uint64_t ka = key[a], kb = key[b];
                const unsigned short ia = idx[a], ib = idx[b];
                const bool gt = ka > kb || (ka == kb && ia > ib);
                if (gt == ((a & k) == 0)) {
                    key[a] = kb;
                    key[b] = ka;
                    idx[a] = ib;
                    idx[b] = ia;
                }
            }
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < n; i += blockDim.x) out[i] = in[idx[i]];
}

// Key range of the elements and the digit passes it needs.  One host round
// trip: the number of launches depends on it.
struct OsPlan {
    uint64_t base = 0;
    int low = 0;  // low bits that all keys share
    int passes = 0;
};

// Launches the range reading of n > 0 elements into counter words 128 + 4
// slot; os_plan_read turns the words into a plan after a synchronisation.
template <typename Item, int FIELD>
static int os_plan_launch(pyg_ctx* ctx, const Item* in, int64_t n, bool is_signed, int slot)
{
    const uint64_t flip = is_signed ? 0x8000000000000000ULL : 0ULL;
    unsigned long long* words = ctx->dcounters + 128 + 4 * slot;
    PYG_CUDA(cudaMemsetAsync(words, 0xFF, 24, ctx->stream));
    os_range_kernel<Item, FIELD><<<grid_for(ctx, n, 512, 4, 4), 512, 0, ctx->stream>>>(in, n, flip, words);
    PYG_LAUNCHED(ctx);
    PYG_CUDA(cudaMemcpyAsync((unsigned long long*)ctx->pinned + 64 + 4 * slot, words, 24, cudaMemcpyDeviceToHost,
                             ctx->stream));
    return PYG_OK;
}

static OsPlan os_plan_read(pyg_ctx* ctx, bool is_signed, int slot)
{
    const unsigned long long* h = (const unsigned long long*)ctx->pinned + 64 + 4 * slot;
    const uint64_t lo = h[0], hi = ~h[1];
    OsPlan plan;
    plan.base = lo ^ (is_signed ? 0x8000000000000000ULL : 0ULL);
    if (hi != lo) {
        plan.low = __builtin_ctzll(~h[2]);
        plan.passes = (64 - __builtin_clzll((hi - lo) >> plan.low) + 7) / 8;
    }
    return plan;
}

template <typename Item, int FIELD>
static int os_plan(pyg_ctx* ctx, const Item* in, int64_t n, bool is_signed, OsPlan* plan)
{
    int rc = os_plan_launch<Item, FIELD>(ctx, in, n, is_signed, 0);
    if (rc) return rc;
    PYG_CUDA(cudaStreamSynchronize(ctx->stream));
    *plan = os_plan_read(ctx, is_signed, 0);
    return PYG_OK;
}

// The passes of a plan: pass p writes dst0 (p even) or dst1 (p odd).
template <typename Item, int FIELD>
static int os_passes(pyg_ctx* ctx, const Item* in, Item* dst0, Item* dst1, int64_t n, const OsPlan& plan)
{
    using S = OsShape<Item>;
    if (plan.passes == 0) return PYG_OK;
    const int64_t tiles = (n + S::TILE - 1) / S::TILE;
    const size_t bytes = sizeof(OsScratch) + (size_t)tiles * OS_BINS * 8;
    OsScratch* sc;
    int rc = dalloc(ctx, (void**)&sc, bytes);
    if (rc) return rc;
    unsigned long long* status = (unsigned long long*)(sc + 1);
    auto run = [&]() -> int {
        PYG_CUDA(cudaMemsetAsync(sc, 0, bytes, ctx->stream));
        const size_t hsm = (size_t)plan.passes * OS_BINS * OS_HREP * 4;
        os_hist_kernel<Item, FIELD>
            <<<grid_for(ctx, n, 512, 16, 4), 512, hsm, ctx->stream>>>(in, n, plan.base, plan.low, plan.passes, sc);
        PYG_LAUNCHED(ctx);
        auto kern = os_pass_kernel<Item, FIELD>;
        PYG_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S::SMEM));
        const Item* src = in;
        int64_t mute = ctx->stall_sort && tiles > 1 ? 0 : -1;
        if (mute == 0) ctx->stall_sort = 0;
        for (int p = 0; p < plan.passes; ++p, mute = -1) {
            Item* dst = p & 1 ? dst1 : dst0;
            kern<<<(unsigned)tiles, S::THREADS, S::SMEM, ctx->stream>>>(src, dst, n, plan.base, plan.low + 8 * p, p, sc,
                                                                        status,
                                                                        (unsigned*)(ctx->dcounters + SORT_ERR_WORD),
                                                                        mute);
            PYG_LAUNCHED(ctx);
            src = dst;
        }
        PYG_CUDA(cudaMemcpyAsync((unsigned long long*)ctx->pinned + SORT_ERR_PINNED, ctx->dcounters + SORT_ERR_WORD, 8,
                                 cudaMemcpyDeviceToHost, ctx->stream));
        return PYG_OK;
    };
    rc = run();
    dfree(ctx, sc);
    return rc;
}

int sort_status(pyg_ctx* ctx)
{
    unsigned long long* h = (unsigned long long*)ctx->pinned + SORT_ERR_PINNED;
    if (*h == 0) return PYG_OK;
    *h = 0;
    PYG_CUDA(cudaMemsetAsync(ctx->dcounters + SORT_ERR_WORD, 0, 8, ctx->stream));
    set_error("sort: a bounded wait for an earlier tile gave up");
    return PYG_ERR_TIMEOUT;
}

template <typename Item, int FIELD>
static int os_small(pyg_ctx* ctx, const Item* in, Item* out, int64_t n, bool is_signed)
{
    os_small_kernel<Item, FIELD><<<1, 1024, OS_SMALL_SMEM, ctx->stream>>>(
        in, (int)n, is_signed ? 0x8000000000000000ULL : 0ULL, out);
    PYG_LAUNCHED(ctx);
    return PYG_OK;
}

// The passes into out, whose last one writes it.
template <typename Item, int FIELD>
static int os_run_to(pyg_ctx* ctx, const Item* in, Item* out, int64_t n, const OsPlan& plan)
{
    if (plan.passes == 0) {  // one key value: the input order is the answer
        PYG_CUDA(cudaMemcpyAsync(out, in, (size_t)n * sizeof(Item), cudaMemcpyDeviceToDevice, ctx->stream));
        return PYG_OK;
    }
    Item* tmp = nullptr;
    int rc;
    if (plan.passes > 1 && (rc = dalloc(ctx, (void**)&tmp, (size_t)n * sizeof(Item)))) return rc;
    rc = plan.passes & 1 ? os_passes<Item, FIELD>(ctx, in, out, tmp, n, plan)
                         : os_passes<Item, FIELD>(ctx, in, tmp, out, n, plan);
    dfree(ctx, tmp);
    return rc;
}

template <typename Item, int FIELD>
static int os_sort_to(pyg_ctx* ctx, const Item* in, Item* out, int64_t n, bool is_signed)
{
    if (n <= 0) return PYG_OK;
    if (n <= OS_SMALL) return os_small<Item, FIELD>(ctx, in, out, n, is_signed);
    OsPlan plan;
    int rc = os_plan<Item, FIELD>(ctx, in, n, is_signed, &plan);
    return rc ? rc : os_run_to<Item, FIELD>(ctx, in, out, n, plan);
}

int radix_sort16_two(pyg_ctx* ctx, const ulonglong2* const in[2], ulonglong2* const out[2], const int64_t n[2])
{
    int rc;
    bool wait = false;
    for (int s = 0; s < 2; ++s)
        if (n[s] > OS_SMALL) {
            if ((rc = os_plan_launch<ulonglong2, 0>(ctx, in[s], n[s], true, s))) return rc;
            wait = true;
        }
    if (wait) PYG_CUDA(cudaStreamSynchronize(ctx->stream));
    for (int s = 0; s < 2; ++s) {
        if (n[s] <= 0) continue;
        if (n[s] <= OS_SMALL) rc = os_small<ulonglong2, 0>(ctx, in[s], out[s], n[s], true);
        else rc = os_run_to<ulonglong2, 0>(ctx, in[s], out[s], n[s], os_plan_read(ctx, true, s));
        if (rc) return rc;
    }
    return PYG_OK;
}

int radix_sort16_to(pyg_ctx* ctx, const ulonglong2* in, ulonglong2* out, int64_t n, int field, bool is_signed)
{
    return field ? os_sort_to<ulonglong2, 1>(ctx, in, out, n, is_signed)
                 : os_sort_to<ulonglong2, 0>(ctx, in, out, n, is_signed);
}

int radix_sort8_to(pyg_ctx* ctx, const uint64_t* in, uint64_t* out, int64_t n, bool is_signed)
{
    return os_sort_to<uint64_t, 0>(ctx, in, out, n, is_signed);
}

template <int FIELD>
static int os_sort_swap(pyg_ctx* ctx, ulonglong2* a, ulonglong2* b, int64_t n, ulonglong2** result)
{
    *result = a;
    if (n <= 1) return PYG_OK;
    if (n <= OS_SMALL) {
        *result = b;
        return os_small<ulonglong2, FIELD>(ctx, a, b, n, false);
    }
    OsPlan plan;
    int rc = os_plan<ulonglong2, FIELD>(ctx, a, n, false, &plan);
    if (rc) return rc;
    if (plan.passes & 1) *result = b;
    return os_passes<ulonglong2, FIELD>(ctx, a, b, a, n, plan);
}

int radix_sort16_swap(pyg_ctx* ctx, ulonglong2* a, ulonglong2* b, int64_t n, int field, ulonglong2** result)
{
    return field ? os_sort_swap<1>(ctx, a, b, n, result) : os_sort_swap<0>(ctx, a, b, n, result);
}

// ---------------------------------------------------------------------------
// Gather, key extraction, sort entry point.

// err: the error word of the sort that ordered the items (row numbers of a
// sort that gave up may be anything).
template <typename V>
__global__ void gather_kernel(const V* __restrict__ in, const ulonglong2* __restrict__ items, int64_t n, int words,
                              V* __restrict__ out, const unsigned* __restrict__ err)
{
    if (*err) return;
    int64_t total = n * words;
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total; t += (int64_t)gridDim.x * blockDim.x) {
        int64_t r = t / words;
        int c = (int)(t - r * words);
        out[t] = in[items[r].y * words + c];
    }
}

int gather_rows(pyg_ctx* ctx, const uint8_t* in, const ulonglong2* items, int64_t n, int32_t tb, uint8_t* out)
{
    if (n <= 0) return PYG_OK;
    const unsigned* err = (const unsigned*)(ctx->dcounters + SORT_ERR_WORD);
    int threads = 256;
    if (tb % 16 == 0 && (uintptr_t)in % 16 == 0 && (uintptr_t)out % 16 == 0) {
        gather_kernel<uint4><<<grid_for(ctx, n * (tb / 16), threads, 4, 8), threads, 0, ctx->stream>>>(
            (const uint4*)in, items, n, tb / 16, (uint4*)out, err);
    } else if (tb % 8 == 0 && (uintptr_t)in % 8 == 0 && (uintptr_t)out % 8 == 0) {
        gather_kernel<uint2><<<grid_for(ctx, n * (tb / 8), threads, 4, 8), threads, 0, ctx->stream>>>(
            (const uint2*)in, items, n, tb / 8, (uint2*)out, err);
    } else if (tb % 4 == 0 && (uintptr_t)in % 4 == 0 && (uintptr_t)out % 4 == 0) {
        gather_kernel<unsigned><<<grid_for(ctx, n * (tb / 4), threads, 4, 8), threads, 0, ctx->stream>>>(
            (const unsigned*)in, items, n, tb / 4, (unsigned*)out, err);
    } else {
        gather_kernel<unsigned char><<<grid_for(ctx, n * tb, threads, 4, 8), threads, 0, ctx->stream>>>(
            in, items, n, tb, out, err);
    }
    PYG_LAUNCHED(ctx);
    return PYG_OK;
}

// (key, row number) items of a relation's tuples.
__global__ void extract_keys_kernel(const uint8_t* __restrict__ base, int64_t n, int32_t tb, int32_t off, int32_t type,
                                    ulonglong2* __restrict__ items)
{
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        items[i] = make_ulonglong2(to_sortable(load_col(base + i * (int64_t)tb, off, type)), (uint64_t)i);
}

// Sorts a device relation by one column into out (device).  16-byte tuples
// with an int64 key are the sort's elements themselves: the first pass
// reads the relation and the last one writes out.  Other layouts sort (key,
// row) items and gather the rows.
int sort_relation(pyg_ctx* ctx, const pyg_rel* r, int32_t key_col, void* out)
{
    int64_t n = r->ntuples;
    if (n == 0) return PYG_OK;
    const size_t bytes = (size_t)n * r->tuple_bytes;
    if ((uintptr_t)out < (uintptr_t)r->base + bytes && (uintptr_t)r->base < (uintptr_t)out + bytes) {
        // In place: the first pass (or the gather) would write tuples that
        // others have yet to read, so a copy is sorted.
        pyg_rel copy = *r;
        void* buf;
        int rc = dalloc(ctx, &buf, bytes);
        if (rc) return rc;
        copy.base = buf;
        cudaError_t e = cudaMemcpyAsync(buf, r->base, bytes, cudaMemcpyDeviceToDevice, ctx->stream);
        rc = e == cudaSuccess ? sort_relation(ctx, &copy, key_col, out) : cuda_status(e, "in-place sort");
        dfree(ctx, buf);
        return rc;
    }
    int32_t off = r->col_offset[key_col], type = r->col_type[key_col];
    if (r->tuple_bytes == 16 && type == PYG_INT64 && (off == 0 || off == 8) && (uintptr_t)r->base % 16 == 0 &&
        (uintptr_t)out % 16 == 0)
        return radix_sort16_to(ctx, (const ulonglong2*)r->base, (ulonglong2*)out, n, off == 8, true);
    ulonglong2 *items, *sorted;
    int rc = dalloc(ctx, (void**)&items, (size_t)2 * n * sizeof(ulonglong2));
    if (rc) return rc;
    extract_keys_kernel<<<grid_for(ctx, n, 256, 4, 8), 256, 0, ctx->stream>>>((const uint8_t*)r->base, n,
                                                                              r->tuple_bytes, off, type, items);
    PYG_LAUNCHED(ctx);
    if (!(rc = radix_sort16_swap(ctx, items, items + n, n, 0, &sorted)))
        rc = gather_rows(ctx, (const uint8_t*)r->base, sorted, n, r->tuple_bytes, (uint8_t*)out);
    dfree(ctx, items);
    return rc;
}

__global__ void lower_bound_kernel(const uint8_t* __restrict__ base, int64_t n, int32_t tb, int32_t off, int32_t type,
                                   const int64_t* __restrict__ q, int64_t nq, int64_t* __restrict__ out)
{
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < nq; i += (int64_t)gridDim.x * blockDim.x) {
        int64_t key = q[i];
        int64_t lo = 0, hi = n;
        while (lo < hi) {
            int64_t mid = lo + (hi - lo) / 2;
            if (load_col(base + mid * (int64_t)tb, off, type) < key) lo = mid + 1;
            else hi = mid;
        }
        out[i] = lo;
    }
}

}  // namespace pyg

using namespace pyg;

extern "C" {

int pyg_sort(pyg_ctx* ctx, const pyg_rel* in, int32_t key_col, void* out)
{
    int rc = check_ctx(ctx);
    if (rc) return rc;
    if ((rc = check_rel(in, "sort input"))) return rc;
    if (key_col < 0 || key_col >= in->ncols || (in->ntuples > 0 && !out)) {
        set_error("pyg_sort: bad key column %d or null out", key_col);
        return PYG_ERR_ARG;
    }
    DevRel r;
    if ((rc = r.stage(ctx, in))) return rc;
    rc = sort_relation(ctx, &r.rel, key_col, out);
    r.release(ctx);
    if (rc) return rc;
    PYG_CUDA(cudaStreamSynchronize(ctx->stream));
    return sort_status(ctx);
}

int pyg_lower_bound(pyg_ctx* ctx, const pyg_rel* sorted, int32_t key_col, const int64_t* queries, int64_t nq,
                    int64_t* out_idx)
{
    int rc = check_ctx(ctx);
    if (rc) return rc;
    if ((rc = check_rel(sorted, "sorted"))) return rc;
    if (key_col < 0 || key_col >= sorted->ncols || nq < 0 || (nq > 0 && (!queries || !out_idx))) {
        set_error("pyg_lower_bound: bad arguments");
        return PYG_ERR_ARG;
    }
    if (!sorted->on_device) {
        set_error("pyg_lower_bound: the sorted relation must be device-resident");
        return PYG_ERR_ARG;
    }
    if (nq == 0) return PYG_OK;
    lower_bound_kernel<<<grid_for(ctx, nq, 256, 1, 8), 256, 0, ctx->stream>>>(
        (const uint8_t*)sorted->base, sorted->ntuples, sorted->tuple_bytes, sorted->col_offset[key_col],
        sorted->col_type[key_col], queries, nq, out_idx);
    PYG_LAUNCHED(ctx);
    return PYG_OK;
}

}  // extern "C"
