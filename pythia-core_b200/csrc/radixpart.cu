// Hash partitioning shared by the radix operators: kernels and host
// helpers (declared in radixpart.cuh).
#include <cuda_runtime.h>
#include <stdint.h>
#include <string.h>

#include <algorithm>
#include <climits>
#include <cmath>
#include <type_traits>
#include <vector>

#include "bulk.cuh"
#include "radixpart.cuh"

namespace pyg {

constexpr unsigned long long kBulkWaitNs = 2000000000ULL;  // 2 s

__device__ __forceinline__ unsigned rj_bin(uint64_t h, int shift, unsigned mask)
{
    return shift >= 64 ? 0u : (unsigned)(h >> shift) & mask;
}

// ---------------------------------------------------------------------------
// 1. Histogram of the top `bits` hash bits (bits <= 15: 128 KB of shared
// counters per CTA).

template <bool MODEL>
__global__ void __launch_bounds__(1024) rj_hist_kernel(const longlong2* __restrict__ in, int64_t n, int64_t step,
                                                       int spread, int bits, int base, int span, unsigned* __restrict__ part,
                                                       long long* __restrict__ mm, RJModel model)
{
    // Counts the bins [base, base + span) of one tuple in every `step`
    // (rj_sample_row; step 1: every tuple); span 32-bit counters in shared memory,
    // stored to this CTA's row of part (rj_hist_sum_kernel adds the rows).
    // With mm: also the key and payload ranges of the tuples read.  MODEL:
    // the bins are the learned model's (rj_model_bin) instead of hash bits.
    extern __shared__ unsigned rj_sh_hist[];
    __shared__ long long sh_mm[4];
    const int P = 1 << bits;
    const int shift = 64 - bits;
    const int64_t m = (n + step - 1) / step;
    for (int b = threadIdx.x; b < span; b += blockDim.x) rj_sh_hist[b] = 0;
    if (threadIdx.x < 4) sh_mm[threadIdx.x] = (threadIdx.x & 1) ? LLONG_MIN : LLONG_MAX;
    __syncthreads();
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    long long kmin = LLONG_MAX, kmax = LLONG_MIN, pmin = LLONG_MAX, pmax = LLONG_MIN;
    auto count = [&](const longlong2 t) {
        const uint64_t code = MODEL ? rj_model_code(model, t.x) : rj_hash((uint64_t)t.x);
        const unsigned r = rj_bin(code, shift, P - 1) - (unsigned)base;
        if (r < (unsigned)span) atomicAdd(&rj_sh_hist[r], 1u);
        kmin = min(kmin, t.x);
        kmax = max(kmax, t.x);
        pmin = min(pmin, t.y);
        pmax = max(pmax, t.y);
    };
    constexpr int U = 8;
    for (; i + (U - 1) * stride < m; i += U * stride) {
        longlong2 t[U];
#pragma unroll
        for (int u = 0; u < U; ++u) t[u] = __ldcs(&in[rj_sample_row(i + u * stride, step, spread, n)]);
#pragma unroll
        for (int u = 0; u < U; ++u) count(t[u]);
    }
    for (; i < m; i += stride) count(__ldcs(&in[rj_sample_row(i, step, spread, n)]));
    if (mm) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            kmin = min(kmin, __shfl_xor_sync(0xffffffffu, kmin, o));
            kmax = max(kmax, __shfl_xor_sync(0xffffffffu, kmax, o));
            pmin = min(pmin, __shfl_xor_sync(0xffffffffu, pmin, o));
            pmax = max(pmax, __shfl_xor_sync(0xffffffffu, pmax, o));
        }
        if ((threadIdx.x & 31) == 0) {
            atomicMin(&sh_mm[0], kmin);
            atomicMax(&sh_mm[1], kmax);
            atomicMin(&sh_mm[2], pmin);
            atomicMax(&sh_mm[3], pmax);
        }
    }
    __syncthreads();
    unsigned* row = part + (size_t)blockIdx.x * span;
    for (int b = threadIdx.x; b < span; b += blockDim.x) row[b] = rj_sh_hist[b];
    if (mm && threadIdx.x == 0) {
        atomicMin(&mm[0], sh_mm[0]);
        atomicMax(&mm[1], sh_mm[1]);
        atomicMin(&mm[2], sh_mm[2]);
        atomicMax(&mm[3], sh_mm[3]);
    }
}

// mm = {LLONG_MAX, LLONG_MIN, LLONG_MAX, LLONG_MIN}: empty key / payload ranges.
__global__ void rj_mm_init_kernel(long long* mm)
{
    if (threadIdx.x < 4) mm[threadIdx.x] = (threadIdx.x & 1) ? LLONG_MIN : LLONG_MAX;
}

// hist[b] = sum over the nrow rows of part[row * span + b], b < span: the
// CTAs' shared-memory histograms added column by column (coalesced and in a
// fixed order) instead of by atomics from every CTA on each bin.
__global__ void rj_hist_sum_kernel(const unsigned* __restrict__ part, int nrow, int span,
                                   unsigned long long* __restrict__ hist)
{
    const int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= span) return;
    unsigned long long sum = 0;
    for (int r = 0; r < nrow; ++r) sum += part[(size_t)r * span + b];
    hist[b] = sum;
}

// Tiles of `tile` elements per segment, as an exclusive prefix (one CTA, one
// thread per segment; at most 2^9 segments): tiles[C] is the pass's tile
// count.  Counts are first clamped to their region's capacity, so a region
// that overflowed (its result is discarded and redone) is never read past its
// end.
__global__ void __launch_bounds__(RJ_LMAX) rj_tile_prefix_kernel(const unsigned long long* __restrict__ cursor, int cstride,
                                                                 unsigned long long* __restrict__ count,
                                                                 const unsigned long long* __restrict__ cap, int C,
                                                                 int tile, unsigned long long* __restrict__ tiles)
{
    __shared__ unsigned long long warp_tot[RJ_LMAX / 32];
    const int c = threadIdx.x, lane = c & 31, w = c >> 5;
    unsigned long long t = 0;
    if (c < C) {
        const unsigned long long reached = cursor[(size_t)c * cstride];
        const unsigned long long n = reached < cap[c] ? reached : cap[c];
        count[c] = n;
        t = (n + tile - 1) / tile;
    }
    unsigned long long incl = t;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += v;
    }
    if (lane == 31) warp_tot[w] = incl;
    __syncthreads();
    for (int v = 0; v < w; ++v) incl += warp_tot[v];
    if (c == 0) tiles[0] = 0;
    if (c < C) tiles[c + 1] = incl;
}

// ---------------------------------------------------------------------------
// 2. Tile partition pass with exact offsets.  The input is a sequence of
// segments (one for the first pass; the coarse partitions for the second);
// tiles never straddle a segment.  Output bin of a tuple = (segment <<
// lbits) | ((rj_hash(key) >> shift) & mask).

struct RJPass {
    const longlong2* in;
    longlong2* out;
    const unsigned long long* seg_start;  // nseg + 1 exact segment bounds in `in`
    const unsigned long long* seg_tile0;  // nseg + 1 prefix of tiles per segment
    int nseg;
    int tile;                             // elements per tile (at most the kernel's largest)
    int shift;
    unsigned mask;
    int lbits;
    const unsigned long long* bin_start;  // output region start per output bin
    unsigned long long* cursor;           // per output bin, zeroed before the pass; bin b at b * cstride
    int cstride;
    unsigned* err;                        // set if a tile's bulk copy never completed
    // Optional (null when offsets are exact):
    const unsigned long long* seg_count;  // tuples in each segment (segment end = start + count)
    const unsigned long long* bin_cap;    // region capacity per output bin
    unsigned* ovf;                        // set when a bin outgrows its region
    unsigned long long dump;              // first of RJ_DUMP elements of `out` that take the runs of such bins
    const unsigned long long* ntiles_dev; // tile count read on the device
    // Range mode (nsplit > 0): bin = number of splitters <= key among the
    // segment's nsplit splitters, split + seg * 2^lbits (one segment: split).
    const long long* split;
    int nsplit;
    // Packed elements: frame of the 8-byte words, and the flag set when a
    // 16-byte input tuple falls outside it.
    unsigned long long kbase, pbase;
    unsigned* frame;
    // Model mode (the kernel's RJ_MODE_MODEL instances): the bin bits come
    // from the learned model's code (rj_model_code) instead of the key's hash.
    RJModel model;
};

// How a pass computes a tuple's bin, fixed per kernel instance so that no
// per-tuple branch chooses it.
// HASH9: hash bins, more than 2^8 of them, of a pass from 16-byte tuples to
// packed words; it has a shape of its own.
enum RJMode { RJ_MODE_HASH = 0, RJ_MODE_MODEL = 1, RJ_MODE_RANGE = 2, RJ_MODE_HASH9 = 3 };

// Element formats: a pass reads 16-byte tuples (the relation, or unpacked
// intermediates) or packed 8-byte words, and writes either.  Packed input
// has bins of at most 2^8, so the staged bin index is one byte.
template <bool IN8, bool OUT8, int MODE>
struct RJFmt {
    using In = typename std::conditional<IN8, unsigned long long, longlong2>::type;
    using Out = typename std::conditional<OUT8, unsigned long long, longlong2>::type;
    using Bin = typename std::conditional<IN8, unsigned char, unsigned short>::type;
    static constexpr int TILE =
        IN8 ? (MODE == RJ_MODE_HASH ? RJ_TILE_8 : RJ_TILE_8M)
            : !OUT8 ? (MODE == RJ_MODE_HASH ? RJ_TILE_U : RJ_TILE_UM)
                    : (MODE == RJ_MODE_HASH ? RJ_TILE_P : MODE == RJ_MODE_HASH9 ? RJ_TILE_P9 : RJ_TILE_PM);  // the largest
};

__device__ __forceinline__ long long rj_key(const longlong2& t, unsigned long long) { return t.x; }
__device__ __forceinline__ long long rj_key(unsigned long long w, unsigned long long kbase)
{
    return (long long)(kbase + (w & 0xFFFFFFFFULL));
}

struct RJTileRange {
    long long begin, end;
    int seg;
};

// The segment of the tiles one CTA issues, kept in the issuing thread's
// registers.  A CTA's tiles come in increasing order, so the segment only
// moves forward: most tiles stay in the current segment and need no global
// load; a tile past its end steps forward (over empty segments too) and
// loads the new segment's bounds.  Over a whole pass a CTA reads each
// segment's bounds at most once.
struct RJSegCursor {
    int seg;               // -1 before the first tile
    long long t0, t1;      // seg_tile0[seg], seg_tile0[seg + 1]
    long long start, end;  // the segment's elements in `in`
};

__device__ RJTileRange rj_tile_range(const RJPass& a, RJSegCursor& c, long long tile)
{
    if (tile >= c.t1) {
        int s = c.seg < 0 ? 0 : c.seg + 1;
        long long t1 = (long long)a.seg_tile0[s + 1];
        while (tile >= t1 && s + 1 < a.nseg) t1 = (long long)a.seg_tile0[++s + 1];
        c.seg = s;
        c.t0 = (long long)a.seg_tile0[s];
        c.t1 = t1;
        c.start = (long long)a.seg_start[s];
        c.end = a.seg_count ? c.start + (long long)a.seg_count[s] : (long long)a.seg_start[s + 1];
    }
    RJTileRange r;
    r.seg = c.seg;
    r.begin = c.start + (tile - c.t0) * a.tile;
    r.end = min(r.begin + a.tile, c.end);
    return r;
}

// Shape of a partition kernel's CTA: worker threads, control warps, resident
// CTAs per SM, input tiles in flight.  Chosen with the tile sizes
// (radixpart.cuh) by measuring both passes of R 2^27 x S 2^30 (hash), the
// learned and sampled MPSM join of 2^26 x 2^28 and the group-by of 2^27:
//   16-byte in, packed out, hash     probe pass 1 4.79 ms.  One CTA per SM and
//     the largest tile: a tile reserves one run per bin, and at 2048-tuple
//     tiles the 64-bit atomics on 128 cursors alone took a third of the pass
//     (7.7 ms; 5.1 ms with them taken out).  2 x 512 threads, 4096: 7.1 ms.
//     2^9 bins keep one control warp busy for longer than a tile: two of them
//     and 960 workers take the join of 2.2 M x 30 M random 31-bit keys from
//     684 to 588 us, x 100 M from 1930 to 1655.  With 2^7 bins that shape
//     costs 1.3% (R 2^27 x S 2^30), so it is taken above 2^8 bins only.
//   packed in and out, hash          probe pass 2 4.03 ms.  256 bins: two
//     control warps reserve four each per lane (one warp: 4.70 ms).
//   16-byte in and out, hash         two control warps and 2688-tuple tiles.
//     With one and 2400, the reservations of 2^9 bins held the tiles up: join
//     of 2.2 M x 30 M wide keys in one pass 877 -> 719 us, x 100 M 2088 -> 1636,
//     group-by of 100 M wide keys, G 2^20, 2729 -> 2310; 2^7 bins gain 4% to 6%.
//     1 x 992 and 5952: 846 us, 1 x 960, two control warps and 5760: 735.
//   model and range bins wait on their leaf and splitter loads and take
//     whichever shape measured best: 2.87 and 2.20 ms (model), 3.71 and
//     2.38 ms (range).
// Against one kernel shape of 2 x 256 or 512 threads without control warps,
// three barriers per tile and reservations waited for inside a tile: 6.78,
// 4.66 (hash), 3.09, 1.95 (model), 3.92 and 3.05 ms (range).
template <int WORKERS, int CONTROL, int CTAS, int STAGES>
struct RJShapeOf {
    static constexpr int T = WORKERS, NC = CONTROL, MINB = CTAS, ST = STAGES, THREADS = T + 32 * NC;
};
template <bool IN8, bool OUT8, int MODE>
struct RJShape : RJShapeOf<480, 1, 2, 1> {};  // second and unpacked passes of model and range bins
template <>
struct RJShape<false, false, RJ_MODE_HASH> : RJShapeOf<448, 2, 2, 1> {};
template <>
struct RJShape<true, true, RJ_MODE_HASH> : RJShapeOf<448, 2, 2, 1> {};
template <>
struct RJShape<false, true, RJ_MODE_HASH> : RJShapeOf<992, 1, 1, 1> {};
template <>
struct RJShape<false, true, RJ_MODE_HASH9> : RJShapeOf<960, 2, 1, 1> {};
template <>
struct RJShape<false, true, RJ_MODE_MODEL> : RJShapeOf<992, 1, 1, 2> {};
template <>
struct RJShape<false, true, RJ_MODE_RANGE> : RJShapeOf<992, 1, 1, 2> {};

// Shared memory of one partition CTA: a ring of input tiles that bulk
// copies fill ahead of use, the grouped (staged) tile, and per-bin
// counters.
template <bool IN8, bool OUT8, int MODE>
struct RJPartSmem {
    using F = RJFmt<IN8, OUT8, MODE>;
    // Model and range passes have at most 2^8 bins (RJ_SPLIT_MAX).
    static constexpr int BINS = MODE == RJ_MODE_HASH || MODE == RJ_MODE_HASH9 ? RJ_LMAX : RJ_SPLIT_MAX;
    static constexpr int ST = RJShape<IN8, OUT8, MODE>::ST;
    typename F::In in[ST][F::TILE];
    typename F::Out stage[F::TILE];
    unsigned long long gdelta[BINS];  // output position of staged slot i = gdelta[bin] + i
    unsigned hist[2][BINS];           // tile counts per bin; tiles alternate
    unsigned loff[BINS];
    typename F::Bin stage_bin[F::TILE];
    uint64_t bar[ST];
    RJTileRange info[ST];
    unsigned total[2];                 // elements of a tile; tiles alternate
    int seg;                           // the tile being reserved: its segment
    unsigned hot;                      // a bin that held many of the last tile's tuples, else no bin
    int ok;
    long long split[2][MODE == RJ_MODE_RANGE ? RJ_SPLIT_MAX : 1];  // the splitters of this tile and the next
    // Model bins of 16-byte tuples: the model's tables, where they fit.  A
    // first pass reads leaves at random: through L1 each lane of a gather is
    // a tag lookup, in shared memory it is a few bank conflicts (both passes'
    // first halves of 2^26 x 2^28, theta 1.0: 3.75 -> 2.87 ms; what bounds
    // them now is shared memory, 76% busy).  Second passes meet the few
    // leaves of one coarse partition and hit L1.
    static constexpr bool TABLES = MODE == RJ_MODE_MODEL && !IN8;
    RJLeaf leaf[TABLES ? RJ_SM_LEAVES : 1];
    int2 hinfo[TABLES ? RJ_SM_LEAVES : 1];
    long long hkey[TABLES ? RJ_SM_HEAVY : 1];
    float hw[TABLES ? RJ_SM_HEAVY : 1];
};
__device__ __forceinline__ unsigned rj_range_bin(const long long* sp, int n, long long k)
{
    int lo = 0;
    while (n > 0) {
        const int half = n >> 1;
        if (k >= sp[lo + half]) {
            lo += half + 1;
            n -= half + 1;
        } else {
            n = half;
        }
    }
    return (unsigned)lo;
}

// One warp: the splitters of segment seg into dst.
__device__ __forceinline__ void rj_load_split(const RJPass& a, long long* dst, int seg, int lane)
{
    const long long* src = a.split + (a.nseg > 1 ? ((long long)seg << a.lbits) : 0);
    for (int i = lane; i < a.nsplit; i += 32) dst[i] = src[i];
}

// Histogram of range bins of one tuple in every `step`: fine bin = coarse bin
// (among C - 1 coarse splitters held in shared memory) * 2^sub + bin among
// that coarse range's 2^sub - 1 fine splitters (read from global memory).
__global__ void __launch_bounds__(1024) rj_hist_range_kernel(const longlong2* __restrict__ in, int64_t n, int64_t step,
                                                             int spread, int CB, int sub, const long long* __restrict__ csplit,
                                                             const long long* __restrict__ fsplit,
                                                             unsigned* __restrict__ part, long long* __restrict__ mm)
{
    extern __shared__ __align__(16) unsigned char rj_hr_raw[];
    const int F = 1 << (CB + sub), C = 1 << CB, L = 1 << sub;
    long long* cs = (long long*)rj_hr_raw;
    unsigned* h = (unsigned*)(cs + RJ_SPLIT_MAX);
    for (int b = threadIdx.x; b < F; b += blockDim.x) h[b] = 0;
    for (int i = threadIdx.x; i < C - 1; i += blockDim.x) cs[i] = csplit[i];
    __syncthreads();
    const int64_t m = (n + step - 1) / step;
    long long kmin = LLONG_MAX, kmax = LLONG_MIN, pmin = LLONG_MAX, pmax = LLONG_MIN;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < m; i += stride) {
        const longlong2 t = __ldcs(&in[rj_sample_row(i, step, spread, n)]);
        const long long k = t.x;
        kmin = min(kmin, t.x);
        kmax = max(kmax, t.x);
        pmin = min(pmin, t.y);
        pmax = max(pmax, t.y);
        unsigned f = rj_range_bin(cs, C - 1, k);
        if (sub) f = (f << sub) | rj_range_bin(fsplit + ((long long)f << sub), L - 1, k);
        atomicAdd(&h[f], 1u);
    }
    if (mm) {  // key and payload ranges of the tuples read
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            kmin = min(kmin, __shfl_xor_sync(0xffffffffu, kmin, o));
            kmax = max(kmax, __shfl_xor_sync(0xffffffffu, kmax, o));
            pmin = min(pmin, __shfl_xor_sync(0xffffffffu, pmin, o));
            pmax = max(pmax, __shfl_xor_sync(0xffffffffu, pmax, o));
        }
        if ((threadIdx.x & 31) == 0) {
            atomicMin(&mm[0], kmin);
            atomicMax(&mm[1], kmax);
            atomicMin(&mm[2], pmin);
            atomicMax(&mm[3], pmax);
        }
    }
    __syncthreads();
    unsigned* row = part + (size_t)blockIdx.x * F;
    for (int b = threadIdx.x; b < F; b += blockDim.x) row[b] = h[b];
}

// Thread 0: starts the bulk copy of tile `tile` into ring slot `slot`.
// Packed tiles start at an even word (regions and tiles are even), and the
// copy is rounded up to 16 bytes: at most one word past the tile, inside
// the buffer's 16-byte tail, which is never used as data.
template <bool IN8, bool OUT8, int MODE>
__device__ __forceinline__ void rj_issue_tile(const RJPass& a, RJPartSmem<IN8, OUT8, MODE>& sm, RJSegCursor& cur,
                                              int slot, long long tile)
{
    using F = RJFmt<IN8, OUT8, MODE>;
    const RJTileRange r = rj_tile_range(a, cur, tile);
    sm.info[slot] = r;
    const unsigned bytes = ((unsigned)(r.end - r.begin) * (unsigned)sizeof(typename F::In) + 15u) & ~15u;
    mbar_arrive_expect_tx(&sm.bar[slot], bytes);
    bulk_load(sm.in[slot], reinterpret_cast<const typename F::In*>(a.in) + r.begin, bytes, &sm.bar[slot]);
}

// One partition pass.  T worker threads move the tuples; the control warps
// make the global reservations, and the first of them also starts the input
// copies and scans the bins, so that no worker waits on an atomic or holds
// the others up with a scan.  Bound: the shared-memory traffic of ranking and
// staging (about 25 wavefronts per 32 tuples) and the workers' instructions;
// the probe side's passes of 2^27 x 2^30 move 5.4 and 4.3 TB/s.  Two tiles are in the works: while tile k waits for the
// reservations of its runs, tile k + 1 is binned and ranked; while the
// control warp scans the bins of tile k + 1, the workers write tile k out.
// Two CTA barriers per tile:
//   workers                                   control warps
//   bin and rank tile k + 1                   reserve the runs of tile k
//   -- barrier 1
//   write out tile k                          next input copy; scan tile k + 1
//   -- barrier 2
//   group tile k + 1 in the stage             (reserve the runs of tile k + 1)
static_assert(sizeof(RJPartSmem<false, true, RJ_MODE_HASH>) <= 232448, "one CTA per SM");
static_assert(sizeof(RJPartSmem<false, true, RJ_MODE_HASH9>) <= 232448, "one CTA per SM");
static_assert(sizeof(RJPartSmem<false, true, RJ_MODE_MODEL>) <= 232448, "one CTA per SM");
static_assert(2 * (sizeof(RJPartSmem<true, true, RJ_MODE_HASH>) + 1024) <= 233472, "two CTAs per SM");
static_assert(2 * (sizeof(RJPartSmem<true, true, RJ_MODE_RANGE>) + 1024) <= 233472, "two CTAs per SM");
static_assert(2 * (sizeof(RJPartSmem<false, false, RJ_MODE_HASH>) + 1024) <= 233472, "two CTAs per SM");
static_assert(2 * (sizeof(RJPartSmem<false, false, RJ_MODE_RANGE>) + 1024) <= 233472, "two CTAs per SM");

template <bool IN8, bool OUT8, int MODE>
__global__ void __launch_bounds__(RJShape<IN8, OUT8, MODE>::THREADS, RJShape<IN8, OUT8, MODE>::MINB)
    rj_partition_kernel(RJPass a, long long ntiles)
{
    using F = RJFmt<IN8, OUT8, MODE>;
    using Smem = RJPartSmem<IN8, OUT8, MODE>;
    using Out = typename F::Out;
    if (a.ntiles_dev) ntiles = (long long)*a.ntiles_dev;
    extern __shared__ __align__(128) unsigned char rj_pt_raw[];
    Smem& sm = *reinterpret_cast<Smem*>(rj_pt_raw);
    constexpr int T = RJShape<IN8, OUT8, MODE>::T;
    constexpr int NC = RJShape<IN8, OUT8, MODE>::NC;
    constexpr int PER = F::TILE / T;
    constexpr int ST = Smem::ST;
    constexpr int BINS = Smem::BINS;
    static_assert(PER * T == F::TILE, "whole rows of elements");
    const int L = 1 << a.lbits;
    const int tid = threadIdx.x, lane = tid & 31;
    for (int b = tid; b < 2 * BINS; b += T + 32 * NC) (&sm.hist[0][0])[b] = 0;
    const bool tables = Smem::TABLES && a.model.L <= RJ_SM_LEAVES && a.model.H <= RJ_SM_HEAVY;
    if constexpr (Smem::TABLES) {
        if (tables) {
            for (int l = tid; l < a.model.L; l += T + 32 * NC) {
                sm.leaf[l] = a.model.leaf[l];
                if (a.model.H) sm.hinfo[l] = a.model.hinfo[l];
            }
            for (int h = tid; h < a.model.H; h += T + 32 * NC) {
                sm.hkey[h] = a.model.hkey[h];
                sm.hw[h] = a.model.hw[h];
            }
        }
    }
    if (tid >= T) {
        // ---- control warps; the first one does all but the reservations
        const int ct = tid - T;
        const bool first = ct < 32;
        RJSegCursor segc{-1, -1, -1, 0, 0};  // lane 0: segment of the tiles it issues
        if (ct == 0) {
            for (int s = 0; s < ST; ++s) mbar_init(&sm.bar[s], 1);
            mbar_fence_init();
            for (int s = 0; s < ST; ++s)
                if (blockIdx.x + (long long)s * gridDim.x < ntiles)
                    rj_issue_tile(a, sm, segc, s, blockIdx.x + (long long)s * gridDim.x);
            sm.ok = 1;
            sm.hot = ~0u;
            sm.total[0] = sm.total[1] = 0;
        }
        __syncwarp();
        if constexpr (MODE == RJ_MODE_RANGE) {
            if (first && blockIdx.x < ntiles) rj_load_split(a, sm.split[0], sm.info[0].seg, lane);
        }
        __syncthreads();
        long long k = 0;
        for (long long tile = blockIdx.x;; tile += gridDim.x, ++k) {
            __syncthreads();  // 1
            if (!sm.ok || tile >= ntiles) {
                // A wait ran out: copies still in flight get as long again to
                // land before this CTA's shared memory is given up.
                if (ct == 0 && !sm.ok) {
                    atomicOr(a.err, 1u);
                    for (int s = 0; s < ST; ++s)
                        if (tile + (long long)s * gridDim.x < ntiles)
                            mbar_wait(&sm.bar[(k + s) % ST], (unsigned)(((k + s) / ST) & 1), kBulkWaitNs);
                }
                break;
            }
            const int slot = (int)(k % ST);
            unsigned* hist = sm.hist[k & 1];
            if (first) {
                __syncwarp();
                if (lane == 0) {
                    sm.seg = sm.info[slot].seg;
                    const long long nt = tile + (long long)ST * gridDim.x;
                    if (nt < ntiles) {
                        fence_proxy_async_smem();
                        rj_issue_tile(a, sm, segc, slot, nt);
                    }
                }
                // Range mode over several segments: the next tile's splitters
                // (its copy has been issued, so its segment is known).
                if constexpr (MODE == RJ_MODE_RANGE) {
                    __syncwarp();
                    if (a.nseg > 1 && tile + gridDim.x < ntiles)
                        rj_load_split(a, sm.split[(k + 1) & 1], sm.info[(k + 1) % ST].seg, lane);
                }
                // Scan of the bins: lane l holds the 4 G consecutive ones from
                // 4 G l (G = 1 below 128 bins).
                const uint4* h4 = reinterpret_cast<const uint4*>(hist);
                uint4* l4 = reinterpret_cast<uint4*>(sm.loff);
                constexpr int GMAX = BINS / 128;
                const int G = L > 128 ? L >> 7 : 1;
                uint4 h[GMAX];
                unsigned sum = 0, top = 0;
#pragma unroll
                for (int g = 0; g < GMAX; ++g) {
                    const int b = 4 * (G * lane + g);
                    h[g] = g < G && b < L ? h4[b >> 2] : make_uint4(0, 0, 0, 0);
                    sum += h[g].x + h[g].y + h[g].z + h[g].w;
                    top = max(top, max(max(h[g].x << 9 | b, h[g].y << 9 | (b + 1)),
                                       max(h[g].z << 9 | (b + 2), h[g].w << 9 | (b + 3))));
                }
                unsigned run = sum;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const unsigned v = __shfl_up_sync(0xffffffffu, run, o);
                    if (lane >= o) run += v;
                }
                unsigned x = run - sum;
#pragma unroll
                for (int g = 0; g < GMAX; ++g) {
                    const int b = 4 * (G * lane + g);
                    if (g < G && b < L) l4[b >> 2] = make_uint4(x, x + h[g].x, x + h[g].x + h[g].y, x + h[g].x + h[g].y + h[g].z);
                    x += h[g].x + h[g].y + h[g].z + h[g].w;
                }
                top = __reduce_max_sync(0xffffffffu, top);
                if (lane == 31) {
                    sm.total[k & 1] = run;
                    sm.hot = (top >> 9) * 4 >= (unsigned)a.tile ? top & 511u : ~0u;
                }
            }
            __syncthreads();  // 2
            const int seg = sm.seg;
            // Each non-empty bin reserves its run with one global atomic and
            // its counter is reset.  A run that outgrows its region goes to
            // the dump; the host redoes the relation from an exact histogram.
            constexpr int CT = 32 * NC, U = BINS / CT < 4 ? BINS / CT : 4;
            for (int b0 = ct; b0 < L; b0 += CT * U) {
                unsigned c[U];
                unsigned long long pos[U], end[U];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const int b = b0 + u * CT;
                    c[u] = b < L ? hist[b] : 0u;
                    if (c[u]) {
                        const unsigned ob = ((unsigned)seg << a.lbits) | (unsigned)b;
                        const unsigned long long start = a.bin_start[ob];
                        end[u] = a.bin_cap ? start + a.bin_cap[ob] : ~0ULL;
                        pos[u] = start + atomicAdd(&a.cursor[(size_t)ob * a.cstride], (unsigned long long)c[u]);
                        hist[b] = 0;
                    }
                }
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const int b = b0 + u * CT;
                    if (c[u]) {
                        const bool over = pos[u] + c[u] > end[u];
                        if (over) atomicOr(a.ovf, 1u);
                        sm.gdelta[b] = (over ? a.dump : pos[u]) - sm.loff[b];
                    }
                }
            }
        }
        return;
    }
    // ---- workers
    Out* out = reinterpret_cast<Out*>(a.out);
    unsigned miss = 0;  // nonzero when a tuple was outside the packed frame
    __syncthreads();
    long long k = 0;
    for (long long tile = blockIdx.x;; tile += gridDim.x, ++k) {
        const bool more = tile < ntiles;  // uniform; the last turn only writes out
        Out t[PER];
        unsigned br[PER];  // bin << 16 | rank
        if (more) {
            const int slot = (int)(k % ST);
            unsigned* hist = sm.hist[k & 1];
            // Every thread waits for the tile; a wait that runs out marks the
            // CTA failed and that thread's tuples are left out, so nothing is
            // written from memory the copy did not fill.
            const bool landed = mbar_wait(&sm.bar[slot], (unsigned)((k / ST) & 1), kBulkWaitNs);
            if (!landed) sm.ok = 0;
            const unsigned n = landed ? (unsigned)(sm.info[slot].end - sm.info[slot].begin) : 0u;
            const unsigned hot = sm.hot;
            // Bin and rank every tuple with a shared atomic.  When one bin
            // held at least a quarter of the last tile (skewed keys), the
            // lanes of that bin take their ranks from one atomic.
            auto bin_rank = [&](int j, bool valid) {
                br[j] = 0xFFFFFFFFu;
                unsigned bin = 0;
                if (valid) {
                    const typename F::In e = sm.in[slot][j * T + tid];
                    const long long key = rj_key(e, a.kbase);
                    if constexpr (IN8 || !OUT8) {
                        t[j] = e;
                    } else {
                        // Pack: (key - kbase) | (payload - pbase) << 32.  The
                        // key offset 2^32 - 1, which marks free slots in the
                        // tables built from the words, is outside the frame
                        // too: dk + 1 then carries into its high half (and dk
                        // itself has one where dk + 1 wraps to 0).  A comparison
                        // dk >= 2^32 - 1 measured 12872 us, this 12816, neither
                        // test 12764 (R 2^27 x S 2^30).
                        const unsigned long long dk = (unsigned long long)e.x - a.kbase;
                        const unsigned long long dp = (unsigned long long)e.y - a.pbase;
                        miss |= (unsigned)(dk >> 32) | (unsigned)((dk + 1) >> 32) | (unsigned)(dp >> 32);
                        t[j] = (dk & 0xFFFFFFFFULL) | (dp << 32);
                    }
                    if constexpr (Smem::TABLES) {
                        if (tables) {
                            RJModel m = a.model;
                            m.leaf = sm.leaf;
                            m.hinfo = a.model.H ? sm.hinfo : nullptr;
                            m.hkey = sm.hkey;
                            m.hw = sm.hw;
                            bin = rj_bin(rj_model_code(m, key), a.shift, a.mask);
                        } else {
                            bin = rj_bin(rj_model_code(a.model, key), a.shift, a.mask);
                        }
                    } else if constexpr (MODE == RJ_MODE_MODEL)
                        bin = rj_bin(rj_model_code(a.model, key), a.shift, a.mask);
                    else if constexpr (MODE == RJ_MODE_RANGE)
                        bin = rj_range_bin(sm.split[a.nseg > 1 ? (k & 1) : 0], a.nsplit, key);
                    else
                        bin = rj_bin(rj_hash((uint64_t)key), a.shift, a.mask);
                }
                if (hot != ~0u) {
                    const unsigned m = __ballot_sync(0xffffffffu, valid && bin == hot);
                    unsigned base = 0;
                    if (m) {
                        const int lead = __ffs(m) - 1;
                        if (lane == lead) base = atomicAdd(&hist[hot], (unsigned)__popc(m));
                        base = __shfl_sync(0xffffffffu, base, lead);
                    }
                    if (valid)
                        br[j] = (bin << 16) | (bin == hot ? base + __popc(m & ((1u << lane) - 1u)) : atomicAdd(&hist[bin], 1u));
                } else if (valid) {
                    br[j] = (bin << 16) | atomicAdd(&hist[bin], 1u);
                }
            };
            if (IN8 && n == (unsigned)F::TILE) {
#pragma unroll
                for (int j = 0; j < PER; ++j) bin_rank(j, true);
            } else {
#pragma unroll
                for (int j = 0; j < PER; ++j) bin_rank(j, j * T + tid < n);
            }
        }
        __syncthreads();  // 1: hist[k] complete, ring slot consumed; stage and gdelta of the tile before complete
        if (!sm.ok) break;
        if (k > 0) {
            // Write the staged tile, each bin's run contiguously.
            const unsigned total = sm.total[(k & 1) ^ 1];
#pragma unroll
            for (int j = 0; j < PER; ++j) {
                const unsigned i = j * T + tid;
                if (i < total) __stcs(&out[sm.gdelta[sm.stage_bin[i]] + i], sm.stage[i]);
            }
        }
        if (!more) break;
        __syncthreads();  // 2: in-tile offsets ready, the stage is free
#pragma unroll
        for (int j = 0; j < PER; ++j)
            if (br[j] != 0xFFFFFFFFu) {
                const unsigned bin = br[j] >> 16;
                const unsigned s = sm.loff[bin] + (br[j] & 0xFFFFu);
                sm.stage[s] = t[j];
                sm.stage_bin[s] = (typename F::Bin)bin;
            }
    }
    if (miss) atomicOr(a.frame, 1u);
}


namespace {

template <bool IN8, bool OUT8, int MODE>
int launch_pass_t(pyg_ctx* ctx, const RJPass& p, long long ntiles)
{
    auto fn = rj_partition_kernel<IN8, OUT8, MODE>;
    const size_t smem = sizeof(RJPartSmem<IN8, OUT8, MODE>);
    PYG_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    int per_sm = 0;
    constexpr int T = RJShape<IN8, OUT8, MODE>::THREADS;
    PYG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, T, smem));
    if (per_sm < 1) per_sm = 1;
    long long grid = std::min<long long>(ntiles, (long long)ctx->sm_count * per_sm);
    fn<<<(unsigned)grid, T, smem, ctx->stream>>>(p, ntiles);
    PYG_LAUNCHED(ctx);
    return PYG_OK;
}

// One pass: 16-byte tuples in and out, 16-byte tuples in and packed words
// out (the first pass of a packed layout), or packed words in and out.
template <int MODE>
int launch_pass_m(pyg_ctx* ctx, const RJPass& p, long long ntiles, bool in8, bool out8)
{
    if (in8) return launch_pass_t<true, true, MODE>(ctx, p, ntiles);
    if (out8) return launch_pass_t<false, true, MODE>(ctx, p, ntiles);
    return launch_pass_t<false, false, MODE>(ctx, p, ntiles);
}

int launch_pass(pyg_ctx* ctx, const RJPass& p, long long ntiles, bool in8, bool out8)
{
    if (ntiles <= 0) return PYG_OK;
    if (p.model.leaf) return launch_pass_m<RJ_MODE_MODEL>(ctx, p, ntiles, in8, out8);
    if (p.nsplit) return launch_pass_m<RJ_MODE_RANGE>(ctx, p, ntiles, in8, out8);
    if (!in8 && out8 && p.lbits > 8) return launch_pass_t<false, true, RJ_MODE_HASH9>(ctx, p, ntiles);
    return launch_pass_m<RJ_MODE_HASH>(ctx, p, ntiles, in8, out8);
}

// Host-side layout of one relation's partitions.  Exact layouts come from a
// full histogram (dense, contiguous partitions); sampled layouts size each
// partition's region from a sample of the rows with six standard deviations of

}  // namespace

// Tiles of the passes; C: the first pass's bins (launch_pass takes HASH9 above
// 2^8 of them).
static void layout_tiles(RJLayout& L, int64_t n, int C, bool pack, bool model)
{
    const int packing = model ? RJ_TILE_PM : (C > 1 << 8 ? RJ_TILE_P9 : RJ_TILE_P);
    L.tile1 = rj_tile(!pack ? (model ? RJ_TILE_UM : RJ_TILE_U) : packing, n);
    L.tile2 = rj_tile(!pack ? (model ? RJ_TILE_UM : RJ_TILE_U) : (model ? RJ_TILE_8M : RJ_TILE_8), n);
}

void layout_exact(const std::vector<unsigned long long>& h, int64_t n, int C, int sub, RJLayout& L, bool pack,
                  bool model)
{
    layout_tiles(L, n, C, pack, model);
    const size_t F = h.size();
    L.sampled = false;
    L.packed = pack;
    // Packed regions are rounded up to an even number of words.
    auto sz = [&](unsigned long long c) { return pack ? (c + 1) & ~1ULL : c; };
    L.fstart.assign(F + 1, 0);
    for (size_t f = 0; f < F; ++f) L.fstart[f + 1] = L.fstart[f] + sz(h[f]);
    L.cstart.assign(C + 1, 0);
    for (int c = 0; c <= C; ++c) L.cstart[c] = L.fstart[(size_t)c << sub];
    L.fcap.clear();
    L.ccap.clear();
    L.tiles2.assign(C + 1, 0);
    if (pack) {
        // The second pass's tiles come from the first pass's cursors (the
        // exact counts), formed on the device as for sampled layouts; the
        // region sizes bound them.
        L.ccap.assign(C, 0);
        L.tiles2_max = 0;
        for (int c = 0; c < C; ++c) {
            L.ccap[c] = L.cstart[c + 1] - L.cstart[c];
            L.tiles2_max += (L.ccap[c] + L.tile2 - 1) / L.tile2;
        }
    } else {
        for (int c = 0; c < C; ++c)
            L.tiles2[c + 1] = L.tiles2[c] + (L.cstart[c + 1] - L.cstart[c] + L.tile2 - 1) / L.tile2;
        L.tiles2_max = L.tiles2[C];
    }
    L.count = h;
    L.p1 = L.p2 = L.fstart[F];
}

// Capacity of a region that c of the samples fell into (rounded up).
static inline unsigned long long sampled_cap(unsigned long long c, long long step, unsigned long long extra)
{
    return (c + 8) * (unsigned long long)step + (unsigned long long)(long long)(6.0 * std::sqrt((double)c) * (double)step) + 1 +
           extra;
}

void layout_sampled(const std::vector<unsigned long long>& sc, long long step, int64_t n, int C, int sub, RJLayout& L,
                    bool pack, bool model)
{
    layout_tiles(L, n, C, pack, model);
    const size_t F = sc.size();
    L.sampled = true;
    L.packed = pack;
    auto sz = [&](unsigned long long c) { return pack ? (c + 1) & ~1ULL : c; };
    L.fcap.assign(F, 0);
    L.fstart.assign(F + 1, 0);
    for (size_t f = 0; f < F; ++f) {
        L.fcap[f] = sz(sampled_cap(sc[f], step, 64));
        L.fstart[f + 1] = L.fstart[f] + L.fcap[f];
    }
    L.ccap.assign(C, 0);
    L.cstart.assign(C + 1, 0);
    L.tiles2_max = 0;
    for (int c = 0; c < C; ++c) {
        unsigned long long cc = 0;
        for (size_t f = (size_t)c << sub; f < (size_t)(c + 1) << sub; ++f) cc += sc[f];
        L.ccap[c] = sz(sampled_cap(cc, step, 1024));
        L.cstart[c + 1] = L.cstart[c] + L.ccap[c];
        L.tiles2_max += (L.ccap[c] + L.tile2 - 1) / L.tile2;
    }
    L.tiles2.clear();
    L.count.clear();
    L.p1 = L.cstart[C];
    L.p2 = L.fstart[F];
}

// A window [base, base + 2^32 - 1) centred on [lo, hi] (offset 2^32 - 1 is
// never used, so a join can take it as its empty-slot marker); a sampled
// range must leave at least 2^30 of margin on each side.
static bool frame_fit(long long lo, long long hi, bool exact, unsigned long long& base)
{
    if (hi < lo) {  // nothing was read
        base = 0;
        return true;
    }
    const unsigned long long span = (unsigned long long)hi - (unsigned long long)lo;
    if (span > (exact ? 0xFFFFFFFEULL : (1ULL << 31))) return false;
    base = (unsigned long long)lo - (0xFFFFFFFEULL - span) / 2;
    return true;
}

bool pack_frame(long long kmin, long long kmax, long long pmin, long long pmax, bool exact, RJLayout& L,
                const unsigned long long* key_base)
{
    unsigned long long kb = 0, pb = 0;
    if (key_base) {
        kb = *key_base;  // a frame shared with another relation, fitted to both ranges
    } else if (!frame_fit(kmin, kmax, exact, kb)) {
        return false;
    }
    if (!frame_fit(pmin, pmax, exact, pb)) return false;
    L.kbase = kb;
    L.pbase = pb;
    return true;
}

bool common_key_frame(const long long* mm0, bool exact0, const long long* mm1, bool exact1, unsigned long long* base)
{
    if (mm0[1] < mm0[0] || mm1[1] < mm1[0]) return false;
    const long long lo = std::min(mm0[0], mm1[0]), hi = std::max(mm0[1], mm1[1]);
    return frame_fit(lo, hi, exact0 && exact1, *base);
}

int upload_layout(pyg_ctx* ctx, const RJLayout& L, const RJSideDev& d, int F, int C, int64_t n)
{
    // fstart, fcap, cstart and ccap are adjacent on the device, and so are
    // tiles2 and whole: two copies.
    int rc;
    std::vector<unsigned long long> m((size_t)(F + 1) + F + (C + 1) + C, 0);
    unsigned long long* p = m.data();
    memcpy(p, L.fstart.data(), (size_t)(F + 1) * 8);
    if (L.sampled) memcpy(p + F + 1, L.fcap.data(), (size_t)F * 8);
    memcpy(p + 2 * F + 1, L.cstart.data(), (size_t)(C + 1) * 8);
    if (L.sampled || L.packed) memcpy(p + 2 * F + C + 2, L.ccap.data(), (size_t)C * 8);
    if ((rc = stage_h2d(ctx, d.fstart, p, m.size() * 8))) return rc;
    std::vector<unsigned long long> t((size_t)(C + 1) + 4, 0);
    if (!L.sampled && !L.packed) memcpy(t.data(), L.tiles2.data(), (size_t)(C + 1) * 8);
    t[C + 2] = (unsigned long long)n;
    t[C + 4] = (unsigned long long)((n + L.tile1 - 1) / L.tile1);
    if ((rc = stage_h2d(ctx, d.tiles2, t.data(), t.size() * 8))) return rc;
    PYG_CUDA(cudaMemsetAsync(d.cur1, 0, ((size_t)C * RJ_CURSOR_STRIDE + F) * 8, ctx->stream));  // cur1 and cur2 are adjacent
    return PYG_OK;
}

// Runs the partition pass(es) of one relation into P1 (and P2).
int run_passes(pyg_ctx* ctx, const longlong2* in, int64_t n, const RJLayout& L, const RJSideDev& d, bool two, int FB,
               int CB, void* P1, void* P2, unsigned* err, unsigned* ovf, const long long* csplit,
               const long long* fsplit, unsigned* frame, cudaEvent_t between, const RJModel* model)
{
    const int C = 1 << CB, sub = FB - CB;
    if (L.packed && (!frame || (two && sub > 8))) {
        set_error("partition: packed layouts need a frame flag and at most 2^8 second-pass bins");
        return PYG_ERR_ARG;
    }
    RJPass p;
    memset(&p, 0, sizeof(p));
    p.in = in;
    p.out = (longlong2*)P1;
    p.seg_start = d.whole;
    p.seg_tile0 = d.wtiles;
    p.nseg = 1;
    p.tile = L.tile1;
    p.shift = 64 - CB;
    p.mask = (unsigned)(C - 1);
    p.lbits = CB;
    p.bin_start = two ? d.cstart : d.fstart;
    p.bin_cap = L.sampled ? (two ? d.ccap : d.fcap) : nullptr;
    p.cursor = d.cur1;
    p.cstride = RJ_CURSOR_STRIDE;
    p.dump = two ? L.p1 : L.p2;
    p.err = err;
    p.ovf = ovf;
    p.kbase = L.kbase;
    p.pbase = L.pbase;
    p.frame = frame;
    if (model) p.model = *model;
    if (csplit) {
        p.split = csplit;
        p.nsplit = C - 1;
    }
    int rc = launch_pass(ctx, p, (n + L.tile1 - 1) / L.tile1, false, L.packed);
    if (rc || !two) return rc;
    if (between) cudaEventRecord(between, ctx->stream);
    long long ntiles2;
    if (L.sampled || L.packed) {
        // Second-pass segments are the first pass's regions, filled to the
        // counts its cursors reached; the tile prefix is formed on the device.
        rj_tile_prefix_kernel<<<1, RJ_LMAX, 0, ctx->stream>>>(d.cur1, RJ_CURSOR_STRIDE, d.count1, d.ccap, C,
                                                          L.tile2, d.tiles2);
        PYG_LAUNCHED(ctx);
        p.seg_count = d.count1;
        p.ntiles_dev = d.tiles2 + C;
        ntiles2 = (long long)L.tiles2_max;
    } else {
        ntiles2 = (long long)L.tiles2[C];
    }
    p.in = (const longlong2*)P1;
    p.out = (longlong2*)P2;
    p.seg_start = d.cstart;
    p.seg_tile0 = d.tiles2;
    p.nseg = C;
    p.tile = L.tile2;
    p.shift = 64 - FB;
    p.mask = (unsigned)((1 << sub) - 1);
    p.lbits = sub;
    p.bin_start = d.fstart;
    p.bin_cap = L.sampled ? d.fcap : nullptr;
    p.cursor = d.cur2;
    p.cstride = 1;
    p.dump = L.p2;
    if (fsplit) {
        p.split = fsplit;
        p.nsplit = (1 << sub) - 1;
    }
    return launch_pass(ctx, p, ntiles2, L.packed, L.packed);
}

int hist_launch(pyg_ctx* ctx, const longlong2* in, int64_t n, int64_t step, int spread, int FB, unsigned long long* hist,
                long long* mm, const RJModel* model)
{
    // At most 2^15 counters (128 KB) per launch: 2^16 bins take two.
    const int F = 1 << FB, span = F < (1 << 15) ? F : (1 << 15);
    const size_t hsm = (size_t)4 * span;
    auto kern = model ? rj_hist_kernel<true> : rj_hist_kernel<false>;
    const RJModel none;
    // The most that any call needs: the attribute is the process's, and a call
    // on another thread may launch the kernel between these lines.
    PYG_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 4 << 15));
    int per = 0;
    PYG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kern, 1024, hsm));
    if (per < 1) per = 1;
    const int64_t m = (n + step - 1) / step;
    const int64_t want = (m + 1024 * 8 - 1) / (1024 * 8);
    const int grid = (int)std::max<int64_t>(1, std::min<int64_t>(want, (int64_t)ctx->sm_count * per));
    unsigned* part = nullptr;
    int rc;
    if ((rc = dalloc(ctx, (void**)&part, (size_t)grid * span * 4))) return rc;
    if (mm) {
        rj_mm_init_kernel<<<1, 32, 0, ctx->stream>>>(mm);
        PYG_LAUNCHED(ctx);
    }
    for (int base = 0; base < F; base += span) {
        // The key and payload ranges are taken in the first launch only.
        kern<<<grid, 1024, hsm, ctx->stream>>>(in, n, step, spread, FB, base, span, part, base ? nullptr : mm,
                                                model ? *model : none);
        PYG_LAUNCHED(ctx);
        rj_hist_sum_kernel<<<(span + 255) / 256, 256, 0, ctx->stream>>>(part, grid, span, hist + base);
        PYG_LAUNCHED(ctx);
    }
    dfree(ctx, part);
    return PYG_OK;
}

int hist_launch_range(pyg_ctx* ctx, const longlong2* in, int64_t n, int64_t step, int spread, int CB, int sub,
                      const long long* csplit, const long long* fsplit, unsigned long long* hist, long long* mm)
{
    const int F = 1 << (CB + sub);
    const size_t hsm = (size_t)RJ_SPLIT_MAX * 8 + (size_t)4 * F;
    PYG_CUDA(cudaFuncSetAttribute(rj_hist_range_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  RJ_SPLIT_MAX * 8 + (4 << RJ_MAX_RANGE_BITS)));  // as in hist_launch
    int per = 0;
    PYG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, rj_hist_range_kernel, 1024, hsm));
    if (per < 1) per = 1;
    const int64_t m = (n + step - 1) / step;
    const int64_t want = (m + 1024 * 8 - 1) / (1024 * 8);
    const int grid = (int)std::max<int64_t>(1, std::min<int64_t>(want, (int64_t)ctx->sm_count * per));
    unsigned* part = nullptr;
    int rc;
    if ((rc = dalloc(ctx, (void**)&part, (size_t)grid * F * 4))) return rc;
    if (mm) {
        rj_mm_init_kernel<<<1, 32, 0, ctx->stream>>>(mm);
        PYG_LAUNCHED(ctx);
    }
    rj_hist_range_kernel<<<grid, 1024, hsm, ctx->stream>>>(in, n, step, spread, CB, sub, csplit, fsplit, part, mm);
    PYG_LAUNCHED(ctx);
    rj_hist_sum_kernel<<<(F + 255) / 256, 256, 0, ctx->stream>>>(part, grid, F, hist);
    PYG_LAUNCHED(ctx);
    dfree(ctx, part);
    return PYG_OK;
}

int rp_partition_sides(pyg_ctx* ctx, RPSide* sd, int ns, int FB, bool two, unsigned* flags, unsigned* hflags,
                       cudaEvent_t hist_done, bool share_key_frame, const RPAfter* after)
{
    // Coarse bits of the first of two passes.  Unpacked layouts split FB
    // evenly; packed layouts keep the second pass at 2^8 bins, so that its
    // tiles use one-byte bin indexes and write runs of about 20 words.  The unpacked split has at least
    // as many coarse partitions, so its metadata size covers both.
    auto coarse_bits = [&](bool packed) { return !two ? FB : (packed ? std::max(1, FB - 8) : (FB + 1) / 2); };
    const int F = 1 << FB;
    const size_t side = RJSideDev::words(F, 1 << coarse_bits(false));
    const size_t per = side + F + 4;  // metadata, histogram, {kmin, kmax, pmin, pmax}
    // Host words per relation: the histogram and the ranges, or the cursors
    // that hold a sampled relation's counts.
    const size_t hper = std::max<size_t>(F, two ? 0 : (size_t)F * RJ_CURSOR_STRIDE) + 4;
    if (ns < 1 || ns > 2 || (size_t)ns * hper * 8 > kPinnedStageBytes) {
        set_error("partition: %d relations of 2^%d partitions exceed the staging area", ns, FB);
        return PYG_ERR_ARG;
    }
    // Per-partition counts come back through pinned memory, so that both
    // relations' histograms cost one host round trip and both relations'
    // passes another.
    unsigned long long* hh = (unsigned long long*)((char*)ctx->pinned + kPinnedScalarBytes);
    unsigned long long* meta = nullptr;
    RJSideDev d[2];
    int CBs[2] = {FB, FB};
    bool sample[2] = {false, false};
    int rc = PYG_OK;
    for (int s = 0; s < ns; ++s) sd[s].P1 = sd[s].P2 = nullptr;
    auto hist_at = [&](int s) { return meta + (size_t)s * per + side; };
    auto hh_at = [&](int s) { return hh + (size_t)s * hper; };
    auto hist_of = [&](int s, int64_t st) {
        if (sd[s].csplit) {
            const int cb = coarse_bits(false);
            return hist_launch_range(ctx, sd[s].in, sd[s].n, st, two ? 2 : 1, cb, FB - cb, sd[s].csplit, sd[s].fsplit, hist_at(s),
                                     sd[s].allow_pack ? (long long*)(hist_at(s) + F) : nullptr);
        }
        return hist_launch(ctx, sd[s].in, sd[s].n, st, two ? 2 : 1, FB, hist_at(s),
                           sd[s].allow_pack ? (long long*)(hist_at(s) + F) : nullptr, sd[s].model);
    };
    // Layout of relation s from host counts h (F counts, then the key and
    // payload ranges): packed when the caller allows it and a frame fits.
    auto form = [&](int s, const unsigned long long* h, int64_t st, bool exact, const unsigned long long* kb) {
        RJLayout& L = sd[s].L;
        const long long* mm = (const long long*)(h + F);
        const bool pack = sd[s].allow_pack && pack_frame(mm[0], mm[1], mm[2], mm[3], exact, L, kb);
        CBs[s] = coarse_bits(pack && !sd[s].csplit);  // the coarse splitters fix the split of range bins
        const int C = 1 << CBs[s], sub = FB - CBs[s];
        std::vector<unsigned long long> hv(h, h + F);
        if (exact) layout_exact(hv, sd[s].n, C, sub, L, pack, sd[s].model || sd[s].csplit);
        else layout_sampled(hv, st, sd[s].n, C, sub, L, pack, sd[s].model || sd[s].csplit);
        d[s].carve(meta + (size_t)s * per, F, C);
    };
    auto launch = [&](int s) {
        const RJLayout& L = sd[s].L;
        int r;
        if ((r = upload_layout(ctx, L, d[s], F, 1 << CBs[s], sd[s].n))) return r;
        dfree(ctx, sd[s].P1);
        dfree(ctx, sd[s].P2);
        sd[s].P1 = sd[s].P2 = nullptr;
        if ((r = dalloc(ctx, &sd[s].P1, pass_bytes(L, L.p1)))) return r;
        if (two && (r = dalloc(ctx, &sd[s].P2, pass_bytes(L, L.p2)))) return r;
        if (sd[s].begin) cudaEventRecord(sd[s].begin, ctx->stream);
        if ((r = run_passes(ctx, sd[s].in, sd[s].n, L, d[s], two, FB, CBs[s], sd[s].P1, sd[s].P2, flags + 4 * s,
                            flags + 4 * s + 1, sd[s].csplit, sd[s].fsplit, flags + 4 * s + 2, sd[s].mid,
                            sd[s].model)))
            return r;
        if (sd[s].done) cudaEventRecord(sd[s].done, ctx->stream);
        return PYG_OK;
    };
    // Relation s's layout from an exact histogram (one host round trip).
    auto form_exact = [&](int s) -> int {
        int r = hist_of(s, 1);
        if (r) return r;
        PYG_CUDA(cudaMemcpyAsync(hh_at(s), hist_at(s), (size_t)(F + 4) * 8, cudaMemcpyDeviceToHost, ctx->stream));
        PYG_CUDA(cudaStreamSynchronize(ctx->stream));
        form(s, hh_at(s), 1, true, nullptr);
        return PYG_OK;
    };
    do {
        if ((rc = dalloc(ctx, (void**)&meta, per * 8 * ns))) break;
        PYG_CUDA(cudaMemsetAsync(flags, 0, (size_t)16 * ns, ctx->stream));
        int64_t step[2] = {1, 1};
        for (int s = 0; s < ns && !rc; ++s) {
            sample[s] = sd[s].allow_sample && sd[s].n >= ((int64_t)1 << 25);
            step[s] = sample[s] ? std::max<int64_t>(1, sd[s].n >> rj_sample_log2(FB)) : 1;
            if ((rc = hist_of(s, step[s]))) break;
            sd[s].hist_tuples = (sd[s].n + step[s] - 1) / step[s];
        }
        if (rc) break;
        if (hist_done) cudaEventRecord(hist_done, ctx->stream);
        for (int s = 0; s < ns; ++s)
            PYG_CUDA(cudaMemcpyAsync(hh_at(s), hist_at(s), (size_t)(F + 4) * 8, cudaMemcpyDeviceToHost, ctx->stream));
        PYG_CUDA(cudaStreamSynchronize(ctx->stream));
        stage_reset(ctx);
        // One key frame for both relations when asked and both ranges fit
        // in it, so that their packed words compare by key offset.
        unsigned long long ckb = 0;
        const bool common = share_key_frame && ns == 2 && sd[0].allow_pack && sd[1].allow_pack && !sd[0].csplit &&
                            !sd[1].csplit &&
                            common_key_frame((const long long*)(hh_at(0) + F), !sample[0],
                                             (const long long*)(hh_at(1) + F), !sample[1], &ckb);
        // The second relation's layout is formed while the first one's
        // passes run.
        for (int s = 0; s < ns && !rc; ++s) {
            form(s, hh_at(s), step[s], !sample[s], common ? &ckb : nullptr);
            rc = launch(s);
            // Not enough memory for a sampled layout's slack (a fifth of the
            // relation with about 2^9 samples per partition): exact regions.
            if (rc == PYG_ERR_OOM && sd[s].L.sampled && !(rc = form_exact(s))) rc = launch(s);
        }
        if (rc) break;
        PYG_CUDA(cudaMemcpyAsync(hflags, flags, (size_t)16 * ns, cudaMemcpyDeviceToHost, ctx->stream));
        if (after) {
            RPDev dev[2];
            for (int s = 0; s < ns; ++s) {
                dev[s].start = d[s].fstart;
                dev[s].count = two ? d[s].cur2 : d[s].cur1;
                dev[s].stride = two ? 1 : RJ_CURSOR_STRIDE;
            }
            if ((rc = after->enqueue(dev))) break;
            PYG_CUDA(cudaStreamSynchronize(ctx->stream));
            if (after->settled()) break;
        }
        for (int s = 0; s < ns; ++s)
            if (sd[s].L.sampled)
                PYG_CUDA(cudaMemcpyAsync(hh_at(s), two ? d[s].cur2 : d[s].cur1,
                                         (size_t)F * 8 * (two ? 1 : RJ_CURSOR_STRIDE), cudaMemcpyDeviceToHost,
                                         ctx->stream));
        PYG_CUDA(cudaStreamSynchronize(ctx->stream));
        for (int s = 0; s < ns && !rc; ++s) {
            if (hflags[4 * s]) {
                set_error("partition: a tile copy did not complete in time");
                rc = PYG_ERR_TIMEOUT;
                break;
            }
            if (sd[s].L.sampled) {
                sd[s].L.count.resize(F);
                for (int f = 0; f < F; ++f) sd[s].L.count[f] = hh_at(s)[(size_t)f * (two ? 1 : RJ_CURSOR_STRIDE)];
            }
            if (!hflags[4 * s + 1] && !hflags[4 * s + 2]) continue;
            // A sampled region overflowed, or a tuple fell outside a frame
            // taken from the sample: redo this relation from an exact
            // histogram, whose key and payload ranges are exact too (exact
            // regions cannot overflow, and an exact frame misses nothing).
            sd[s].overflowed = true;
            sd[s].done = sd[s].begin = sd[s].mid = nullptr;  // the redo's time is not attributed to the relation
            if ((rc = form_exact(s))) break;
            PYG_CUDA(cudaMemsetAsync(flags + 4 * s, 0, 16, ctx->stream));
            if ((rc = launch(s))) break;
            PYG_CUDA(cudaMemcpyAsync(hflags + 4 * s, flags + 4 * s, 16, cudaMemcpyDeviceToHost, ctx->stream));
            PYG_CUDA(cudaStreamSynchronize(ctx->stream));
            if (hflags[4 * s]) {
                set_error("partition: a tile copy did not complete in time");
                rc = PYG_ERR_TIMEOUT;
            } else if (hflags[4 * s + 1] || hflags[4 * s + 2]) {
                set_error("partition: an exact layout overflowed a region or missed its frame");
                rc = PYG_ERR_CAPACITY;
            }
        }
    } while (0);
    dfree(ctx, meta);
    if (rc) {
        for (int s = 0; s < ns; ++s) {
            dfree(ctx, sd[s].P1);
            dfree(ctx, sd[s].P2);
            sd[s].P1 = sd[s].P2 = nullptr;
        }
    }
    return rc;
}

}  // namespace pyg
