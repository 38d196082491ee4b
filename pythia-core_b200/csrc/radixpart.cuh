// Hash partitioning of 16-byte (int64 key, int64 payload) tuples by the
// top bits of a multiplicative hash of the key, shared by the radix
// operators (join, group-by).
//
//   histogram   rj_hist_kernel counts the top `bits` bits of every tuple (or
//               of a sample of the rows) in shared memory.
//   layout      exact (dense partitions from a full histogram) or sampled
//               (regions sized from the sample with six standard deviations
//               of slack; a region that overflows is reported and the caller
//               redoes the side exactly).
//   passes      one tile pass (<= 9 bits) or two (coarse bits, then the rest
//               inside each coarse partition).  A CTA receives tiles of a few
//               thousand tuples by bulk copy, groups a tile by bin in shared
//               memory and writes each bin's run contiguously after one
//               global reservation per (tile, bin).
//   packing     (callers that opt in) when the histogram's reading of the
//               relation shows that key - kbase and payload - pbase both
//               fit in 32 bits for some frame (kbase, pbase), the passes
//               write 8-byte words (key - kbase) | (payload - pbase) << 32
//               instead of 16-byte tuples: frame-of-reference encoding,
//               exact, and half the bytes of every intermediate write and
//               re-read.  A tuple outside the frame (possible when the
//               histogram read a sample) sets a flag and the relation is
//               redone with 16-byte intermediates.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <functional>
#include <vector>

#include "pyg_internal.cuh"

typedef struct pyg_cdf pyg_cdf;

namespace pyg {

// Largest tiles (elements) of a partition pass by what it reads and writes
// (the kernels' shapes are in radixpart.cu).
constexpr int RJ_TILE_U = 2688;    // 16-byte tuples in and out: hash bins
constexpr int RJ_TILE_UM = 2400;   //   model and range bins
constexpr int RJ_TILE_P = 7936;    // 16-byte tuples in, packed words out: hash bins
constexpr int RJ_TILE_P9 = 7680;   //   hash bins, more than 2^8
constexpr int RJ_TILE_PM = 3968;   //   model and range bins
constexpr int RJ_TILE_8 = 5376;    // packed words in and out: hash bins
constexpr int RJ_TILE_8M = 4800;   //   model and range bins
// Largest model whose tables a first pass keeps in shared memory.
constexpr int RJ_SM_LEAVES = 1024;
constexpr int RJ_SM_HEAVY = 512;
constexpr int RJ_TILE_MIN = 1024;
// Tile of a pass over n elements: the largest, halved until a pass has about
// two tiles for each of the 148 SMs (small relations would otherwise leave
// SMs without a tile).
constexpr int64_t RJ_TILES_MIN = 2 * 148;
inline int rj_tile(int largest, int64_t n)
{
    int t = largest;
    while (t > RJ_TILE_MIN && n < t * RJ_TILES_MIN) t = (t >> 1) & ~1;  // even: tiles of packed words start 16-byte aligned
    return t;
}
constexpr int RJ_MAX_LOCAL_BITS = 9;     // bins of one partition pass
constexpr int RJ_LMAX = 1 << RJ_MAX_LOCAL_BITS;
constexpr int RJ_SPLIT_MAX = 256;        // range mode: splitters per pass segment (<= 2^8 bins)
// Largest fine partition counts (log2); the histogram kernels keep up to
// 2^15 32-bit counters in shared memory.
constexpr int RJ_MAX_FINE_BITS = 16;   // hash mode (histograms run in halves above 2^15 bins)
constexpr int RJ_MAX_RANGE_BITS = 15;  // range mode (one 2^15-counter histogram)
// Sampled layouts count one tuple in every n >> rj_sample_log2: about 2^9
// samples per partition, at most 2^22 (0.1 ms per relation; a sample costs a
// 32-byte sector, 78 us for 2^22 of 2^27 tuples against 12 us for 2^17).
// Fewer samples give regions more slack, which costs device memory, not
// traffic.
inline int rj_sample_log2(int FB) { return FB < 8 ? 17 : (FB > 13 ? 22 : FB + 9); }

// Partition bins computed by a learned CDF model instead of a search
// (range partitioning without splitters in the passes).  For a model with
// L leaves over keys (kmin, kmax) and 2^fbits bins:
//   x = (float)(k - kmin) * scale                     normalised key (the
//                                                     offset as unsigned)
//   r = a0 x + b0, l = clamp(floor(L r), 0, L - 1)     root line -> leaf
//   u = clamp(L r - l, 0, 1)                           leaf-local coordinate
//   g = clamp(A_l u + B_l, lo_l, hi_l)                 the leaf's line
//   g = min(g + (masses of the leaf's heavy keys below k), hi_l)
//   bin(k) = min(2^fbits - 1, trunc(g 2^fbits))
// with bin 0 for k <= kmin and the last bin for k >= kmax.  Every step is a
// correctly rounded fp32 operation that does not decrease when its input
// grows (A_l and the masses are >= 0), and hi_l <= lo_{l+1}, so bin(k)
// never decreases with k: the bins are key ranges, and their splitters
// (the first key of each bin, found by bisection over the same function)
// reproduce them exactly.  The model's accuracy only decides how even the
// bins are.
struct RJLeaf {
    float A, B;    // the leaf's line over u
    float lo, hi;  // its range of g
};
struct RJModel {
    const RJLeaf* leaf = nullptr;  // device, L leaves (null: no model)
    const int2* hinfo = nullptr;   // device, per leaf {first heavy key, count}; null without heavy keys
    const long long* hkey = nullptr;  // device, heavy keys ascending
    const float* hw = nullptr;        // device, their masses
    long long kmin = 0, kmax = 0;
    float scale = 0;
    float a0 = 0, b0 = 0;
    int L = 0;
    int H = 0;  // heavy keys
    int fbits = 0;
};

__device__ __forceinline__ unsigned rj_model_bin(const RJModel& m, long long k)
{
    const unsigned last = (1u << m.fbits) - 1u;
    if (k <= m.kmin) return 0u;
    if (k >= m.kmax) return last;
    const float x = __fmul_rn(__ull2float_rn((unsigned long long)k - (unsigned long long)m.kmin), m.scale);
    const float lr = __fmul_rn(__fmaf_rn(m.a0, x, m.b0), (float)m.L);
    const float fl = floorf(lr);
    const int l = fl < 0.f ? 0 : (fl > (float)(m.L - 1) ? m.L - 1 : (int)fl);
    const float u = fminf(1.f, fmaxf(0.f, __fsub_rn(lr, (float)l)));
    const RJLeaf p = m.leaf[l];
    float g = fminf(p.hi, fmaxf(p.lo, __fmaf_rn(p.A, u, p.B)));
    if (m.hinfo) {
        const int2 hi = m.hinfo[l];
        for (int h = hi.x; h < hi.x + hi.y && m.hkey[h] < k; ++h) g = __fadd_rn(g, m.hw[h]);
        g = fminf(g, p.hi);
    }
    const float b = __fmul_rn(g, (float)(1u << m.fbits));
    return b >= (float)last ? last : (unsigned)b;
}

// Bins of a trained CDF model (cdf.cu): *out refers to device tables the
// model keeps until pyg_cdf_free.  model_splitters: the 2^fbits - 1
// splitters of those bins into host array out (bin(k) = number of
// splitters <= k).
int cdf_bin_model(pyg_ctx* ctx, const pyg_cdf* m, int fbits, RJModel* out);
int model_splitters(pyg_ctx* ctx, const RJModel& m, int64_t* out);

// The 64-bit code whose top fbits bits are the model's bin (the hash
// operators take their partition bits from the top of such a word).
__device__ __forceinline__ uint64_t rj_model_code(const RJModel& m, long long k)
{
    return (uint64_t)rj_model_bin(m, k) << (64 - m.fbits);
}

// Host-side layout of one relation's partitions.
struct RJLayout {
    bool sampled = false;
    // Packed (8-byte) intermediates and their frame: key = kbase + low 32
    // bits, payload = pbase + high 32 bits (64-bit wrap-around arithmetic).
    // Packed layouts start every region at an even word, so that each
    // region's tiles begin 16-byte aligned for bulk copies.
    bool packed = false;
    unsigned long long kbase = 0, pbase = 0;
    std::vector<unsigned long long> fstart;  // F + 1 fine region starts
    std::vector<unsigned long long> fcap;    // F fine region capacities (sampled)
    std::vector<unsigned long long> cstart;  // C + 1 coarse region starts
    std::vector<unsigned long long> ccap;    // C coarse region capacities (sampled)
    std::vector<unsigned long long> tiles2;  // C + 1 tile prefix of the second pass (exact)
    std::vector<unsigned long long> count;   // F tuples per fine partition, once known
    unsigned long long p1 = 0, p2 = 0;       // tuples in the pass-1 / pass-2 buffers
    int tile1 = 0, tile2 = 0;                // elements per tile of either pass
    unsigned long long tiles2_max = 0;       // upper bound of the second pass's tiles (sampled)
};

// Exact layout of n tuples from exact per-fine-partition counts h (F = h.size()).
// pack: regions rounded up to an even number of words (packed layouts).
// model: the passes' bins are a learned model's or key ranges.
void layout_exact(const std::vector<unsigned long long>& h, int64_t n, int C, int sub, RJLayout& L,
                  bool pack = false, bool model = false);
// Sampled layout from the counts sc of one tuple in every `step`: each region is
// sized with six standard deviations of slack.
void layout_sampled(const std::vector<unsigned long long>& sc, long long step, int64_t n, int C, int sub, RJLayout& L,
                    bool pack = false, bool model = false);
// Frame of a packed layout from the key and payload ranges seen by the
// histogram ([kmin, kmax], [pmin, pmax], signed).  exact: the ranges cover
// every tuple; else they come from a sample and must leave a margin of at
// least 2^30 on each side.  Key offsets stay below 2^32 - 1: an exact frame
// ends there, and a pass reports a tuple that a sampled frame put there or
// beyond as a frame miss.  key_base (when
// given) is a key frame shared with another relation (common_key_frame).
// Returns false when no frame fits.
bool pack_frame(long long kmin, long long kmax, long long pmin, long long pmax, bool exact, RJLayout& L,
                const unsigned long long* key_base = nullptr);
// One key frame covering two relations' key ranges mm = {kmin, kmax, ...},
// so that their packed words carry comparable 32-bit key offsets.
bool common_key_frame(const long long* mm0, bool exact0, const long long* mm1, bool exact1, unsigned long long* base);
// Bytes of one intermediate element of a layout.
inline int elem_bytes(const RJLayout& L) { return L.packed ? 8 : 16; }

// The first pass's cursors lie 128 bytes apart: 64-bit atomics on one line
// are served one after another, and a tile's reservations are otherwise a
// few lines that every CTA hits at once.
constexpr int RJ_CURSOR_STRIDE = 16;

// Device copy of one relation's partition metadata (u64 words).
struct RJSideDev {
    unsigned long long *fstart, *fcap, *cstart, *ccap, *cur1, *cur2, *count1, *tiles2, *whole, *wtiles;
    static size_t words(int F, int C)
    {
        return (size_t)(F + 1) + F + (C + 1) + C + (size_t)C * RJ_CURSOR_STRIDE + F + C + (C + 1) + 4;
    }
    void carve(unsigned long long* m, int F, int C)
    {
        fstart = m;
        fcap = fstart + F + 1;
        cstart = fcap + F;
        ccap = cstart + C + 1;
        cur1 = ccap + C;
        cur2 = cur1 + (size_t)C * RJ_CURSOR_STRIDE;
        count1 = cur2 + F;
        tiles2 = count1 + C;
        whole = tiles2 + C + 1;
        wtiles = whole + 2;
    }
};

// Copies a layout to the device and zeroes its cursors.
int upload_layout(pyg_ctx* ctx, const RJLayout& L, const RJSideDev& d, int F, int C, int64_t n);
// Histogram of the top FB hash bits of one tuple in every `step` (at a
// multiple of `spread` inside it, rj_sample_row) into hist
// (2^FB device words, zeroed here).  mm (optional, 4 words): receives the
// minimum and maximum key and payload of the tuples read, as signed
// {kmin, kmax, pmin, pmax}.
int hist_launch(pyg_ctx* ctx, const longlong2* in, int64_t n, int64_t step, int spread, int FB, unsigned long long* hist,
                long long* mm = nullptr, const RJModel* model = nullptr);
// Partition pass(es) of one relation into P1 (and P2 when two): *err is set
// if a tile's bulk copy never landed, *ovf if a sampled region overflowed,
// *frame if a tuple fell outside a packed layout's frame.  After two passes
// d.cur2 holds the tuples written per fine partition; after one, d.cur1 at
// RJ_CURSOR_STRIDE words each.
// Range mode when csplit is set: pass 1 bins by the 2^CB - 1 coarse
// splitters, pass 2 by the fine splitters (F - 1, ascending; coarse
// splitter i = fine splitter (i + 1) * 2^(FB - CB) - 1).
int run_passes(pyg_ctx* ctx, const longlong2* in, int64_t n, const RJLayout& L, const RJSideDev& d, bool two, int FB,
               int CB, void* P1, void* P2, unsigned* err, unsigned* ovf, const long long* csplit = nullptr,
               const long long* fsplit = nullptr, unsigned* frame = nullptr, cudaEvent_t between = nullptr,
               const RJModel* model = nullptr);
// Elements past a pass buffer's last region: the runs of bins that outgrow
// their sampled region go there (at most one tile at a time per CTA; nothing
// reads them), and a last tile's copy of packed words, rounded up to 16
// bytes, stays inside the buffer.
constexpr int RJ_DUMP = 8192;
static_assert(RJ_DUMP >= RJ_TILE_U && RJ_DUMP >= RJ_TILE_UM && RJ_DUMP >= RJ_TILE_P && RJ_DUMP >= RJ_TILE_P9 &&
                  RJ_DUMP >= RJ_TILE_PM && RJ_DUMP >= RJ_TILE_8 && RJ_DUMP >= RJ_TILE_8M,
              "a run is at most a tile");
// Device bytes of a layout's pass buffer of `words` elements.
inline size_t pass_bytes(const RJLayout& L, unsigned long long words)
{
    return ((size_t)words + RJ_DUMP) * elem_bytes(L);
}
// Histogram of range bins (see run_passes) of one tuple in every `step`.
int hist_launch_range(pyg_ctx* ctx, const longlong2* in, int64_t n, int64_t step, int spread, int CB, int sub,
                      const long long* csplit, const long long* fsplit, unsigned long long* hist,
                      long long* mm = nullptr);
// One relation for rp_partition_sides.  In: in, n, allow_sample, the
// splitters (range mode) and an optional event recorded after the
// relation's passes.  Out: the layout (counts included), the pass buffers
// (the caller frees them), the tuples its histogram read and whether a
// sampled region overflowed (then the relation was redone exactly).
struct RPSide {
    const longlong2* in = nullptr;
    int64_t n = 0;
    bool allow_sample = true;
    bool allow_pack = false;  // the caller reads packed intermediates (L.packed tells)
    const long long* csplit = nullptr;
    const long long* fsplit = nullptr;
    // Learned-model bins (rj_model_bin) instead of hash bits; model->fbits
    // must equal the partition bits.
    const RJModel* model = nullptr;
    cudaEvent_t begin = nullptr;  // recorded before the first pass (optional)
    cudaEvent_t mid = nullptr;    // between the two passes (optional)
    cudaEvent_t done = nullptr;
    RJLayout L;
    void* P1 = nullptr;
    void* P2 = nullptr;
    int64_t hist_tuples = 0;
    bool overflowed = false;
};

// One relation's partitions on the device, valid in stream order: partition
// f starts at start[f] and holds count[f * stride] elements (more than its
// region holds if it overflowed: the relation's flags then say so).
struct RPDev {
    const unsigned long long* start;
    const unsigned long long* count;
    int stride;
};

// What a caller does with the partitions before the host has seen their
// counts: enqueue launches it behind the passes (its kernels must do nothing
// when a relation's flags are set), settled is asked after the stream was
// synchronised and the flags are on the host; true: the answer stands, and
// the counts and the redo are not needed.
struct RPAfter {
    std::function<int(const RPDev*)> enqueue;
    std::function<bool()> settled;
};

// Partitions one or two relations with the same bits: both histograms, one
// host round trip, both relations' passes (the second relation's layout is
// formed while the first one's passes run), one more round trip for the
// counts and flags, and an exact redo of a relation whose sampled region
// overflowed or whose packed frame missed a tuple (the redo is packed again
// where the exact ranges fit a frame).  A sampled layout whose slack does not
// fit in device memory is replaced by an exact one.
// flags: 4 device words per relation (bulk copy never landed, region
// overflow, frame miss, unused); hflags: as many pinned host words.
// hist_done (optional) is recorded after the histograms.
// share_key_frame: pack both relations with one key frame when their key
// ranges fit one (a redone relation gets its own frame).
// after (optional): work on the partitions that needs no host round trip.
int rp_partition_sides(pyg_ctx* ctx, RPSide* sd, int ns, int FB, bool two, unsigned* flags, unsigned* hflags,
                       cudaEvent_t hist_done, bool share_key_frame = false, const RPAfter* after = nullptr);

// Hash of the radix operators: multiplication by 2^64 / golden ratio
// (Fibonacci hashing) after three xor-shifts.  Bit j of the product depends
// on bits 0..j of the shifted key, so the top bits mix the whole key:
// partitions take the top `fb` bits and shared-memory tables the 32 bits
// below them.  Dense key ranges spread almost evenly over the partitions
// and over the slots of a partition's table (consecutive multiples of an
// irrational fraction; the xor-shifts permute aligned blocks of 2^16 keys
// onto themselves, so a dense range keeps this).  Without the xor-shifts,
// keys that are multiples of 2^16 or of a Fibonacci number (987, 1597, ...)
// see the product's weaker lower bits and pile into long probe chains
// (30-110 probes per insert at a third of the table instead of about 1.3);
// with these three shifts, strides, Fibonacci multiples and packed
// (a << s) | b keys stay at 1.0-2.1.
constexpr uint64_t kRjHashMul = 0x9E3779B97F4A7C15ULL;
__host__ __device__ __forceinline__ uint64_t rj_hash(uint64_t k)
{
    k ^= k >> 32;
    k ^= k >> 21;
    k ^= k >> 16;
    return k * kRjHashMul;
}

// Row that sample i of a relation reads: one row of every `step`, at a
// multiple of `spread` that the MurmurHash3 32-bit finaliser of i picks.
// Rows at a fixed stride see a few values of keys that repeat with the row
// number (row % 2^16 at a stride of 2^8: one in 2^8): most regions of a layout
// overflow then, and the relation is partitioned twice.  spread is 1 for one
// pass.  For two it is 2: the test of that redo hides keys from the sample in
// the odd rows of an even stride.
__device__ __forceinline__ int64_t rj_sample_row(int64_t i, int64_t step, int spread, int64_t n)
{
    if (step == 1) return i;
    unsigned h = (unsigned)i;
    h ^= h >> 16;
    h *= 0x85ebca6bu;
    h ^= h >> 13;
    h *= 0xc2b2ae35u;
    h ^= h >> 16;
    return min(i * step + spread * (int64_t)(((uint64_t)h * (uint64_t)(step / spread)) >> 32), n - 1);
}

// Slot of key k in a shared-memory table of TS slots, for keys of one
// partition of 2^fb (fb = 0: one partition): multiply-high of the 32 hash
// bits below the partition bits.
__device__ __forceinline__ unsigned rj_slot(uint64_t k, int fb, unsigned TS)
{
    return __umulhi((unsigned)(rj_hash(k) >> (32 - fb)), TS);
}

}  // namespace pyg
