// The scan's filter and unions from grouped tuples instead of sorted ones.
//
// The mischief filter judges every run of equal k-mers by its adjacency-code counts (metapart.c:2270-2519) and
// the unions join the reads of every run (metapart.c:2520-2800); neither depends on the order of the tuples inside
// a run, nor on the order of the runs but for two places: a thread range's last run is never judged, and the
// sweeps' initial state (the scan's last k-mer, its first read).  So a scan is not sorted here: one or two
// multi-split passes bring it into units of consecutive m-mer buckets that fit shared memory, a hash table per
// unit groups its tuples by k-mer, and the two exceptions are taken from the units' bucket ranges (the largest
// k-mer of a unit that ends a thread range; k_gp_quirk).
#include <algorithm>
#include <cstdlib>
#include <mutex>
#include <type_traits>
#include <vector>

#include "k_group.cuh"
#include "k_readtile.cuh"

namespace mp {

constexpr unsigned FULLG = 0xFFFFFFFFu;

// ------------------------------------------------------------------ plan

constexpr int GP_UNIT_SHIFT = 12;        // units end where the tuple prefix crosses a multiple of 4096
constexpr int GP_CAP_S = 6128;           // most tuples of a unit for the small blocks (two per SM)
constexpr int GP_CAP_L = 12288;          // and for the 1024-thread blocks; a larger bucket takes the device-wide sort
constexpr uint32_t GP_DIGITS = 1024;     // digits of a split pass: bins of a segment, units of a bin
constexpr uint64_t GP_SMALL = 1500000;   // tuples of a segment that fit GP_DIGITS units however they are spread
constexpr int GP_COUNT_BLOCK = 512;      // buckets per block of the planning kernels, one per thread
constexpr uint32_t GP_NONE = 0x7FFFFFFFu;  // a grouped id that stands for no read
constexpr size_t PLAN_MAIL = DeviceArena::MAIL - 4096;  // where the plan's counters arrive in the mailbox
constexpr int QW = 8;  // words per segment: tuples found before the last run, last run's, its read, the run's place

struct PlanCtx {
    const uint64_t *hist;
    uint64_t lo, hi;          // buckets of the scan
    const uint32_t *brk;      // a bit per bucket (from lo): a thread range starts there
    const uint32_t *seg_sh;   // per segment: its bins hold 2^seg_sh buckets
    const uint32_t *seg_bin0; // per segment: its first bin
    uint32_t seg_lo;          // where a segment's bins count from (GroupScan::anchor, or 0 with several)
};

// The bin width of a segment of n tuples over `span` buckets.  A bin of at most 1024 buckets has at most 1024 units, so
// the second pass finds a tuple's unit in a table of the bin's buckets; the widest such bins, as the first pass stores a
// tile's tuples in runs by bin (20M x 150 bp, 2 scans, each with both passes: 512 bins 33.3 + 16.6 ms, 1024 bins 35.6 + 15.4).
// A segment of at most GP_SMALL tuples has at most 1024 units in all and takes bins of about 16384 tuples instead, which
// fill the second pass's tiles.
static int bin_width(uint64_t n, uint64_t span)
{
    const uint64_t want = n <= GP_SMALL ? std::max<uint64_t>(1, n >> 14) : std::max<uint64_t>((span + 1023) / 1024, 1);
    int s = 0;
    while (s < 16 && ((span - 1) >> s) + 1 > want) s++;  // a bucket within its bin takes 16 bits
    return s;
}

constexpr uint64_t GP_NO_BUCKET = ~0ull;

// The last index of [a, z) whose prefix is below x, by one warp; hist[a] < x <= hist[z].
__device__ __forceinline__ uint64_t last_below(const uint64_t *hist, uint64_t a, uint64_t z, uint64_t x)
{
    const int lane = threadIdx.x & 31;
    while (z - a > 1) {
        const uint64_t step = (z - a + 32) / 33, m = a + (uint64_t)(lane + 1) * step;
        const int n = __popc(__ballot_sync(FULLG, m < z && hist[m] < x));
        a += (uint64_t)n * step;
        z = min(z, a + step);
    }
    return a;
}

struct PrevSmem {
    int last[GP_COUNT_BLOCK / 32];
    uint64_t before;
};

// The populated bucket before b within b's segment (GP_NO_BUCKET: none), for a block's buckets b0 + thread, which are of
// one segment; s: b's prefix; populated: b is asked for.  All threads come here.  Only the block's first populated bucket
// has to search (every one of a sparse histogram searching for itself was 20 dependent loads: 20 us of each planning kernel
// for 10,000 reads).
__device__ __forceinline__ uint64_t prev_bucket(const PlanCtx &c, uint64_t b0, bool populated, PrevSmem &sm)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t m = __ballot_sync(FULLG, populated);
    if (lane == 0) sm.last[warp] = m ? warp * 32 + 31 - __clz(m) : -1;
    if (warp == 0) {
        const uint64_t first = max(c.lo, b0 & ~(uint64_t)(NB - 1)), s0 = c.hist[b0];
        uint64_t p = GP_NO_BUCKET;
        if (b0 > first && c.hist[first] != s0) {
            const uint64_t q = b0 - 1 - lane;
            const uint32_t near = __ballot_sync(FULLG, q >= first && q < b0 && c.hist[q] < s0);
            p = near ? b0 - (uint64_t)__ffs(near) : last_below(c.hist, first, b0, s0);
        }
        if (lane == 0) sm.before = p;
    }
    __syncthreads();
    const uint32_t lower = m & ((1u << lane) - 1);
    if (lower) return b0 + (uint64_t)(warp * 32 + 31 - __clz(lower));
    for (int w = warp - 1; w >= 0; w--)
        if (sm.last[w] >= 0) return b0 + (uint64_t)sm.last[w];
    return sm.before;
}

// Whether bucket b (populated, prefix [s, e) from the scan's start, p the one before) starts a unit (bit 0) and a thread range (bit 3).
// Units never cross a thread range, a segment, a bin or a multiple of 2^GP_UNIT_SHIFT tuples, except that a bucket which
// would make its unit larger than GP_CAP_S is a unit of its own: every decision is local to the bucket and its
// predecessor, so the plan is two parallel passes (a greedy packing by one thread per 256 buckets took 140-210 us).
__device__ __forceinline__ uint32_t plan_flags(const PlanCtx &c, uint64_t b, uint64_t s, uint64_t e, uint64_t p)
{
    if (p == GP_NO_BUCKET) return 9u;
    const uint64_t sp = c.hist[p] - c.hist[c.lo];
    const uint64_t rel = b - c.lo;
    const bool brk = (c.brk[rel >> 5] >> (rel & 31)) & 1u;
    const uint32_t sh = c.seg_sh[b / NB];
    const bool bin = (((uint32_t)b & (NB - 1)) - c.seg_lo) >> sh != (((uint32_t)p & (NB - 1)) - c.seg_lo) >> sh;
    const uint64_t q = s >> GP_UNIT_SHIFT;
    const bool unit = brk || bin || q != (sp >> GP_UNIT_SHIFT) || e - (q << GP_UNIT_SHIFT) > (uint64_t)GP_CAP_S;
    return (unit ? 1u : 0u) | (brk ? 8u : 0u);
}

// The bucket that starts at each thread range's first tuple, a warp each: the last one whose prefix is not above that is the
// populated one.
__global__ void k_gp_marks(const uint64_t *hist, uint64_t lo, uint64_t hi, const uint64_t *bounds, int nb, uint32_t *brk)
{
    const int t = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (t >= nb) return;
    const uint64_t x = bounds[t] + hist[lo];
    if (x >= hist[hi]) return;
    const uint64_t a = last_below(hist, lo, hi, x + 1);
    if ((threadIdx.x & 31) == 0) atomicOr(&brk[(a - lo) >> 5], 1u << ((a - lo) & 31));
}

__device__ __forceinline__ uint64_t block_scan_excl(uint64_t v, uint64_t *total, uint64_t *ws)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    uint64_t x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint64_t y = __shfl_up_sync(FULLG, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) ws[warp] = x;
    __syncthreads();
    uint64_t before = 0, tot = 0;
    for (int w = 0; w < nw; w++) {
        const uint64_t t = ws[w];
        before += w < warp ? t : 0;
        tot += t;
    }
    __syncthreads();
    *total = tot;
    return before + x - v;
}

// Units starting in each block of GP_COUNT_BLOCK buckets.  The plan's arrays have room for the units of a prefix that never
// falls; the caller's may come from a file, so one that does is told here (GC_ERR), and nothing is planned.
__global__ void __launch_bounds__(GP_COUNT_BLOCK) k_gp_count(PlanCtx c, uint64_t *blk, uint32_t *ctr)
{
    __shared__ PrevSmem ps;
    const uint64_t b0 = c.lo + (uint64_t)blockIdx.x * GP_COUNT_BLOCK, b = b0 + threadIdx.x;
    uint64_t s = 0, e = 0;
    if (b < c.hi) {
        s = c.hist[b];
        e = c.hist[b + 1];
    }
    const uint64_t h0 = c.hist[c.lo], p = prev_bucket(c, b0, s != e, ps);
    const bool f = s != e && (plan_flags(c, b, s - h0, e - h0, p) & 1u);
    const int n = __syncthreads_count(f);
    if (threadIdx.x == 0) blk[blockIdx.x] = (uint64_t)n;
    if (e < s) atomicOr(&ctr[GC_ERR], 2u);
}

// Exclusive scan of the blocks' counts by one block; the sentinels past the last unit and bin.
__global__ void __launch_bounds__(1024) k_gp_scan(uint64_t *blk, uint32_t nblk, uint32_t n, uint32_t nbins, uint32_t *ctr,
                                                  uint32_t *ustart, uint32_t *bstart, uint32_t *bu0)
{
    __shared__ uint64_t ws[32];
    uint64_t carry = 0;
    if (ctr[GC_ERR]) nblk = 0;  // no units
    for (uint32_t i0 = 0; i0 < nblk; i0 += 1024) {
        const uint32_t i = i0 + threadIdx.x;
        uint64_t tot;
        const uint64_t x = block_scan_excl(i < nblk ? blk[i] : 0, &tot, ws);
        if (i < nblk) blk[i] = carry + x;
        carry += tot;
    }
    if (threadIdx.x == 0) {
        ctr[GC_UNITS] = (uint32_t)carry;
        ustart[carry] = n;
        bstart[nbins] = n;
        bu0[nbins] = (uint32_t)carry;
    }
}

// The unit and bin arrays.  A bucket above GP_CAP_S tuples is a unit of its own (plan_flags), so its size is known here.
// One bucket per thread and one block scan: with eight buckets per thread in turn (eight scans) this and k_gp_count took
// 36 and 31 us for a scan of all buckets.
__global__ void __launch_bounds__(GP_COUNT_BLOCK) k_gp_write(PlanCtx c, const uint64_t *blk, uint32_t *ctr, uint32_t *ustart,
                                                             uint32_t *ub0, uint32_t *ucur, uint32_t *bstart, uint32_t *bu0,
                                                             uint32_t *bcur, uint32_t *bsh, uint32_t *bfirst, uint32_t *unit_of,
                                                             uint32_t *mid, uint32_t *big)
{
    __shared__ uint32_t ws[GP_COUNT_BLOCK / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    __shared__ PrevSmem ps;
    if (ctr[GC_ERR]) return;  // (set by k_gp_count alone until here)
    const uint64_t b0 = c.lo + (uint64_t)blockIdx.x * GP_COUNT_BLOCK, b = b0 + threadIdx.x;
    uint64_t s = 0, e = 0;
    if (b < c.hi) {
        const uint64_t h0 = c.hist[c.lo];
        s = c.hist[b] - h0;
        e = c.hist[b + 1] - h0;
    }
    const uint64_t p = prev_bucket(c, b0, s != e, ps);
    const uint32_t f = s != e ? plan_flags(c, b, s, e, p) : 0u;
    const uint32_t m = __ballot_sync(FULLG, f & 1u);
    if (lane == 0) ws[warp] = (uint32_t)__popc(m);
    __syncthreads();
    if (b >= c.hi) return;
    uint32_t u = (uint32_t)blk[blockIdx.x] + (uint32_t)__popc(m & ((1u << lane) - 1));  // units that start before b
    for (int w = 0; w < warp; w++) u += ws[w];
    const uint32_t seg = (uint32_t)(b / NB), rel = ((uint32_t)b & (NB - 1)) - c.seg_lo, sh = c.seg_sh[seg];
    if ((rel & ((1u << sh) - 1)) == 0 || b == c.lo) {  // (a merged scan's first bin may begin before the scan)
        const uint32_t bin = c.seg_bin0[seg] + (rel >> sh);
        bstart[bin] = (uint32_t)s;
        if (bcur) bcur[bin] = (uint32_t)s;
        bu0[bin] = u;
        bfirst[bin] = (uint32_t)(b - c.lo) - (rel & ((1u << sh) - 1));
        bsh[bin] = sh;
    }
    unit_of[b - c.lo] = u + (f & 1u) - 1u;  // (before the first unit: ~0)
    if (f & 1u) {
        ustart[u] = ucur[u] = (uint32_t)s;
        ub0[u] = (uint32_t)b | (f & 8u ? 0x80000000u : 0u);
    }
    if (e - s > (uint64_t)GP_CAP_S) {
        if (e - s <= (uint64_t)GP_CAP_L) mid[atomicAdd(&ctr[GC_MID], 1u)] = u;
        else {
            big[atomicAdd(&ctr[GC_BIG], 1u)] = u;
            atomicAdd(&ctr[GC_BIG_TUPLES], (uint32_t)(e - s));
        }
    }
}

// ------------------------------------------------------------------ split

constexpr int SP_THREADS = 512, SP_ITEMS = 12, SP_TILE = SP_THREADS * SP_ITEMS;
constexpr uint32_t SP_EXTRA = GROUP_MAX_MERGED - 1;  // digits above GP_DIGITS: a bin that a scan's bounds cut counts once more

// Tiles of the second pass, every bin's own: first tuple, tuples, bin.  Every block counts the tiles and writes its share
// (one block with a bin's tiles per thread took 115 us at 200,000 tiles).
__global__ void __launch_bounds__(1024) k_gp_tiles(const uint32_t *bstart, uint32_t nb, uint32_t *ctr, uint4 *tiles)
{
    __shared__ uint64_t ws[32];
    __shared__ uint32_t at[1024], sb[1025];
    uint32_t carry = 0;
    if (ctr[GC_ERR]) nb = 0;  // no tiles
    for (uint32_t i0 = 0; i0 < nb; i0 += 1024) {
        const uint32_t i = i0 + threadIdx.x, s = bstart[min(i, nb)], e = bstart[min(i + 1, nb)];
        uint64_t tot;
        at[threadIdx.x] = (uint32_t)block_scan_excl((e - s + SP_TILE - 1) / SP_TILE, &tot, ws);
        sb[threadIdx.x] = s;
        if (threadIdx.x == 1023) sb[1024] = e;
        __syncthreads();
        for (uint32_t t = blockIdx.x * 1024 + threadIdx.x; t < (uint32_t)tot; t += gridDim.x * 1024) {
            uint32_t x = 0;  // the last bin whose first tile is not after t (it has tiles)
#pragma unroll
            for (uint32_t w = 512; w; w >>= 1)
                if (at[x + w] <= t) x += w;
            const uint32_t o = (t - at[x]) * SP_TILE;
            tiles[carry + t] = make_uint4(sb[x] + o, min((uint32_t)SP_TILE, sb[x + 1] - sb[x] - o), i0 + x, 0);
        }
        __syncthreads();
        carry += (uint32_t)tot;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) ctr[GC_TILES] = carry;
}

struct SplitSmem {
    uint64_t key[SP_TILE];
    uint32_t id[SP_TILE];
    uint16_t dig[SP_TILE];      // a place's digit, times 4
    uint32_t hist[GP_DIGITS + SP_EXTRA];   // tuples per digit, then the digit's first place in the tile
    uint32_t delta[GP_DIGITS + SP_EXTRA];  // global place of a digit's first tuple less its place in the tile
    uint32_t ws[SP_THREADS / 32];
};
constexpr uint32_t SP_PACKED = 4096;  // words of packed reads
struct BinSmem : SplitSmem {
    uint32_t packed[SP_PACKED];
};
struct UnitSmem : SplitSmem {
    uint16_t cell[GP_DIGITS];   // the bin's buckets in 1024 cells: the digit (times 4) of a cell's first bucket
    uint16_t b0[GP_DIGITS];     // first bucket of every unit within the bin (bins of more than 1024 buckets)
};
constexpr uint32_t SP_CHUNK = 4;  // most tiles of the second pass a block takes at a time
static_assert(2 * (sizeof(UnitSmem) + 1024) <= 228 * 1024 && 2 * (sizeof(BinSmem) + 3 * 1024) <= 228 * 1024, "two split blocks per SM");

__device__ __forceinline__ uint32_t &at_byte(uint32_t *p, uint32_t off) { return *reinterpret_cast<uint32_t *>(reinterpret_cast<char *>(p) + off); }

// Unstable, so there are no ballots and no look-back: ranks by shared-memory atomics, places by one global atomic per
// digit and tile (the order of a digit's tuples is free; its latency passes while the tile is reordered), a
// shared-memory reorder so that a digit's tuples are stored side by side.  rd: digit times 4 (bits 0-15) and the tuple's rank
// in it (16-31), or ~0 for none, as the caller's atomics on sm.hist gave them.  Returns the tile's tuples.  EXTRA: with
// the SP_EXTRA digits above GP_DIGITS.
template <bool EXTRA, class LoadId>
__device__ __forceinline__ uint32_t split_order(SplitSmem &sm, const uint32_t (&kl)[SP_ITEMS], const uint32_t (&kh)[SP_ITEMS],
                                                const uint32_t (&rd)[SP_ITEMS], uint32_t *cur, uint32_t nd, LoadId load_id)
{
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    uint32_t id[SP_ITEMS];
#pragma unroll
    for (int j = 0; j < SP_ITEMS; j++) id[j] = load_id(j);
    __syncthreads();
    static_assert(GP_DIGITS == 2 * SP_THREADS, "two digits per thread");
    const uint2 c = *reinterpret_cast<const uint2 *>(&sm.hist[2 * tid]);
    const uint32_t g0 = c.x && 2 * tid < nd ? atomicAdd(&cur[2 * tid], c.x) : 0u;
    const uint32_t g1 = c.y && 2 * tid + 1 < nd ? atomicAdd(&cur[2 * tid + 1], c.y) : 0u;
    static_assert(SP_EXTRA == 2, "two extra digits");
    uint32_t ex = 0, ey = 0, ge = 0;  // the extra digits' tuples, the place of this thread's one
    if constexpr (EXTRA) {
        ex = sm.hist[GP_DIGITS];
        ey = sm.hist[GP_DIGITS + 1];
        const uint32_t n0 = tid ? ey : ex;
        if (tid < 2 && n0 && GP_DIGITS + tid < nd) ge = atomicAdd(&cur[GP_DIGITS + tid], n0);
    }
    uint32_t x = c.x + c.y;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(FULLG, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) sm.ws[warp] = x;
    __syncthreads();
    uint32_t before = x - c.x - c.y, nv = 0;
#pragma unroll
    for (int w = 0; w < SP_THREADS / 32; w++) {
        const uint32_t v = sm.ws[w];
        before += w < warp ? v : 0u;
        nv += v;
    }
    *reinterpret_cast<uint2 *>(&sm.hist[2 * tid]) = make_uint2(before, before + c.x);
    if constexpr (EXTRA) {
        if (tid < 2) {
            const uint32_t at = nv + (tid ? ex : 0u);
            sm.hist[GP_DIGITS + tid] = at;
            sm.delta[GP_DIGITS + tid] = ge - at;
        }
        nv += ex + ey;
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < SP_ITEMS; j++) {
        if (rd[j] != ~0u) {
            const uint32_t d = rd[j] & 0xFFFFu, p = at_byte(sm.hist, d) + (rd[j] >> 16);
            sm.key[p] = ((uint64_t)kh[j] << 32) | kl[j];
            sm.id[p] = id[j];
            sm.dig[p] = (uint16_t)d;
        }
    }
    *reinterpret_cast<uint2 *>(&sm.delta[2 * tid]) = make_uint2(g0 - before, g1 - before - c.x);
    __syncthreads();
    return nv;
}

// A digit with more tuples than the histogram gave it (which is then not the tuples': k_split_units and k_group tell) runs on
// into the next one's places, and past all n of them the tuples are left out: every place that a cursor passed holds a
// tuple, so what is read of it later is in range.
template <bool EXTRA>
__device__ __forceinline__ void split_store(SplitSmem &sm, uint32_t nv, uint64_t *out_k, uint32_t *out_id, uint32_t n)
{
#pragma unroll 4
    for (uint32_t p = threadIdx.x; p < nv; p += SP_THREADS) {
        const uint32_t o = p + at_byte(sm.delta, sm.dig[p]);
        if (o < n) {
            out_k[o] = sm.key[p];
            out_id[o] = sm.id[p];
        }
    }
    *reinterpret_cast<uint2 *>(&sm.hist[2 * threadIdx.x]) = make_uint2(0, 0);
    if (EXTRA && threadIdx.x < SP_EXTRA) sm.hist[GP_DIGITS + threadIdx.x] = 0;
}

// The tiles of a pass over segments: tile0[q] the segment's first tile, start[q] its first read or tuple, tile_seg the
// segment of every tile; null for one segment.
struct SegTiles {
    const uint32_t *tile_seg = nullptr, *tile0 = nullptr, *start = nullptr;
    const uint4 *shape = nullptr;  // of reads: the tiling of each segment's reads (P, spr, rounds, rpt of ReadTiles)
};

__global__ void k_gp_segtiles(const uint32_t *tile0, int nseg, uint32_t *tile_seg)
{
    const int q = blockIdx.x;
    for (uint32_t t = tile0[q] + threadIdx.x; t < tile0[q + 1]; t += blockDim.x) tile_seg[t] = (uint32_t)q;
}

// First pass, one of two sources: the reads (k_readtile.cuh; the tuples of the scan's buckets), or tuples enumerated
// before (lo = k-mer << 8 | adj, hi = k-mer >> 56; the 3-minimizer variant).
struct BinCtx {
    ReadTiles t;
    uint32_t n_reads = 0, check_many = 0;
    const uint32_t *label = nullptr;
    const uint64_t *lo = nullptr;
    const uint8_t *hi = nullptr;
    const uint32_t *id = nullptr;
    uint32_t tiles = 0, n = 0;
    uint64_t k_lo = 0, k_span = 0;  // the scan's k-mers: [k_lo, k_lo + k_span)
    int bsh = 0;
    const uint32_t *seg_bin0 = nullptr, *seg_sh = nullptr;
    uint32_t *bcur = nullptr, *err = nullptr;
    SegTiles sg;
    uint64_t *out_k = nullptr;
    uint32_t *out_id = nullptr;
    uint32_t m_digits = 0, m_sh = 0;                    // merged scans (group_bins_scans): the digits, the bins' width
    uint64_t m_start[SP_EXTRA] = {~0ull, ~0ull};        // the first k-mer of every scan but the first, less k_lo
};

__device__ __forceinline__ void bin_tile(const BinCtx &c, uint32_t tile, uint32_t per, uint32_t all, uint32_t &seg, uint32_t &base,
                                         uint32_t &end)
{
    seg = c.sg.tile_seg ? c.sg.tile_seg[tile] : 0u;
    base = tile * per;
    end = all;
    if (c.sg.tile_seg) {
        base = c.sg.start[seg] + (tile - c.sg.tile0[seg]) * per;
        end = c.sg.start[seg + 1];
    }
    end = min(end, base + per);
}

// Bound by the instructions of the k-mers (about 90 per position at 38 % issue; two blocks' 64 registers a thread hold 32
// warps per SM) and the shared-memory reorder; the random stores and the ranks' atomics are about a fifth each.  20M x
// 150 bp, 2 scans: 23.9 ms together (33.6 with a pass per scan) for what counting (6.1), enumerating (14.3) and a first split
// over 13-byte tuples (29.3) took.
//
// HI: 2k >= 34 and bins of at least 2^32 k-mers, so a k-mer's bin is a shift of its high word.
//
// SR_MERGED: the tuples of all scans (group_bins_scans).  Packing the reads and rolling through them was half of the pass.
// SR_SEGMENTS: each segment's reads have their own tiling (samples of reads of 100 bases tiled as ones of 250 left two
// threads of three idle).
enum { SR_ONE = 0, SR_MERGED = 1, SR_SEGMENTS = 2 };
template <bool HI, int MODE>
__global__ void __launch_bounds__(SP_THREADS, 2) k_split_reads(BinCtx c)
{
    extern __shared__ __align__(16) unsigned char smraw[];
    BinSmem &sm = *reinterpret_cast<BinSmem *>(smraw);
    __shared__ uint32_t many[SP_THREADS];
    const int tid = threadIdx.x;
    for (uint32_t d = tid; d < GP_DIGITS + SP_EXTRA; d += SP_THREADS) sm.hist[d] = 0;
    constexpr bool MERGED = MODE == SR_MERGED;
    ReadTiles t = c.t;
    uint32_t seg = 0, base = 0, end = 0, rr = tid / t.spr, i0 = (tid - rr * t.spr) * t.P;
    auto take = [&](uint32_t tile) {  // the tile's reads, packed
        if constexpr (MODE == SR_SEGMENTS) {
            const uint4 s = c.sg.shape[c.sg.tile_seg[tile]];
            t.P = s.x;
            t.spr = s.y;
            t.rounds = s.z;
            t.rpt = s.w;
            rr = tid / t.spr;
            i0 = (tid - rr * t.spr) * t.P;
        }
        bin_tile(c, tile, t.rpt, c.n_reads, seg, base, end);
        rt_pack(t, base, end - base, sm.packed);
    };
    if (blockIdx.x < c.tiles) take(blockIdx.x);
    for (uint32_t tile = blockIdx.x; tile < c.tiles; tile += gridDim.x) {
        const uint32_t d0 = MERGED ? 0u : c.seg_bin0[seg], nd = MERGED ? c.m_digits : c.seg_bin0[seg + 1] - d0;
        const int bits = c.bsh + (int)(MERGED ? c.m_sh : c.seg_sh[seg]);  // a k-mer's bits within its bin
        const uint64_t mask = (1ull << bits) - 1;
        const uint32_t r = base + rr, L = rr < t.rpt && r < end ? c.t.seq_len[r] : 0u;
        uint32_t id = r;
        if (c.label && L) {
            const uint32_t p = c.label[r];
            id = p == BAD ? r : p;  // findRoot after full compression (metapart.c:543-568)
        }
        if (c.check_many) many[tid] = 0;
        __syncthreads();  // the tile before is stored, this one's reads are packed
        uint32_t kl[SP_ITEMS], kh[SP_ITEMS], rd[SP_ITEMS];
        {
            KmerRoll<HI> s = {};
            if (L > (uint32_t)c.t.k && i0 <= L - (uint32_t)c.t.k) s.init(t, sm.packed + rr * rt_stride(t), L, i0);
            const uint32_t mh = (uint32_t)(mask >> 32), dsh = HI ? bits - 32 : bits;
            const uint32_t cn[2] = {s.compl_nibbles(s.an[0]), s.compl_nibbles(s.an[1])};
            const uint32_t cp[2] = {s.compl_nibbles(s.ap[0]), s.compl_nibbles(s.ap[1])};
            uint32_t got = 0;
            auto position = [&](auto J) {
                constexpr int j = decltype(J)::value;
                const uint64_t f = s.fwd(), q = s.rc();
                const bool fw = f < q;
                const uint64_t rel = (fw ? f : q) - c.k_lo;
                const uint32_t a6 = s.template adj6<j>(fw, cn, cp);
                rd[j] = ~0u;
                if (((s.vm >> j) & 1u) && rel < c.k_span) {
                    uint32_t d = HI ? (uint32_t)(rel >> 32) >> dsh : (uint32_t)(rel >> dsh);
                    if constexpr (MERGED) {  // one more for every scan that began
#pragma unroll
                        for (uint32_t q = 0; q < SP_EXTRA; q++) d += rel >= c.m_start[q];
                    }
                    if constexpr (HI) {
                        kl[j] = ((uint32_t)rel << 6) | a6;
                        kh[j] = __funnelshift_l((uint32_t)rel, (uint32_t)(rel >> 32) & mh, 6);
                    } else {
                        const uint64_t key = ((rel & mask) << 6) | a6;
                        kl[j] = (uint32_t)key;
                        kh[j] = (uint32_t)(key >> 32);
                    }
                    rd[j] = (d << 2) | (atomicAdd(&sm.hist[d], 1u) << 16);
                    got++;
                }
                s.next();
            };
            static_assert(SP_ITEMS == 12, "positions below");
            position(std::integral_constant<int, 0>{});
            position(std::integral_constant<int, 1>{});
            position(std::integral_constant<int, 2>{});
            position(std::integral_constant<int, 3>{});
            position(std::integral_constant<int, 4>{});
            position(std::integral_constant<int, 5>{});
            position(std::integral_constant<int, 6>{});
            position(std::integral_constant<int, 7>{});
            position(std::integral_constant<int, 8>{});
            position(std::integral_constant<int, 9>{});
            position(std::integral_constant<int, 10>{});
            position(std::integral_constant<int, 11>{});
            // the reference counts a read's k-mers of one scan in 8 bits (enumerateKmers.c:152)
            if (c.check_many && got && atomicAdd(&many[rr], got) + got > 255u) atomicOr(c.err, 4u);
        }
        const uint32_t nv = split_order<MERGED>(sm, kl, kh, rd, c.bcur + d0, nd, [&](int) { return id; });
        split_store<MERGED>(sm, nv, c.out_k, c.out_id, c.n);
        // the next tile's reads while others store (its bytes fetched before the stores instead cost registers that spill: 37.5
        // against 35.7 ms at 20M x 150 bp, 2 scans with a pass each)
        const uint32_t next = tile + gridDim.x;
        if (next < c.tiles) take(next);
    }
}

__global__ void __launch_bounds__(SP_THREADS, 2) k_split_tuples(BinCtx c)
{
    extern __shared__ __align__(16) unsigned char smraw[];
    SplitSmem &sm = *reinterpret_cast<SplitSmem *>(smraw);
    const int tid = threadIdx.x;
    for (uint32_t d = tid; d < GP_DIGITS; d += SP_THREADS) sm.hist[d] = 0;
    for (uint32_t tile = blockIdx.x; tile < c.tiles; tile += gridDim.x) {
        uint32_t seg, base, end;
        bin_tile(c, tile, SP_TILE, c.n, seg, base, end);
        const uint32_t d0 = c.seg_bin0[seg], nd = c.seg_bin0[seg + 1] - d0, nv = end - base;
        const int bits = c.bsh + (int)c.seg_sh[seg];
        const uint64_t mask = (1ull << bits) - 1;
        __syncthreads();  // the tile before is stored
        uint32_t kl[SP_ITEMS], kh[SP_ITEMS], rd[SP_ITEMS];
#pragma unroll
        for (int j = 0; j < SP_ITEMS; j++) {
            const uint32_t e = j * SP_THREADS + tid;
            rd[j] = ~0u;
            if (e < nv) {
                const uint64_t v = c.lo[base + e], km = (v >> 8) | (c.hi ? (uint64_t)c.hi[base + e] << 56 : 0ull);
                const uint64_t rel = km - c.k_lo;
                if (rel < c.k_span) {
                    const uint64_t key = ((rel & mask) << 6) | (v & 63u);
                    const uint32_t d = (uint32_t)(rel >> bits);
                    kl[j] = (uint32_t)key;
                    kh[j] = (uint32_t)(key >> 32);
                    rd[j] = (d << 2) | (atomicAdd(&sm.hist[d], 1u) << 16);
                }
            }
        }
        const uint32_t got = split_order<false>(
            sm, kl, kh, rd, c.bcur + d0, nd,
            [&](int j) { const uint32_t e = j * SP_THREADS + tid; return e < nv ? c.id[base + e] : 0u; });
        split_store<false>(sm, got, c.out_k, c.out_id, c.n);
    }
}

// Second pass: a bin's tuples into its units.  Blocks take four consecutive tiles at a time, so all of them work in a few
// neighbouring bins: with long stretches per block instead (a bin or more), 300 bins of 560 units were open at once, L2
// evicted their half-filled lines, and 2.39 G tuples moved 102 GB through DRAM where they take 57 (26.5 ms; 17.5 in stretches
// of four, and 21.5 with a later scan's component lookups, at 20M x 150 bp, 2 scans).
__global__ void __launch_bounds__(SP_THREADS, 2) k_split_units(const uint64_t *__restrict__ kk, const uint32_t *__restrict__ id,
                                                               uint32_t n, int bsh, uint32_t seg_lo, uint32_t *ctr, uint32_t nbins,
                                                               const uint32_t *__restrict__ bstart,
                                                               const uint32_t *__restrict__ bfirst,
                                                               const uint32_t *__restrict__ bu0,
                                                               const uint32_t *__restrict__ bcur,
                                                               const uint32_t *__restrict__ bin_sh,
                                                               const uint32_t *__restrict__ ub0, uint32_t *ucur,
                                                               const uint32_t *__restrict__ unit_of, uint32_t nbk,
                                                               const uint4 *__restrict__ tile_of, uint32_t tuple0,
                                                               const uint32_t *__restrict__ label, uint64_t *out_k,
                                                               uint32_t *out_id)
{
    extern __shared__ __align__(16) unsigned char smraw[];
    UnitSmem &sm = *reinterpret_cast<UnitSmem *>(smraw);
    const int tid = threadIdx.x, bits = bsh + 6;
    const uint32_t tiles = ctr[GC_TILES];
    uint32_t have = ~0u, d0 = 0, nd = 0;
    int cs = 0;  // buckets per cell: 2^cs, 0 for bins of at most 1024 buckets
    bool whole = false;
    for (uint32_t d = tid; d < GP_DIGITS; d += SP_THREADS) sm.hist[d] = 0;
    // every bin, those without a tuple in the histogram too, holds as many as that says, or the histogram is not the tuples'
    for (uint32_t x = blockIdx.x * SP_THREADS + tid; x < nbins; x += gridDim.x * SP_THREADS)
        if (bcur[x] - tuple0 != bstart[x + 1]) atomicOr(&ctr[GC_ERR], 2u);
    const uint32_t chunk = min(SP_CHUNK, max(1u, tiles / gridDim.x));  // (few tiles: one for each block)
    auto tile_at = [&](uint32_t i) { return ((i / chunk) * gridDim.x + blockIdx.x) * chunk + i % chunk; };
    uint32_t kl[SP_ITEMS], kh[SP_ITEMS];
    auto load = [&](const uint4 &t) {
        const uint64_t *kp = kk + t.x + tid;
#pragma unroll
        for (int j = 0; j < SP_ITEMS; j++) {
            const uint64_t v = j * SP_THREADS + tid < t.y ? kp[j * SP_THREADS] : 0ull;
            kl[j] = (uint32_t)v;
            kh[j] = (uint32_t)(v >> 32);
        }
    };
    uint4 now = make_uint4(0, 0, 0, 0);
    if (tile_at(0) < tiles) {
        now = tile_of[tile_at(0)];
        load(now);
    }
    for (uint32_t i = 0; tile_at(i) < tiles; i++) {
        const uint32_t base = now.x, nv = now.y, bin = now.z;
        __syncthreads();  // the tile before is stored
        if (bin != have) {
            have = bin;
            whole = bcur[bin] - tuple0 == bstart[bin + 1];  // else some of its places may hold nothing
            d0 = bu0[bin];
            nd = min(bu0[bin + 1] - d0, GP_DIGITS);
            const uint32_t s = bin_sh[bin], b0 = bfirst[bin];
            cs = s > 10 ? (int)s - 10 : 0;
            for (uint32_t x = tid; x < GP_DIGITS; x += SP_THREADS) {
                const uint32_t r = b0 + (x << cs);
                const uint32_t u = x < (1u << (s - cs)) && r < nbk ? unit_of[r] : d0;
                sm.cell[x] = (uint16_t)((u + 1 > d0 + 1 ? min(u - d0, nd - 1) : 0u) << 2);
                if (cs && x < nd) sm.b0[x] = (uint16_t)(((ub0[d0 + x] & (NB - 1)) - seg_lo) & ((1u << s) - 1));
            }
            __syncthreads();
        }
        uint32_t got = 0;
        if (whole) {
            uint32_t rd[SP_ITEMS];
#pragma unroll
            for (int j = 0; j < SP_ITEMS; j++) {
                const uint32_t b = bits >= 32 ? kh[j] >> (bits - 32) : __funnelshift_r(kl[j], kh[j], bits);
                uint32_t d4 = sm.cell[(b >> cs) & (GP_DIGITS - 1)];  // (a tuple of another bin, where that one runs over)
                if (cs)
                    while (d4 / 4 + 1 < nd && sm.b0[d4 / 4 + 1] <= b) d4 += 4;
                rd[j] = j * SP_THREADS + tid < nv ? d4 | (atomicAdd(&at_byte(sm.hist, d4), 1u) << 16) : ~0u;
            }
            const uint32_t *ip = id + base + tid;
            got = split_order<false>(
                sm, kl, kh, rd, ucur + d0, nd,
                [&](int j) {
                    uint32_t v = j * SP_THREADS + tid < nv ? ip[j * SP_THREADS] : 0u;
                    if (label) {
                        const uint32_t p = label[v];
                        v = p == BAD ? v : p;
                    }
                    return v;
                });
        }
        if (tile_at(i + 1) < tiles) {  // the next tile's keys on their way while this one's tuples are stored
            now = tile_of[tile_at(i + 1)];
            load(now);
        }
        split_store<false>(sm, got, out_k, out_id, n);
    }
}

// ------------------------------------------------------------------ group and filter

// ratio_above_02 of k_graph.cu for counts below 2^24 (a unit's run): (float)s / deg > 0.2 compared as a double.
__device__ __forceinline__ bool ratio_above_02_small(uint32_t s, uint32_t deg) { return ((uint64_t)s << 27) > 26843545ull * deg; }

template <int THREADS, int ITEMS, int SLOT_BITS>
struct GroupSmem {
    static constexpr int CAP = THREADS * ITEMS, SLOTS = 1 << SLOT_BITS;
    // first the table's keys; then, once every tuple knows its slot, the counters of the runs that branch on one
    // side (16 bytes each: seven 16-bit counts and the slot), later overwritten by the grouped ids, and behind
    // them each slot's first place among the grouped ids
    union {
        unsigned long long key[SLOTS];
        struct {
            uint32_t pool[(SLOTS * 8 - SLOTS * 2) / 4];
            uint16_t off[SLOTS];
        } b;
    } u;
    uint32_t info[SLOTS];  // count (bits 0-15), before codes seen (16-22), after codes seen (23-29); later see k_group
    uint32_t ws[THREADS / 32];
    unsigned long long maxkey;
    uint32_t npool, slot_ex, base, next;
};

constexpr uint32_t GI_KEPT = 1u << 31;

__device__ __forceinline__ uint32_t key_hash(uint64_t k) { return (uint32_t)k * 0x9E3779B1u + (uint32_t)(k >> 32) * 0x85EBCA77u; }

struct GroupCtx {
    const uint64_t *kk;
    const uint32_t *ids;
    const uint32_t *ustart, *ub0, *fill, *lrs, *list;  // list: the units to take (null: all)
    uint32_t *ctr, *qlist, *quirk;
    int work, count;          // counters of the units taken and of the units there are
    bool ends_range, ends_scan;  // of the last unit (GroupScan)
    uint32_t cap_lo, cap_hi;  // takes units of cap_lo < tuples <= cap_hi
    uint32_t *out, *parent;
    uint8_t *filtered;
};

// Bound by shared memory (random accesses and atomics: about five per tuple), its instructions and the block's barriers;
// two small blocks per SM overlap each other's.  20M x 150 bp, 2 scans (2.39 G tuples): 26.3 ms for both block shapes,
// where sorting the units (66.8 ms) and judging the sorted runs (31.9 ms) took 98.7.  A tuple's slot, its number there
// and its codes share a word, so that 768 threads of 8 tuples keep 40 registers: 512 of 12 took 27.9 ms, 1024 of 6 27.2;
// every tuple's info read again for the marks and the rare tests in the probe loop 30.4; probing pairs of slots at once
// gained nothing.
//
// One block per unit (persistent, units handed out by a counter): the unit's tuples into a hash table of its
// k-mers (open addressing in shared memory), the filter's judgement of every k-mer, its marks, and the reads of
// every k-mer that joins reads (at least two tuples, not zeroed, not the zero k-mer) side by side into out.
//
// A run acts in the filter only if its tuples carry two or more before-codes or after-codes, which the masks in
// info tell; with both sides branching the run is zeroed whatever its counts, so counts are taken only for the
// runs branching on one side.  The last run of a unit that ends a thread range is not judged.
//
// Later use of info: count (0-13), branching side (14-15: 0 none, 1 before, 2 after, 3 both), the run's counters
// in pool (16-28), then the judgement (16-18 most frequent code, 19 second count above 0.2), kept (31).
template <int THREADS, int ITEMS, int SLOT_BITS>
__global__ void __launch_bounds__(THREADS, SLOT_BITS == 13 ? 2 : 1) k_group(GroupCtx c)
{
    typedef GroupSmem<THREADS, ITEMS, SLOT_BITS> Smem;
    constexpr uint32_t SLOTS = Smem::SLOTS, SMASK = SLOTS - 1;
    constexpr unsigned long long EMPTY = ~0ull;
    extern __shared__ __align__(16) unsigned char smraw[];
    Smem &sm = *reinterpret_cast<Smem *>(smraw);
    volatile unsigned long long *vkey = sm.u.key;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t nunits = c.ctr[c.count], nall = c.ctr[GC_UNITS];
    if (tid == 0) sm.next = atomicAdd(&c.ctr[c.work], 1u);
    for (;;) {
        __syncthreads();
        const uint32_t w = sm.next;
        if (w >= nunits) return;
        const uint32_t u = c.list ? c.list[w] : w;
        const uint32_t start = c.ustart[u], cnt = c.ustart[u + 1] - start, b0 = c.ub0[u] & 0x7FFFFFFFu;
        const bool take = cnt > c.cap_lo && cnt <= c.cap_hi;
        const bool last = u + 1 == nall;
        const uint32_t nextb = last ? ~0u : c.ub0[u + 1];
        const bool ends = last ? c.ends_range : nextb >> 31, seg_last = last ? c.ends_scan : (nextb & 0x7FFFFFFFu) / NB != b0 / NB;
        const uint32_t seg = b0 / NB;
        const bool singles = start >= c.lrs[seg];  // in the segment's last range every read that may join counts (k_gp_quirk)
        __syncthreads();
        if (tid == 0) {
            sm.next = atomicAdd(&c.ctr[c.work], 1u);
            sm.npool = 0;
            sm.slot_ex = ~0u;
            sm.maxkey = 0;
        }
        if (!take) continue;
        if (c.fill[u] != start + cnt) {  // the histogram is not the tuples': part of the unit was never written
            if (tid == 0) atomicOr(&c.ctr[GC_ERR], 2u);
            continue;
        }
        uint64_t key[ITEMS];
#pragma unroll
        for (int j = 0; j < ITEMS; j++) {
            const uint32_t e = j * THREADS + tid;
            key[j] = e < cnt ? c.kk[start + e] : 0ull;
        }
        {
            ulonglong2 *k2 = reinterpret_cast<ulonglong2 *>(sm.u.key);
            for (uint32_t i = tid; i < SLOTS / 2; i += THREADS) k2[i] = make_ulonglong2(EMPTY, EMPTY);
            uint4 *i4 = reinterpret_cast<uint4 *>(sm.info);
            for (uint32_t i = tid; i < SLOTS / 4; i += THREADS) i4[i] = make_uint4(0, 0, 0, 0);
        }
        __syncthreads();
        if (ends) {
            unsigned long long m = 0;
#pragma unroll
            for (int j = 0; j < ITEMS; j++)
                if (j * THREADS + tid < cnt) m = max(m, (unsigned long long)(key[j] >> 6));
#pragma unroll
            for (int o = 16; o; o >>= 1) m = max(m, __shfl_xor_sync(FULLG, m, o));
            if (lane == 0) atomicMax(&sm.maxkey, m);
            __syncthreads();
        }
        // ---- every tuple's slot, its number within the slot and its codes, in one word where they fit
        constexpr bool PACK = 2 * SLOT_BITS + 6 <= 32;
        uint32_t sr[ITEMS] = {}, ac[PACK ? 1 : ITEMS] = {};
        auto slot = [&](int j) { return sr[j] & SMASK; };
        auto number = [&](int j) { return (sr[j] >> SLOT_BITS) & SMASK; };
        auto code6 = [&](int j) { return PACK ? sr[j] >> 26 : ac[PACK ? 0 : j]; };
        auto set_code6 = [&](int j, uint32_t v) {
            if (PACK) sr[j] = (sr[j] & 0x3FFFFFFu) | (v << 26);
            else ac[PACK ? 0 : j] = v;
        };
#pragma unroll
        for (int j = 0; j < ITEMS; j++) {
            if (j * THREADS + tid < cnt) {
                const unsigned long long k = key[j] >> 6;
                const uint32_t kh = key_hash(k), step = kh | 1u, code = (uint32_t)key[j] & 63u;
                uint32_t h = kh >> (32 - SLOT_BITS);
                for (;;) {
                    unsigned long long v = vkey[h];
                    if (v == EMPTY) {
                        v = atomicCAS(&sm.u.key[h], EMPTY, k);
                        if (v == EMPTY) v = k;
                    }
                    if (v == k) break;
                    h = (h + step) & SMASK;
                }
                const uint32_t m = ((0x10000u << (code & 7u)) & 0x7F0000u) | ((0x800000u << (code >> 3)) & 0x3F800000u);
                const uint32_t old = atomicAdd(&sm.info[h], 1u);
                if (m & ~old) atomicOr(&sm.info[h], m);
                sr[j] = h | ((old & SMASK) << SLOT_BITS);
                set_code6(j, code);
            }
        }
        uint32_t zeros = 0, kept_here = 0;  // a bit per tuple: the zero k-mer's; the first of a slot whose reads are kept
        const bool zero_bucket = (b0 & (NB - 1)) == 0;
        if (ends || zero_bucket) {
            const unsigned long long mx = sm.maxkey;
#pragma unroll
            for (int j = 0; j < ITEMS; j++) {
                if (j * THREADS + tid < cnt) {
                    const unsigned long long k = key[j] >> 6;
                    if (zero_bucket && k == 0) zeros |= 1u << j;
                    if (ends && k == mx) sm.slot_ex = slot(j);
                }
            }
        }
        uint32_t id[ITEMS];
#pragma unroll
        for (int j = 0; j < ITEMS; j++) {
            const uint32_t e = j * THREADS + tid;
            id[j] = e < cnt ? c.ids[start + e] : 0u;
        }
        __syncthreads();
        // ---- a slot's first tuple decides its side, its counters and whether its reads are kept
        const uint32_t ex = sm.slot_ex;
        uint32_t kept = 0;
#pragma unroll
        for (int j = 0; j < ITEMS; j++) {
            if (j * THREADS + tid < cnt && number(j) == 0) {
                const uint32_t h = slot(j), inf = sm.info[h], n = inf & 0xFFFFu;
                uint32_t side = 0;
                if (h != ex) side = (__popc(inf & 0x7F0000u) > 1 ? 1u : 0u) | (__popc(inf & 0x3F800000u) > 1 ? 2u : 0u);
                uint32_t ni = n | (side << 14);
                if (side == 1u || side == 2u) {
                    const uint32_t p = atomicAdd(&sm.npool, 1u);
                    reinterpret_cast<uint4 *>(sm.u.b.pool)[p] = make_uint4(0, 0, 0, h << 16);
                    ni |= p << 16;
                }
                if (side != 3u && !((zeros >> j) & 1u) && (n >= 2u || singles)) {
                    ni |= GI_KEPT;
                    kept += n;
                    kept_here |= 1u << j;
                }
                sm.info[h] = ni;
            }
        }
        uint32_t x = kept;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(FULLG, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) sm.ws[warp] = x;
        __syncthreads();
        uint32_t at = x - kept, sums = lane < THREADS / 32 ? sm.ws[lane] : 0u;  // the warps', then up to each
#pragma unroll
        for (int o = 1; o < THREADS / 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(FULLG, sums, o);
            if (lane >= o) sums += y;
        }
        const uint32_t total = __shfl_sync(FULLG, sums, THREADS / 32 - 1), before = __shfl_sync(FULLG, sums, (warp + 31) & 31);
        at += warp ? before : 0u;
        if (tid == 0) sm.base = atomicAdd(&c.ctr[GC_OUT], total);
#pragma unroll
        for (int j = 0; j < ITEMS; j++) {
            if ((kept_here >> j) & 1u) {
                const uint32_t h = slot(j);
                sm.u.b.off[h] = (uint16_t)at;
                at += sm.info[h] & 0x3FFFu;
            }
        }
        // ---- code counts of the runs branching on one side; then code6: such a run's tuple (bit 3) and its code there, kept (4)
#pragma unroll
        for (int j = 0; j < ITEMS; j++) {
            if (j * THREADS + tid < cnt) {
                const uint32_t inf = sm.info[slot(j)], side = (inf >> 14) & 3u;
                const uint32_t code = side == 1u ? code6(j) & 7u : code6(j) >> 3;
                uint32_t v = inf & GI_KEPT ? 16u : 0u;
                if (side == 1u || side == 2u) {
                    v |= 8u | code;
                    if (code < 7u) atomicAdd(&sm.u.b.pool[((inf >> 16) & 0x1FFFu) * 4 + (code >> 1)], 1u << (16 * (code & 1)));
                }
                set_code6(j, v);
            }
        }
        __syncthreads();
        // ---- their judgement (metapart.c:2296-2451): the first code of the largest count, the second count's ratio
        for (uint32_t p = tid; p < sm.npool; p += THREADS) {
            const uint4 v = reinterpret_cast<const uint4 *>(sm.u.b.pool)[p];
            const uint32_t cc[7] = {v.x & 0xFFFFu, v.x >> 16, v.y & 0xFFFFu, v.y >> 16, v.z & 0xFFFFu, v.z >> 16, v.w & 0xFFFFu};
            uint32_t mx = 0, m1 = 0, m2 = 0;
#pragma unroll
            for (uint32_t q = 0; q < 7; q++) {
                const bool g = cc[q] > m1;
                m2 = g ? m1 : max(m2, cc[q]);
                mx = g ? q : mx;
                m1 = max(m1, cc[q]);
            }
            const uint32_t h = v.w >> 16, inf = sm.info[h];
            const uint32_t r = ratio_above_02_small(m2, inf & 0x3FFFu) ? 1u << 19 : 0u;
            sm.info[h] = (inf & (GI_KEPT | 0xFFFFu)) | (mx << 16) | r;
        }
        __syncthreads();
        // ---- marks, and the kept reads in their places
        uint32_t *stage = sm.u.b.pool;
#pragma unroll
        for (int j = 0; j < ITEMS; j++) {
            if (j * THREADS + tid < cnt) {
                const uint32_t h = slot(j), v = code6(j);
                if (v & 8u) {
                    const uint32_t inf = sm.info[h];
                    if ((v & 7u) != ((inf >> 16) & 7u) || (inf & (1u << 19))) {
                        c.parent[id[j]] = BAD;
                        c.filtered[id[j]] = 1;
                    }
                }
                if (v & 16u) stage[sm.u.b.off[h] + number(j)] = id[j] | (number(j) == 0 ? 0x80000000u : 0u);
            }
        }
        if (singles && tid == 0) {
            const uint32_t base = sm.base;
            if (total) {
                uint32_t *e = c.qlist + 3 * (size_t)atomicAdd(&c.ctr[GC_QLIST], 1u);
                e[0] = base;
                e[1] = total;
                e[2] = seg;
            }
            if (seg_last && ex != ~0u && (sm.info[ex] & GI_KEPT)) {
                c.quirk[seg * QW + 3] = base + sm.u.b.off[ex];
                c.quirk[seg * QW + 4] = sm.info[ex] & 0x3FFFu;
            }
        }
        __syncthreads();
        uint32_t *o = c.out + sm.base;
        for (uint32_t i = tid; i < total; i += THREADS) o[i] = stage[i];
    }
}
constexpr int GP_THREADS = 768, GP_ITEMS = 8;  // small blocks (k_group)
typedef GroupSmem<GP_THREADS, GP_ITEMS, 13> GroupSmemS;
typedef GroupSmem<1024, 12, 14> GroupSmemL;
static_assert(GP_CAP_S <= GroupSmemS::CAP && GP_CAP_L <= GroupSmemL::CAP, "a unit fits its block's slots");
static_assert(GP_CAP_S * 8 <= GroupSmemS::SLOTS * 6 && GP_CAP_L * 8 <= GroupSmemL::SLOTS * 6,
              "counters of half as many runs as tuples");
static_assert(2 * (sizeof(GroupSmemS) + 1024) <= 228 * 1024 && sizeof(GroupSmemL) <= 227 * 1024, "blocks per SM");

// ------------------------------------------------------------------ units above a block's capacity

struct BigUnit {
    uint32_t u, start, cnt, off;  // off: among the gathered tuples of its batch
};

__global__ void k_big_units(const uint32_t *big, uint32_t nb, const uint32_t *ustart, const uint32_t *ub0, uint32_t nunits,
                            const uint32_t *fill, bool ends_range, uint32_t *out)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nb) return;
    const uint32_t u = big[i];
    out[4 * i] = u;
    out[4 * i + 1] = ustart[u];
    out[4 * i + 2] = ustart[u + 1] - ustart[u];
    out[4 * i + 3] = (u + 1 == nunits ? ends_range : ub0[u + 1] >> 31) ? 1u : 0u;  // ends a thread range
    if (fill[u] != ustart[u + 1]) out[4 * i + 2] = 0;  // the histogram is not the tuples': the caller stops here
}

// Gathered keys: unit index << (2 (k - 10) + 8) | low k-mer bits << 8 | adjacency codes.
__global__ void k_gbig_gather(const BigUnit *bu, const uint64_t *kk, const uint32_t *ids, uint64_t *tk, uint32_t *tid, int bsh)
{
    const BigUnit b = bu[blockIdx.x];
    const uint64_t lowmask = (1ull << (bsh + 6)) - 1;
    for (uint32_t e = threadIdx.x + blockDim.x * blockIdx.y; e < b.cnt; e += blockDim.x * gridDim.y) {
        const uint64_t v = kk[b.start + e] & lowmask;
        tk[b.off + e] = ((uint64_t)blockIdx.x << (bsh + 8)) | ((v >> 6) << 8) | (v & 63u);
        tid[b.off + e] = ids[b.start + e];
    }
}

// The sorted units' ids into out, as k_group leaves them (a zeroed tuple or the zero k-mer's stands for no read, each a run
// of its own: nothing looks back through them).
__global__ void k_gbig_emit(const BigUnit *bu, const uint32_t *base, const uint64_t *tk, const uint32_t *tid, const uint32_t *z,
                            const uint32_t *ub0, uint32_t nunits, bool ends_scan, const uint32_t *lrs, int bsh, uint32_t *ctr,
                            uint32_t *qlist, uint32_t *quirk, uint32_t *out)
{
    const BigUnit b = bu[blockIdx.x];
    const uint32_t b0 = ub0[b.u] & 0x7FFFFFFFu, seg = b0 / NB, o = *base + b.off;
    const bool zero_bucket = (b0 & (NB - 1)) == 0;
    const uint64_t lowmask = (1ull << bsh) - 1;
    for (uint32_t e = threadIdx.x + blockDim.x * blockIdx.y; e < b.cnt; e += blockDim.x * gridDim.y) {
        const uint32_t i = b.off + e;
        const uint64_t km = tk[i] >> 8;
        const bool head = e == 0 || (tk[i - 1] >> 8) != km;
        const bool none = ((z[i >> 5] >> (i & 31)) & 1u) || (zero_bucket && (km & lowmask) == 0);
        out[o + e] = (none ? GP_NONE : tid[i]) | (head || none ? 0x80000000u : 0u);
    }
    if (blockIdx.y == 0 && threadIdx.x == 0 && b.start >= lrs[seg]) {
        uint32_t *q = qlist + 3 * (size_t)atomicAdd(&ctr[GC_QLIST], 1u);
        q[0] = o;
        q[1] = b.cnt;
        q[2] = seg;
        if (b.u + 1 == nunits ? ends_scan : (ub0[b.u + 1] & 0x7FFFFFFFu) / NB != seg) {  // the segment's last run
            const uint64_t km = tk[b.off + b.cnt - 1] >> 8;
            uint32_t a = b.off, y = b.off + b.cnt - 1;
            while (a < y) {
                const uint32_t m = (a + y) >> 1;
                if ((tk[m] >> 8) < km) a = m + 1; else y = m;
            }
            quirk[seg * QW + 3] = o + (a - b.off);
            quirk[seg * QW + 4] = b.off + b.cnt - a;
        }
    }
}

// first: the first batch of oversized units; their ids are out's last (GC_LONG).
__global__ void k_gbig_reserve(uint32_t *ctr, uint32_t n, uint32_t *base, bool first)
{
    *base = atomicAdd(&ctr[GC_OUT], n);
    if (first) ctr[GC_LONG] = *base;
}

// ------------------------------------------------------------------ unions

// The sweeps' initial state (metapart.c:2539-2548): a thread range's first valid tuple joins the scan's first
// read when it carries the scan's last k-mer, which only the last range with tuples can hold and only if no
// smaller k-mer of that range has a read that is not BAD.  Per segment, over the grouped stretches of its last
// range: [0] a read outside the last run, [1] one inside, [2] its id.
// A block looks at a segment's stretches until it or another has found a read outside, and asks for that once a stretch
// (asked for at every read by every thread, and set by every one that found it, the words of one segment were a queue: 245
// us of 20M reads' scans).
__global__ void __launch_bounds__(256) k_gp_quirk(const uint32_t *ctr, const uint32_t *qlist, const uint32_t *out,
                                                  const uint8_t *filtered, int nseg, uint32_t *quirk)
{
    volatile uint32_t *vq = quirk;
    const uint32_t nq = ctr[GC_QLIST];
    uint32_t known = ~0u;  // a segment with a read outside
    for (uint32_t q = blockIdx.x; q < nq; q += gridDim.x) {
        const uint32_t o = qlist[3 * (size_t)q], len = qlist[3 * (size_t)q + 1], seg = qlist[3 * (size_t)q + 2];
        if (seg != known) {
            const uint32_t l0 = quirk[seg * QW + 3], l1 = l0 + quirk[seg * QW + 4];
            bool found = __syncthreads_or(threadIdx.x == 0 && vq[seg * QW]);
            for (uint32_t i0 = 0; i0 < len && !found; i0 += blockDim.x) {
                const uint32_t i = i0 + threadIdx.x, id = i < len ? out[o + i] & 0x7FFFFFFFu : GP_NONE;
                const bool good = id != GP_NONE && !filtered[id], in = o + i >= l0 && o + i < l1;
                if (good && in) {
                    quirk[seg * QW + 2] = id;
                    quirk[seg * QW + 1] = 1;
                }
                found = __syncthreads_or(good && !in);
                if (found && threadIdx.x == 0) quirk[seg * QW] = 1;
            }
            if (found) known = seg;
        }
        if (nseg == 1 && known == seg) return;
    }
}

constexpr uint32_t GE_SEG = 1024;  // most grouped ids per warp and turn
constexpr uint32_t GE_BLOCKS = 8;   // blocks per SM

// Whether a stretch among the oversized units' ids has neither a run's start nor a read that is not BAD: k_gp_union passes by
// it when it looks for a read of a run that began earlier.  A run of a few million tuples whose reads are all BAD (the inner
// k-mers of an adapter, when its ends' branches make its reads BAD) was looked through from every stretch of it: 2M reads, 33
// runs of 1.8M, the unions 142 -> 0.8 ms.
__global__ void __launch_bounds__(256) k_gp_blank(const uint32_t *ctr, const uint32_t *__restrict__ out,
                                                  const uint8_t *__restrict__ filtered, uint32_t per, uint8_t *blank)
{
    const uint32_t m = ctr[GC_OUT], first = (ctr[GC_LONG] + per - 1) / per, nseg = (m + per - 1) / per;
    const int lane = threadIdx.x & 31;
    const uint32_t nw = (gridDim.x * blockDim.x) >> 5;
    for (uint32_t sgm = first + ((blockIdx.x * blockDim.x + threadIdx.x) >> 5); sgm < nseg; sgm += nw) {
        const uint32_t p0 = sgm * per, p1 = min(m, p0 + per);
        bool some = false;
        for (uint32_t p = p0; p < p1 && !some; p += 32) {
            const uint32_t v = p + lane < p1 ? out[p + lane] : GP_NONE, id = v & 0x7FFFFFFFu;
            some = __any_sync(FULLG, (v >> 31) || (id != GP_NONE && !filtered[id]));
        }
        if (lane == 0) blank[sgm] = !some;
    }
}

// Bound by the random reads of the BAD flags and parents in L2.  It reads 4 bytes per joining tuple where the
// sweep over sorted tuples read 13 per tuple: 6.2 ms against 21.0 at 20M x 150 bp, 2 scans.
//
// The unions of every k-mer's reads (metapart.c:2537-2727): each read that is not BAD joins its k-mer's first one
// of the stretch.  A stretch that starts inside a run looks back for one read of it, so long runs are shared by
// many warps (at most a large block's tuples back, or past stretches known to be blank: k_gp_blank; null without oversized
// units).
__global__ void __launch_bounds__(256) k_gp_union(const uint32_t *ctr, const uint32_t *__restrict__ out, uint32_t *parent,
                                                  const uint8_t *__restrict__ filtered, const uint8_t *__restrict__ blank,
                                                  uint32_t per, uint32_t *err, uint32_t uf_cap)
{
    const uint32_t m = ctr[GC_OUT];
    const int lane = threadIdx.x & 31;
    const uint32_t le = (lane == 31) ? FULLG : ((2u << lane) - 1);
    const uint32_t nw = (gridDim.x * blockDim.x) >> 5, nseg = (m + per - 1) / per;
    for (uint32_t sgm = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; sgm < nseg; sgm += nw) {
        const uint32_t p0 = sgm * per, p1 = min(m, p0 + per);
        bool has = false;
        uint32_t anchor = 0;
        if (!(out[p0] >> 31)) {  // the run's reads before the stretch, a window at a time
            uint32_t back = sgm;
            if (blank) {
                const uint32_t first = (ctr[GC_LONG] + per - 1) / per;
                for (uint32_t n = 32; n == 32 && back > first;) {
                    const uint32_t some = __ballot_sync(FULLG, back < first + 1 + lane || !blank[back - 1 - lane]);
                    n = some ? (uint32_t)__ffs(some) - 1 : 32u;
                    back -= n;
                }
            }
            for (uint32_t q = back * per; q >= 32;) {
                q -= 32;
                const uint32_t v = out[q + lane], id = v & 0x7FFFFFFFu;
                const uint32_t H = __ballot_sync(FULLG, v >> 31);
                uint32_t G = __ballot_sync(FULLG, id != GP_NONE && !filtered[id]);
                if (H) G &= FULLG << (31 - __clz(H));
                if (G) {
                    has = true;
                    anchor = __shfl_sync(FULLG, id, __ffs(G) - 1);
                }
                if (H || G) break;
            }
        }
        uint32_t nv = p0 + lane < p1 ? out[p0 + lane] : 0x80000000u | GP_NONE;
        for (uint32_t p = p0; p < p1; p += 32) {
            const uint32_t v = nv, id = v & 0x7FFFFFFFu;
            nv = p + 32 + lane < p1 ? out[p + 32 + lane] : 0x80000000u | GP_NONE;
            const bool good = id != GP_NONE && !filtered[id];
            const uint32_t H = __ballot_sync(FULLG, v >> 31), G = __ballot_sync(FULLG, good);
            const int s = (H & le) ? 31 - __clz(H & le) : -1;  // the lane that starts this lane's run (-1: carried in)
            const uint32_t before = G & le & (s >= 0 ? FULLG << s : FULLG);
            const int fg = before ? __ffs(before) - 1 : lane;  // the run's first read here
            const uint32_t a = __shfl_sync(FULLG, id, fg);
            const bool carried = s < 0 && has;
            const uint32_t target = carried ? anchor : a;
            if (good && (carried || lane != fg) && target != id) uf_union(parent, target, id, err, uf_cap);
            const uint32_t tail = H ? G & (FULLG << (31 - __clz(H))) : G;  // reads of the run open at the window's end
            if (H || !has) {
                has = tail != 0;
                anchor = __shfl_sync(FULLG, id, tail ? __ffs(tail) - 1 : 0);
            }
        }
    }
}

// The first tuple in (k-mer, adjacency, position) order, in three reductions over best: [0] high k-mer byte and
// the bits of lo above it do not fit one word, so (hi, lo) is taken as hi first, then lo, then the position.
__global__ void k_first_pass(const uint64_t *lo, const uint8_t *hi, uint64_t n, int step, unsigned long long *best)
{
    unsigned long long v = ~0ull;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        const unsigned long long h = hi ? hi[i] : 0;
        if (step == 0) v = min(v, h);
        else if (h == best[0] && step == 1) v = min(v, (unsigned long long)lo[i]);
        else if (h == best[0] && lo[i] == best[1] && step == 2) v = min(v, (unsigned long long)i);
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) v = min(v, __shfl_xor_sync(FULLG, v, o));
    if ((threadIdx.x & 31) == 0 && v != ~0ull) atomicMin(&best[step], v);
}

__global__ void k_join_pair(uint32_t *parent, uint32_t a, uint32_t b, uint32_t *err, uint32_t uf_cap)
{
    if (a != b) uf_union(parent, a, b, err, uf_cap);
}

// ------------------------------------------------------------------ host side

static unsigned blocks_of(uint64_t n, int t) { return (unsigned)((n + t - 1) / t); }

// A scan takes the grouped path when its tuple positions fit 32 bits and its read ids 31.
bool group_fits(uint64_t n, uint64_t n_reads, const SortSegments *segs)
{
    return n >= 1 && n <= GROUP_MAX_TUPLES && n_reads < GROUP_MAX_READS && (!segs || segs->nseg < 2048);
}

static void group_kernel_attrs()
{
    static std::once_flag once[64];
    int dev = 0;
    cudaGetDevice(&dev);
    std::call_once(once[dev & 63], [] {
        for (auto f : {k_split_reads<true, SR_ONE>, k_split_reads<false, SR_ONE>, k_split_reads<true, SR_MERGED>, k_split_reads<false, SR_MERGED>,
                       k_split_reads<true, SR_SEGMENTS>, k_split_reads<false, SR_SEGMENTS>})
            cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(BinSmem));
        cudaFuncSetAttribute(k_split_tuples, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(SplitSmem));
        cudaFuncSetAttribute(k_split_units, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(UnitSmem));
        cudaFuncSetAttribute(k_group<GP_THREADS, GP_ITEMS, 13>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(GroupSmemS));
        cudaFuncSetAttribute(k_group<1024, 12, 14>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(GroupSmemL));
    });
}

int group_plan(GroupScan &g, DeviceArena &arena, cudaStream_t st)
{
    const int nseg = (int)g.seg_tstart.size() - 1;
    const uint32_t nbounds = (uint32_t)g.bounds.size();
    const uint64_t nbk = g.hi - g.lo;
    // host side of the plan: every segment's bins and the first tuple of its last range with tuples
    std::vector<uint32_t> &h = g.h_plan;
    h.assign(3 * (size_t)nseg + 1, 0);
    uint32_t *bin0 = h.data(), *sh = bin0 + nseg + 1, *lrs = sh + nseg;
    for (int q = 0, t = 0; q < nseg; q++) {
        const uint64_t n = g.seg_tstart[q + 1] - g.seg_tstart[q], span = nseg > 1 ? (uint64_t)NB : nbk;
        sh[q] = g.merged ? (uint32_t)g.merged->sh : (uint32_t)bin_width(n, span);
        bin0[q + 1] = bin0[q] + (uint32_t)((g.merged ? g.hi - 1 - g.anchor : span - 1) >> sh[q]) + 1;
        uint64_t b = g.seg_tstart[q];
        for (; t < (int)nbounds && g.bounds[t] < g.seg_tstart[q + 1]; t++) b = std::max(b, g.bounds[t]);
        lrs[q] = g.part ? g.last_range : (uint32_t)b;
    }
    g.bins = bin0[nseg];
    g.seg_lo = nseg > 1 ? 0u : (uint32_t)(g.merged ? g.anchor : g.lo);
    // units: a start per thread range, segment and bin, and at most two per 2^GP_UNIT_SHIFT tuples
    g.max_units = 2 * (uint32_t)(g.n >> GP_UNIT_SHIFT) + nbounds + g.bins + 2u * (uint32_t)nseg + 8;
    g.max_tiles = (uint32_t)(g.n / SP_TILE) + g.bins + 1;
    const uint32_t nblk = blocks_of(nbk, GP_COUNT_BLOCK);
    const size_t brk_words = nbk / 32 + 1;
    uint32_t *brk = arena.alloc<uint32_t>(brk_words + GC_N + (size_t)nseg * QW);
    uint64_t *blk = arena.alloc<uint64_t>(nblk), *d_bounds = arena.alloc<uint64_t>(nbounds);
    g.ustart = arena.alloc<uint32_t>(3 * (size_t)(g.max_units + 1));
    g.bstart = arena.alloc<uint32_t>(5 * (size_t)(g.bins + 1));
    g.unit_of = arena.alloc<uint32_t>(nbk);
    g.seg_bin0 = arena.alloc<uint32_t>(h.size());
    g.tiles = arena.alloc<uint4>(g.max_tiles);
    g.mid = arena.alloc<uint32_t>(2 * (size_t)(g.n / GP_CAP_S + 1));
    g.qlist = arena.alloc<uint32_t>(3 * (size_t)(g.max_units + 1));
    if (!brk || !blk || !d_bounds || !g.ustart || !g.bstart || !g.seg_bin0 || !g.tiles || !g.mid || !g.qlist || !g.unit_of)
        return set_error(MP_ENOMEM, "device memory for the scan's plan");
    g.ub0 = g.ustart + g.max_units + 1;
    g.ucur = g.ub0 + g.max_units + 1;
    g.bu0 = g.bstart + g.bins + 1;
    g.bcur = g.merged ? g.merged->cur + g.digit0 : g.bu0 + g.bins + 1;
    g.bin_sh = g.bu0 + 2 * (size_t)(g.bins + 1);
    g.bfirst = g.bin_sh + g.bins + 1;
    g.seg_sh = g.seg_bin0 + nseg + 1;
    g.lrs = g.seg_sh + nseg;
    g.big = g.mid + g.n / GP_CAP_S + 1;
    g.ctr = brk + brk_words;
    g.quirk = g.ctr + GC_N;
    MP_CUDA(cudaMemsetAsync(brk, 0, (brk_words + GC_N + (size_t)nseg * QW) * 4, st));
    MP_CUDA(cudaMemcpyAsync(d_bounds, g.bounds.data(), nbounds * 8, cudaMemcpyHostToDevice, st));
    MP_CUDA(cudaMemcpyAsync(g.seg_bin0, h.data(), h.size() * 4, cudaMemcpyHostToDevice, st));
    const PlanCtx c{g.d_hist, g.lo, g.hi, brk, g.seg_sh, g.seg_bin0, g.seg_lo};
    (count_launch(), k_gp_marks<<<blocks_of(nbounds, 4), 128, 0, st>>>(g.d_hist, g.lo, g.hi, d_bounds, (int)nbounds, brk));
    (count_launch(), k_gp_count<<<nblk, GP_COUNT_BLOCK, 0, st>>>(c, blk, g.ctr));
    (count_launch(), k_gp_scan<<<1, 1024, 0, st>>>(blk, nblk, (uint32_t)g.n, g.bins, g.ctr, g.ustart, g.bstart, g.bu0));
    (count_launch(), k_gp_write<<<nblk, GP_COUNT_BLOCK, 0, st>>>(c, blk, g.ctr, g.ustart, g.ub0, g.ucur, g.bstart, g.bu0,
                                                                  g.merged ? nullptr : g.bcur, g.bin_sh, g.bfirst, g.unit_of, g.mid, g.big));
    (count_launch(), k_gp_tiles<<<std::min(32u, g.max_tiles / 2048 + 1), 1024, 0, st>>>(g.bstart, g.bins, g.ctr, g.tiles));
    ReadBack<uint32_t> rb(arena, GC_N, PLAN_MAIL);
    if (!arena.mail) {
        g.h_ctr.assign(GC_N, 0);
        rb.p = g.h_ctr.data();
    }
    if (!g.planned) MP_CUDA(cudaEventCreateWithFlags(&g.planned, cudaEventDisableTiming));
    MP_CUDA(cudaMemcpyAsync(rb.p, g.ctr, GC_N * 4, cudaMemcpyDeviceToHost, st));
    MP_CUDA(cudaEventRecord(g.planned, st));
    MP_CUDA(cudaGetLastError());
    return 0;
}

// The plan's counters, once they have arrived (the split passes run meanwhile).
static int group_counts(GroupScan &g, DeviceArena &arena)
{
    MP_CUDA(cudaEventSynchronize(g.planned));
    const uint32_t *p = arena.mail ? reinterpret_cast<const uint32_t *>(arena.mail + PLAN_MAIL) : g.h_ctr.data();
    std::copy(p, p + GC_N, g.hctr);
    return 0;
}

// seg_shape: every segment's tiling of its reads (null: c.t for all).
static int launch_bins(GroupScan &g, BinCtx &c, const std::vector<uint64_t> &seg_start, const std::vector<uint32_t> *seg_shape,
                       DeviceArena &arena, cudaStream_t st)
{
    group_kernel_attrs();
    const int nseg = (int)g.seg_tstart.size() - 1;
    const bool reads = c.lo == nullptr;
    const uint32_t per = reads ? c.t.rpt : (uint32_t)SP_TILE;
    c.tiles = blocks_of(reads ? c.n_reads : g.n, (int)per);
    if (nseg > 1) {
        std::vector<uint32_t> &h = g.h_tiles;
        const size_t shapes = seg_shape ? 4 * (size_t)nseg : 0;  // first: they are read 16 bytes at a time
        h.assign(shapes + 2 * (size_t)nseg + 2, 0);
        c.tiles = 0;
        for (int q = 0; q <= nseg; q++) {
            h[shapes + q] = c.tiles;
            h[shapes + nseg + 1 + q] = (uint32_t)seg_start[q];
            if (q < nseg) c.tiles += blocks_of(seg_start[q + 1] - seg_start[q], seg_shape ? (int)(*seg_shape)[4 * q + 3] : (int)per);
        }
        if (seg_shape) std::copy(seg_shape->begin(), seg_shape->end(), h.begin());
        uint32_t *d = arena.alloc<uint32_t>(h.size() + c.tiles);
        if (!d) return set_error(MP_ENOMEM, "device memory for the scan's tiles");
        MP_CUDA(cudaMemcpyAsync(d, h.data(), h.size() * 4, cudaMemcpyHostToDevice, st));
        if (shapes) c.sg.shape = reinterpret_cast<const uint4 *>(d);
        c.sg.tile0 = d + shapes;
        c.sg.start = d + shapes + nseg + 1;
        c.sg.tile_seg = d + h.size();
        (count_launch(), k_gp_segtiles<<<nseg, 256, 0, st>>>(d + shapes, nseg, d + h.size()));
    }
    c.n = (uint32_t)g.n;
    c.bsh = 2 * (g.k - 10);
    c.k_lo = (uint64_t)g.seg_lo << c.bsh;
    c.k_span = (nseg > 1 ? (uint64_t)NB : g.hi - g.lo) << c.bsh;
    c.seg_bin0 = g.seg_bin0;
    c.seg_sh = g.seg_sh;
    c.bcur = g.bcur;
    c.err = g.ctr + GC_ERR;
    uint32_t least = 16;  // the narrowest bins
    for (int q = 0; q < nseg; q++) least = std::min(least, g.h_plan[(size_t)nseg + 1 + q]);
    const bool high = g.k >= 17 && c.bsh + (int)least >= 32;
    auto kern = !reads        ? k_split_tuples
                : c.sg.shape ? (high ? k_split_reads<true, SR_SEGMENTS> : k_split_reads<false, SR_SEGMENTS>)
                             : (high ? k_split_reads<true, SR_ONE> : k_split_reads<false, SR_ONE>);
    const unsigned blocks = std::min<unsigned>(c.tiles, 2u * (unsigned)sm_count());
    if (blocks) (count_launch(), kern<<<blocks, SP_THREADS, reads ? sizeof(BinSmem) : sizeof(SplitSmem), st>>>(c));
    MP_CUDA(cudaGetLastError());
    return 0;
}

int group_bins_reads(GroupScan &g, const uint8_t *fq, const ParsedReads &pr, const std::vector<uint64_t> &seg_reads,
                     const uint32_t *label, uint64_t *k1, uint32_t *id1, DeviceArena &arena, cudaStream_t st,
                     const std::vector<uint32_t> &seg_len)
{
    std::vector<uint32_t> shape;
    for (uint32_t n : seg_len) {
        const ReadTiles t = read_tiles(fq, pr, g.k, std::max(n, 1u), SP_THREADS, SP_PACKED);
        shape.insert(shape.end(), {t.P, t.spr, t.rounds, t.rpt});
    }
    BinCtx c;
    c.t = read_tiles(fq, pr, g.k, pr.max_len, SP_THREADS, SP_PACKED);
    c.n_reads = (uint32_t)pr.n_reads;
    c.check_many = pr.max_len > (uint32_t)g.k + 254u;  // a read with 256 positions or more
    c.label = label;
    c.out_k = k1;
    c.out_id = id1;
    return launch_bins(g, c, seg_reads, shape.empty() ? nullptr : &shape, arena, st);
}

int group_bins_tuples(GroupScan &g, const uint64_t *lo, const uint8_t *hi, const uint32_t *id, uint64_t *k1, uint32_t *id1,
                      DeviceArena &arena, cudaStream_t st)
{
    BinCtx c;
    c.lo = lo;
    c.hi = hi;
    c.id = id;
    c.out_k = k1;
    c.out_id = id1;
    return launch_bins(g, c, g.seg_tstart, nullptr, arena, st);
}

// The first tuple of every bin of the merged scans.
__global__ void k_gp_cursors(const uint64_t *hist, uint64_t lo, uint64_t hi, int sh, uint64_t s1, uint64_t s2, uint32_t digits,
                             uint32_t *cur)
{
    const uint32_t d = blockIdx.x * blockDim.x + threadIdx.x;
    if (d >= digits) return;
    uint32_t s = 0;
    uint64_t first = lo;  // of the digit's scan
    if (s1 < hi && d >= (uint32_t)((s1 - lo) >> sh) + 1) s = 1, first = s1;
    if (s2 < hi && d >= (uint32_t)((s2 - lo) >> sh) + 2) s = 2, first = s2;
    const uint64_t b = max(first, lo + ((uint64_t)(d - s) << sh));
    cur[d] = (uint32_t)(hist[min(b, hi)] - hist[lo]);
}

bool group_merge(MergedScans &m, const uint64_t *hist, const std::vector<uint32_t> &scan, uint32_t max_len, int k)
{
    const int S = (int)scan.size() - 1;
    if (S < 2 || S > GROUP_MAX_MERGED || max_len > (uint32_t)k + 254u) return false;
    int small = 0;
    bool large = false;
    for (int s = 0; s < S; s++) {
        if (scan[s] >= scan[s + 1]) return false;
        const uint64_t n = hist[scan[s + 1]] - hist[scan[s]];
        small = std::max(small, bin_width(n, scan[s + 1] - scan[s]));
        large |= n > GP_SMALL;
    }
    m.scan = scan;
    m.n = hist[scan[S]] - hist[scan[0]];
    m.sh = large ? 10 : small;
    m.digits = ((scan[S] - 1 - scan[0]) >> m.sh) + (uint32_t)S;
    return m.digits <= GP_DIGITS + SP_EXTRA && m.n >= 1 && m.n <= GROUP_MAX_TUPLES;
}

int group_bins_scans(MergedScans &m, const uint64_t *d_hist, int k, const uint8_t *fq, const ParsedReads &pr, cudaStream_t st)
{
    group_kernel_attrs();
    const int S = (int)m.scan.size() - 1;
    const uint64_t lo = m.scan[0], hi = m.scan[S];
    (count_launch(), k_gp_cursors<<<blocks_of(m.digits, 256), 256, 0, st>>>(d_hist, lo, hi, m.sh, m.scan[1], S > 2 ? m.scan[2] : hi,
                                                                           m.digits, m.cur));
    BinCtx c;
    c.t = read_tiles(fq, pr, k, pr.max_len, SP_THREADS, SP_PACKED);
    c.n_reads = (uint32_t)pr.n_reads;
    c.out_k = m.k1;
    c.out_id = m.id1;
    c.n = (uint32_t)m.n;
    c.tiles = blocks_of(c.n_reads, (int)c.t.rpt);
    c.bsh = 2 * (k - 10);
    c.k_lo = lo << c.bsh;
    c.k_span = (hi - lo) << c.bsh;
    c.bcur = m.cur;
    c.m_digits = m.digits;
    c.m_sh = (uint32_t)m.sh;
    for (int s = 1; s < S; s++) c.m_start[s - 1] = (m.scan[s] - lo) << c.bsh;
    auto kern = k >= 17 && c.bsh + m.sh >= 32 ? k_split_reads<true, SR_MERGED> : k_split_reads<false, SR_MERGED>;
    const unsigned blocks = std::min<unsigned>(c.tiles, 2u * (unsigned)sm_count());
    if (blocks) (count_launch(), kern<<<blocks, SP_THREADS, sizeof(BinSmem), st>>>(c));
    MP_CUDA(cudaGetLastError());
    return 0;
}

void group_take(GroupScan &g, const MergedScans &m, int s, const uint32_t *label, const std::vector<uint64_t> &tuple0)
{
    const uint64_t rel = g.lo - m.scan[0];
    g.merged = &m;
    g.anchor = m.scan[0] + (rel >> m.sh << m.sh);
    g.digit0 = (uint32_t)(rel >> m.sh) + (uint32_t)s;
    g.tuple0 = (uint32_t)tuple0[s];
    g.late_label = s ? label : nullptr;
}

int group_units(GroupScan &g, const uint64_t *k1, const uint32_t *id1, uint64_t *k2, uint32_t *id2, cudaStream_t st)
{
    (count_launch(), k_split_units<<<std::min(g.max_tiles, 2u * (unsigned)sm_count()), SP_THREADS, sizeof(UnitSmem), st>>>(
        k1, id1, (uint32_t)g.n, 2 * (g.k - 10), g.seg_lo, g.ctr, g.bins, g.bstart, g.bfirst, g.bu0, g.bcur, g.bin_sh, g.ub0,
        g.ucur, g.unit_of, (uint32_t)(g.hi - g.lo), g.tiles, g.tuple0, g.late_label, k2, id2));
    MP_CUDA(cudaGetLastError());
    return 0;
}

int group_filter(GroupScan &g, const uint64_t *kk, const uint32_t *ids, uint32_t *out, uint32_t *parent, uint8_t *filtered,
                 DeviceArena &arena, cudaStream_t st)
{
    group_kernel_attrs();
    if (const int rc = group_counts(g, arena)) return rc;
    const uint32_t *fill = g.ucur;
    GroupCtx c{kk, ids, g.ustart, g.ub0, fill, g.lrs, nullptr, g.ctr, g.qlist, g.quirk, GC_WORK_S, GC_UNITS,
               g.ends_range, g.ends_scan, 0, (uint32_t)GP_CAP_S, out, parent, filtered};
    const unsigned sms = (unsigned)sm_count();
    (count_launch(), k_group<GP_THREADS, GP_ITEMS, 13><<<std::min(2 * sms, std::max(1u, g.hctr[GC_UNITS])), GP_THREADS, sizeof(GroupSmemS), st>>>(c));
    if (g.hctr[GC_MID]) {
        c.list = g.mid;
        c.work = GC_WORK_L;
        c.count = GC_MID;
        c.cap_lo = (uint32_t)GP_CAP_S;
        c.cap_hi = (uint32_t)GP_CAP_L;
        (count_launch(), k_group<1024, 12, 14><<<std::min(sms, g.hctr[GC_MID]), 1024, sizeof(GroupSmemL), st>>>(c));
    }
    const uint32_t nb = g.hctr[GC_BIG];
    if (nb) {
        // units above GP_CAP_L: gathered, sorted device-wide, judged as runs of the sorted tuples
        const int bsh = 2 * (g.k - 10), lowbits = bsh + 8;
        uint32_t *d_l = arena.alloc<uint32_t>(4 * (size_t)nb);
        BigUnit *d_b = arena.alloc<BigUnit>(nb);
        uint32_t *d_base = arena.alloc<uint32_t>(1);
        if (!d_l || !d_b || !d_base) return set_error(MP_ENOMEM, "device memory for oversized buckets");
        (count_launch(), k_big_units<<<blocks_of(nb, 128), 128, 0, st>>>(g.big, nb, g.ustart, g.ub0, g.hctr[GC_UNITS], fill,
                                                                        g.ends_range, d_l));
        std::vector<uint32_t> hl(4 * (size_t)nb);
        MP_CUDA(cudaMemcpyAsync(hl.data(), d_l, hl.size() * 4, cudaMemcpyDeviceToHost, st));
        MP_CUDA(cudaStreamSynchronize(st));
        for (size_t i = 0; i < nb; i++)
            if (hl[4 * i + 2] == 0) return set_error(MP_EFMT, "the histogram does not match the scan's tuples");
        const size_t per_batch = lowbits >= 44 ? ((size_t)1 << (64 - lowbits)) : ((size_t)1 << 20);
        std::vector<BigUnit> hb(nb);
        uint64_t most = 0;
        for (size_t b0 = 0; b0 < nb; b0 += per_batch) {
            uint64_t acc = 0;
            for (size_t i = b0; i < nb && i < b0 + per_batch; i++) {
                hb[i] = BigUnit{hl[4 * i], hl[4 * i + 1], hl[4 * i + 2], (uint32_t)acc};
                acc += hb[i].cnt;
            }
            most = std::max(most, acc);
        }
        MP_CUDA(cudaMemcpyAsync(d_b, hb.data(), nb * sizeof(BigUnit), cudaMemcpyHostToDevice, st));
        SortBufs t;
        for (int q = 0; q < 2; q++) {
            t.lo[q] = arena.alloc<uint64_t>(most + 1);
            t.id[q] = arena.alloc<uint32_t>(most + 1);
            if (!t.lo[q] || !t.id[q]) return set_error(MP_ENOMEM, "device memory for oversized buckets");
        }
        for (size_t b0 = 0; b0 < nb; b0 += per_batch) {
            const size_t b1 = std::min<size_t>(nb, b0 + per_batch);
            std::vector<uint64_t> ends{0};
            uint64_t acc = 0;
            for (size_t i = b0; i < b1; i++) {
                acc += hb[i].cnt;
                if (hl[4 * i + 3]) ends.push_back(acc);
            }
            const dim3 grid((unsigned)(b1 - b0), 16);
            t.cur = 0;
            (count_launch(), k_gbig_gather<<<grid, 256, 0, st>>>(d_b + b0, kk, ids, t.lo[0], t.id[0], bsh));
            int rc = radix_sort(t, acc, false, arena, st, nullptr);
            if (rc) return rc;
            Tuples tp;
            tp.lo = t.lo[t.cur];
            tp.id = t.id[t.cur];
            tp.n = acc;
            if ((rc = filter_scan(tp, ends, parent, filtered, arena, st, false))) return rc;
            (count_launch(), k_gbig_reserve<<<1, 1, 0, st>>>(g.ctr, (uint32_t)acc, d_base, b0 == 0));
            (count_launch(), k_gbig_emit<<<grid, 256, 0, st>>>(d_b + b0, d_base, tp.lo, tp.id, tp.z, g.ub0, g.hctr[GC_UNITS], g.ends_scan, g.lrs,
                                                              bsh, g.ctr, g.qlist, g.quirk, out));
            MP_CUDA(cudaStreamSynchronize(st));  // ends is this turn's
        }
    }
    MP_CUDA(cudaGetLastError());
    return 0;
}

int group_union(GroupScan &g, const uint32_t *out, uint32_t *parent, const uint8_t *filtered, uint64_t n_reads,
                DeviceArena &arena, cudaStream_t st, std::vector<GroupQuirk> &open)
{
    const int nseg = (int)g.seg_tstart.size() - 1;
    open.clear();
    (count_launch(), k_gp_quirk<<<std::min(2u * (unsigned)sm_count(), g.hctr[GC_UNITS] / 16 + 1), 256, 0, st>>>(g.ctr, g.qlist, out, filtered, nseg,
                                                                                                            g.quirk));
    // a stretch for every warp there is room for, of whole windows (600 reads: stretches of 1024 ids on a few
    // warps took 23 us, of 32 take 6)
    const uint64_t warps = 8ull * GE_BLOCKS * (uint64_t)sm_count();
    const uint32_t per = std::min(GE_SEG, ((uint32_t)(g.n / warps) + 63u) / 32u * 32u);
    const unsigned blocks = std::min<unsigned>(GE_BLOCKS * (unsigned)sm_count(), blocks_of(g.n, (int)per * 8));
    uint32_t *err = arena.alloc<uint32_t>(1);
    uint8_t *blank = g.hctr[GC_BIG] ? arena.alloc<uint8_t>(g.n / per + 1) : nullptr;
    if (!err || (g.hctr[GC_BIG] && !blank)) return set_error(MP_ENOMEM, "device memory");
    MP_CUDA(cudaMemsetAsync(err, 0, 4, st));
    if (blank) (count_launch(), k_gp_blank<<<blocks, 256, 0, st>>>(g.ctr, out, filtered, per, blank));
    (count_launch(), k_gp_union<<<blocks, 256, 0, st>>>(g.ctr, out, parent, filtered, blank, per, err, arena.lim.union_retries));
    compress_parents(parent, n_reads, st);
    const size_t words = GC_N + (size_t)nseg * QW;
    ReadBack<uint32_t> h(arena, words + 1);
    MP_CUDA(cudaMemcpyAsync(h.p, g.ctr, words * 4, cudaMemcpyDeviceToHost, st));
    MP_CUDA(cudaMemcpyAsync(h.p + words, err, 4, cudaMemcpyDeviceToHost, st));
    MP_CUDA(cudaStreamSynchronize(st));
    MP_CUDA(cudaGetLastError());
    const uint32_t herr = h[words];
    if (h[GC_ERR] & 4u)
        return set_error(MP_EUNSUP, "a read has 256 or more k-mers in one scan (the reference counts them in 8 bits, "
                                    "enumerateKmers.c:152)");
    if (h[GC_ERR] & 2u) return set_error(MP_EFMT, "the histogram does not match the scan's tuples");
    if (herr) return set_error(MP_EDEVICE, "union-find retry limit reached (flags 0x%x)", herr);
    for (int q = 0; q < nseg; q++) {
        const uint32_t *w = h.p + GC_N + (size_t)q * QW;
        g.outside = w[0];
        g.inside = w[1];
        g.anchor_read = w[2];
        if (!w[0] && w[1]) open.push_back(GroupQuirk{q, w[2]});
    }
    return 0;
}

int first_tuple_id(const uint64_t *lo, const uint8_t *hi, const uint32_t *id, uint64_t n, DeviceArena &arena, cudaStream_t st,
                   uint32_t *out)
{
    unsigned long long *best = arena.alloc<unsigned long long>(3);
    if (!best) return set_error(MP_ENOMEM, "device memory");
    MP_CUDA(cudaMemsetAsync(best, 0xFF, 24, st));
    const unsigned blocks = std::min<unsigned>(4u * (unsigned)sm_count(), blocks_of(n, 256));
    for (int s = 0; s < 3; s++) (count_launch(), k_first_pass<<<blocks, 256, 0, st>>>(lo, hi, n, s, best));
    unsigned long long h[3];
    MP_CUDA(cudaMemcpyAsync(h, best, 24, cudaMemcpyDeviceToHost, st));
    MP_CUDA(cudaStreamSynchronize(st));
    if (h[2] >= n) return set_error(MP_EDEVICE, "the scan's first tuple was not found");
    MP_CUDA(cudaMemcpyAsync(out, id + h[2], 4, cudaMemcpyDeviceToHost, st));
    MP_CUDA(cudaStreamSynchronize(st));
    return 0;
}

int group_finish(uint32_t *parent, uint64_t n_reads, uint32_t first, uint32_t anchor, DeviceArena &arena, cudaStream_t st,
                 uint32_t *hooked)
{
    uint32_t *w = arena.alloc<uint32_t>(3);  // error flags, the anchor run's read, the hooked read
    if (!w) return set_error(MP_ENOMEM, "device memory");
    uint32_t h[3] = {0, anchor, ~0u}, p = 0;
    MP_CUDA(cudaMemcpyAsync(w, h, sizeof h, cudaMemcpyHostToDevice, st));
    MP_CUDA(cudaMemcpyAsync(&p, parent + first, 4, cudaMemcpyDeviceToHost, st));
    MP_CUDA(cudaStreamSynchronize(st));
    if (p == BAD) hook_bad_anchor(parent, first, w + 1, w + 2, st);
    else (count_launch(), k_join_pair<<<1, 1, 0, st>>>(parent, first, anchor, w, arena.lim.union_retries));
    compress_parents(parent, n_reads, st);
    MP_CUDA(cudaMemcpyAsync(h, w, sizeof h, cudaMemcpyDeviceToHost, st));
    MP_CUDA(cudaStreamSynchronize(st));
    MP_CUDA(cudaGetLastError());
    if (h[0]) return set_error(MP_EDEVICE, "union-find retry limit reached (flags 0x%x)", h[0]);
    *hooked = h[2];
    return 0;
}

}  // namespace mp
