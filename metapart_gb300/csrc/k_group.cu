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
#include <vector>

#include "k_group.cuh"
#include "k_readtile.cuh"

namespace mp {

constexpr unsigned FULLG = 0xFFFFFFFFu;

// ------------------------------------------------------------------ plan

constexpr int GP_UNIT_SHIFT = 12;        // units end where the tuple prefix crosses a multiple of 4096
constexpr int GP_CAP_S = 6128;           // most tuples of a unit for the 512-thread blocks (two per SM)
constexpr int GP_CAP_L = 12288;          // and for the 1024-thread blocks; a larger bucket takes the device-wide sort
constexpr uint32_t GP_MAX_BINS = 1024;   // digits of the first split pass
constexpr uint32_t GP_MAX_UNITS = 2048;  // digits of the second (units of a bin), up to a bin shift of 21
constexpr uint32_t GP_MAX_UNITS_L = 4096;  // and above it (scans of more than 2^31 tuples; one block per SM)
constexpr int GP_COUNT_ITEMS = 8, GP_COUNT_THREADS = 256, GP_COUNT_BLOCK = GP_COUNT_ITEMS * GP_COUNT_THREADS;
constexpr uint32_t GP_NONE = 0x7FFFFFFFu;  // a grouped id that stands for no read
constexpr int QW = 8;  // words per segment: tuples found before the last run, last run's, its read, the run's place

struct PlanCtx {
    const uint64_t *hist;
    uint64_t lo, hi;         // buckets of the scan
    const uint32_t *brk;     // a bit per bucket (from lo): a thread range starts there
    int unit_shift, bin_shift;
    bool two_level;
};

// The populated bucket before b within b's segment: its index, or ~0 when b is the segment's first.
__device__ __forceinline__ uint64_t prev_bucket(const PlanCtx &c, uint64_t b)
{
    const uint64_t s = c.hist[b], first = max(c.lo, b & ~(uint64_t)(NB - 1));
    if (c.hist[first] == s) return ~0ull;
    uint64_t p = b - 1;
    for (int i = 0; i < 4; i++, p--)
        if (c.hist[p] != s) return p;
    uint64_t a = first, z = p + 1;  // the first index whose prefix is s ends the bucket before b
    while (a < z) {
        const uint64_t m = (a + z) >> 1;
        if (c.hist[m] < s) a = m + 1; else z = m;
    }
    return a - 1;
}

// Whether bucket b (populated, prefix [s, e) from the scan's start) starts a unit (bit 0), a bin (bit 1), its
// segment (bit 2), or a thread range (bit 3).  Units never cross a thread range, a segment, a multiple of 2^16
// buckets (the bucket within a bin takes 16 bits) or a multiple of 2^unit_shift tuples, except that a bucket which
// would make its unit larger than GP_CAP_S is a unit of its own: every decision is local to the bucket and its
// predecessor, so the plan is two parallel passes (a greedy packing by one thread per 256 buckets took 140-210 us).
__device__ __forceinline__ uint32_t plan_flags(const PlanCtx &c, uint64_t b, uint64_t s, uint64_t e)
{
    const uint64_t p = prev_bucket(c, b);
    if (p == ~0ull) return 15u;
    const uint64_t sp = c.hist[p] - c.hist[c.lo];
    const uint64_t rel = b - c.lo;
    const bool brk = (c.brk[rel >> 5] >> (rel & 31)) & 1u;
    const bool far = (p >> 16) != (b >> 16);
    const uint64_t q = s >> c.unit_shift;
    const bool unit = brk || far || q != (sp >> c.unit_shift) || e - (q << c.unit_shift) > (uint64_t)GP_CAP_S;
    const bool bin = c.two_level ? far || (s >> c.bin_shift) != (sp >> c.bin_shift) : unit;
    return (unit || bin ? 1u : 0u) | (bin ? 2u : 0u) | (brk ? 8u : 0u);
}

// The bucket that starts at each thread range's first tuple.
__global__ void k_gp_marks(const uint64_t *hist, uint64_t lo, uint64_t hi, const uint64_t *bounds, int nb, uint32_t *brk)
{
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= nb) return;
    const uint64_t x = bounds[t] + hist[lo];
    uint64_t a = lo, z = hi;  // the last bucket whose prefix is x is the populated one
    while (a < z) {
        const uint64_t m = (a + z) >> 1;
        if (hist[m + 1] <= x) a = m + 1; else z = m;
    }
    if (a < hi) atomicOr(&brk[(a - lo) >> 5], 1u << ((a - lo) & 31));
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

// Units (low word) and bins (high word) starting in each block of GP_COUNT_BLOCK buckets.
__global__ void __launch_bounds__(GP_COUNT_THREADS) k_gp_count(PlanCtx c, uint64_t *blk)
{
    __shared__ uint64_t ws[GP_COUNT_THREADS / 32];
    uint64_t v = 0;
    const uint64_t h0 = c.hist[c.lo];
    for (int i = 0; i < GP_COUNT_ITEMS; i++) {
        const uint64_t b = c.lo + (uint64_t)blockIdx.x * GP_COUNT_BLOCK + (uint64_t)i * GP_COUNT_THREADS + threadIdx.x;
        if (b >= c.hi) break;
        const uint64_t s = c.hist[b], e = c.hist[b + 1];
        if (s == e) continue;
        const uint32_t f = plan_flags(c, b, s - h0, e - h0);
        v += (f & 1u) | ((uint64_t)((f >> 1) & 1u) << 32);
    }
    uint64_t tot;
    block_scan_excl(v, &tot, ws);
    if (threadIdx.x == 0) blk[blockIdx.x] = tot;
}

// Exclusive scan of the blocks' counts by one block; the sentinels past the last unit and bin.
__global__ void __launch_bounds__(1024) k_gp_scan(uint64_t *blk, uint32_t nblk, uint32_t n, int nseg, uint32_t *ctr,
                                                  uint32_t *ustart, uint32_t *bstart, uint32_t *bu0, uint32_t *seg_bin0)
{
    __shared__ uint64_t ws[32];
    uint64_t carry = 0;
    for (uint32_t i0 = 0; i0 < nblk; i0 += 1024) {
        const uint32_t i = i0 + threadIdx.x;
        uint64_t tot;
        const uint64_t x = block_scan_excl(i < nblk ? blk[i] : 0, &tot, ws);
        if (i < nblk) blk[i] = carry + x;
        carry += tot;
    }
    if (threadIdx.x == 0) {
        const uint32_t nu = (uint32_t)carry, nb = (uint32_t)(carry >> 32);
        ctr[GC_UNITS] = nu;
        ctr[GC_BINS] = nb;
        ustart[nu] = n;
        bstart[nb] = n;
        bu0[nb] = nu;
        seg_bin0[nseg] = nb;
    }
}

// The unit and bin arrays.  A bucket above GP_CAP_S tuples is a unit of its own (plan_flags), so its size is known here.
__global__ void __launch_bounds__(GP_COUNT_THREADS) k_gp_write(PlanCtx c, const uint64_t *blk, uint32_t *ctr, uint32_t *ustart,
                                                               uint32_t *ub0, uint32_t *ucur, uint32_t *bstart, uint32_t *bb0,
                                                               uint32_t *bu0, uint32_t *bcur, uint32_t *seg_bin0,
                                                               uint32_t *mid, uint32_t *big)
{
    __shared__ uint64_t ws[GP_COUNT_THREADS / 32];
    const uint64_t h0 = c.hist[c.lo];
    uint64_t at = blk[blockIdx.x];
    for (int i = 0; i < GP_COUNT_ITEMS; i++) {
        const uint64_t b = c.lo + (uint64_t)blockIdx.x * GP_COUNT_BLOCK + (uint64_t)i * GP_COUNT_THREADS + threadIdx.x;
        uint64_t s = 0, e = 0;
        uint32_t f = 0;
        if (b < c.hi) {
            s = c.hist[b] - h0;
            e = c.hist[b + 1] - h0;
            if (s != e) f = plan_flags(c, b, s, e);
        }
        uint64_t tot;
        const uint64_t x = at + block_scan_excl((f & 1u) | ((uint64_t)((f >> 1) & 1u) << 32), &tot, ws);
        at += tot;
        const uint32_t u = (uint32_t)x, bin = (uint32_t)(x >> 32);
        if (f & 1u) {
            ustart[u] = ucur[u] = (uint32_t)s;
            ub0[u] = (uint32_t)b | (f & 8u ? 0x80000000u : 0u);
        }
        if (f & 2u) {
            bstart[bin] = bcur[bin] = (uint32_t)s;
            bb0[bin] = (uint32_t)b;
            bu0[bin] = u;
        }
        if (f & 4u) seg_bin0[b / NB] = bin;
        if (e - s > (uint64_t)GP_CAP_S) {
            if (e - s <= (uint64_t)GP_CAP_L) mid[atomicAdd(&ctr[GC_MID], 1u)] = u;
            else {
                big[atomicAdd(&ctr[GC_BIG], 1u)] = u;
                atomicAdd(&ctr[GC_BIG_TUPLES], (uint32_t)(e - s));
            }
        }
    }
}

// ------------------------------------------------------------------ split

constexpr int SP_THREADS = 512, SP_ITEMS = 12, SP_TILE = SP_THREADS * SP_ITEMS;

// Tiles of the second pass: every bin's own, from its first tuple.
__global__ void __launch_bounds__(1024) k_gp_tiles(const uint32_t *bstart, uint32_t *ctr, uint32_t *tile_first, uint32_t *tile_bin)
{
    __shared__ uint64_t ws[32];
    const uint32_t nb = ctr[GC_BINS];
    uint64_t carry = 0;
    for (uint32_t i0 = 0; i0 < nb; i0 += 1024) {
        const uint32_t i = i0 + threadIdx.x;
        const uint32_t t = i < nb ? (bstart[i + 1] - bstart[i] + SP_TILE - 1) / SP_TILE : 0;
        uint64_t tot;
        const uint64_t x = carry + block_scan_excl(t, &tot, ws);
        if (i < nb) {
            tile_first[i] = (uint32_t)x;
            for (uint32_t q = 0; q < t; q++) tile_bin[x + q] = i;
        }
        carry += tot;
    }
    if (threadIdx.x == 0) ctr[GC_TILES] = (uint32_t)carry;
}

// Digit lookup: a segment's (or a bin's) bucket range in CELLS cells of 2^shift buckets, each with the digits of its first
// and its last bucket (low and high half); where they differ, a search between them.  One shared-memory read per tuple
// in nearly all cases: a binary search over the digits' first buckets instead (10 dependent reads) held the passes to
// 2.6 TB/s with the shared-memory pipe 83 % busy.
constexpr uint32_t CELLS_1 = 2048, CELLS_2 = 1024;

__host__ __device__ __forceinline__ int cell_shift(uint64_t span, uint32_t cells)
{
    int s = 0;
    while (((span - 1) >> s) >= cells) s++;
    return s;
}

__global__ void __launch_bounds__(256) k_gp_cells(const uint32_t *bb0, const uint32_t *seg_bin0, uint32_t b_lo, uint32_t b_hi,
                                                  int shift, uint32_t *cells)
{
    const uint32_t seg = blockIdx.y, c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= CELLS_1) return;
    const uint32_t d0 = seg_bin0[seg], nd = seg_bin0[seg + 1] - d0;
    uint32_t v[2];
    for (int q = 0; q < 2; q++) {
        const uint64_t x = min((uint64_t)b_hi - 1, b_lo + ((uint64_t)(c + q) << shift) - q);
        uint32_t a = 0, z = nd - 1;  // the last bin whose first bucket is at or below x
        while (a < z) {
            const uint32_t m = (a + z + 1) >> 1;
            if ((bb0[d0 + m] & (NB - 1)) <= x) a = m; else z = m - 1;
        }
        v[q] = a;
    }
    cells[(size_t)seg * CELLS_1 + c] = v[0] | (v[1] << 16);
}

template <class B>
__device__ __forceinline__ uint32_t cell_digit(const uint32_t *cells, const B *b0, int shift, uint32_t rel, uint32_t b)
{
    const uint32_t v = cells[rel >> shift];
    uint32_t a = v & 0xFFFFu, z = v >> 16;
    while (a < z) {
        const uint32_t m = (a + z + 1) >> 1;
        if (b0[m] <= b) a = m; else z = m - 1;
    }
    return a;
}

template <int DIGITS, class B, uint32_t CELLS> struct SplitSmem {
    uint64_t key[SP_TILE];   // (the packed reads of k_enum_bins before)
    uint32_t id[SP_TILE];
    uint16_t dig[SP_TILE];
    B b0[DIGITS];            // first bucket of every digit
    uint32_t hist[DIGITS];   // tuples per digit, then the digit's first place in the tile
    uint32_t delta[DIGITS];  // global place of a digit's first tuple less its place in the tile
    uint32_t cells[CELLS];
    uint32_t ws[SP_THREADS / 32];
};
typedef SplitSmem<GP_MAX_BINS, uint32_t, CELLS_1> BinSmem;
template <int DIGITS> using UnitSmem = SplitSmem<DIGITS, uint16_t, CELLS_2>;
static_assert(2 * (sizeof(BinSmem) + 1024) <= 228 * 1024 && 2 * (sizeof(UnitSmem<GP_MAX_UNITS>) + 1024) <= 228 * 1024,
              "two split blocks per SM");

// Unstable, so there are no ballots and no look-back: ranks by shared-memory atomics, places by one global atomic per
// digit and tile (the order of a digit's tuples is free), a shared-memory reorder so that a digit's tuples are stored
// side by side.  rd: digit in (0xFFFF = no tuple).
template <class Smem, int DIGITS, class LoadId>
__device__ __forceinline__ void split_tile(Smem &sm, const uint64_t (&key)[SP_ITEMS], uint32_t (&rd)[SP_ITEMS], uint32_t *cur,
                                           uint32_t nd, LoadId load_id, uint64_t *out_k, uint32_t *out_id, uint32_t n)
{
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
#pragma unroll
    for (int j = 0; j < SP_ITEMS; j++)
        if (rd[j] != 0xFFFFu) rd[j] |= atomicAdd(&sm.hist[rd[j]], 1u) << 16;
    uint32_t id[SP_ITEMS];
#pragma unroll
    for (int j = 0; j < SP_ITEMS; j++) id[j] = load_id(j);
    __syncthreads();
    constexpr int PER = DIGITS / SP_THREADS;
    uint32_t c[PER], s = 0;
#pragma unroll
    for (int q = 0; q < PER; q++) {
        c[q] = sm.hist[tid * PER + q];
        s += c[q];
    }
    uint32_t g[PER];
#pragma unroll
    for (int q = 0; q < PER; q++) g[q] = c[q] && tid * PER + q < nd ? atomicAdd(&cur[tid * PER + q], c[q]) : 0u;
    uint32_t x = s;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(FULLG, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) sm.ws[warp] = x;
    __syncthreads();
    uint32_t before = x - s, nv = 0;
    for (int w = 0; w < SP_THREADS / 32; w++) {
        const uint32_t v = sm.ws[w];
        before += w < warp ? v : 0u;
        nv += v;
    }
#pragma unroll
    for (int q = 0; q < PER; q++) {
        sm.hist[tid * PER + q] = before;
        sm.delta[tid * PER + q] = g[q] - before;
        before += c[q];
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < SP_ITEMS; j++) {
        const uint32_t d = rd[j] & 0xFFFFu;
        if (d != 0xFFFFu) {
            const uint32_t p = sm.hist[d] + (rd[j] >> 16);
            sm.key[p] = key[j];
            sm.id[p] = id[j];
            sm.dig[p] = (uint16_t)d;
        }
    }
    __syncthreads();
    for (uint32_t p = tid; p < nv; p += SP_THREADS) {
        const uint32_t o = p + sm.delta[sm.dig[p]];
        if (o < n) {  // (a histogram that does not match the tuples is reported by the group kernel)
            out_k[o] = sm.key[p];
            out_id[o] = sm.id[p];
        }
    }
#pragma unroll
    for (int q = 0; q < PER; q++) sm.hist[tid * PER + q] = 0;  // (read last before the barrier above)
}

// The tiles of a pass over segments: tile0[q] the segment's first tile, start[q] its first read or tuple, tile_seg the
// segment of every tile; null for one segment.
struct SegTiles {
    const uint32_t *tile_seg = nullptr, *tile0 = nullptr, *start = nullptr;
};

__global__ void k_gp_segtiles(const uint32_t *tile0, int nseg, uint32_t *tile_seg)
{
    const int q = blockIdx.x;
    for (uint32_t t = tile0[q] + threadIdx.x; t < tile0[q + 1]; t += blockDim.x) tile_seg[t] = (uint32_t)q;
}

// First pass, one of two sources: the reads (k_readtile.cuh; the tuples of the buckets [b_lo, b_hi)), or tuples enumerated
// before (lo = k-mer << 8 | adj, hi = k-mer >> 56; the 3-minimizer variant).
struct BinCtx {
    ReadTiles t;
    uint32_t n_reads = 0, check_many = 0;
    const uint32_t *label = nullptr;
    const uint64_t *lo = nullptr;
    const uint8_t *hi = nullptr;
    const uint32_t *id = nullptr;
    uint32_t tiles = 0, n = 0, b_lo = 0, b_hi = 0;
    int bsh = 0, shift = 0;
    const uint32_t *bb0 = nullptr, *seg_bin0 = nullptr, *cells = nullptr;
    uint32_t *bcur = nullptr, *err = nullptr;
    SegTiles sg;
    uint64_t *out_k = nullptr;
    uint32_t *out_id = nullptr;
};

template <bool READS>
__global__ void __launch_bounds__(SP_THREADS, 2) k_split_bins(BinCtx c)
{
    extern __shared__ __align__(16) unsigned char smraw[];
    BinSmem &sm = *reinterpret_cast<BinSmem *>(smraw);
    __shared__ uint32_t many[READS ? SP_THREADS : 1];
    const int tid = threadIdx.x;
    const uint64_t lowmask = (1ull << c.bsh) - 1;
    uint32_t have = ~0u, d0 = 0, nd = 0;  // the segment whose digits are in shared memory
    for (uint32_t d = tid; d < GP_MAX_BINS; d += SP_THREADS) sm.hist[d] = 0;
    for (uint32_t tile = blockIdx.x; tile < c.tiles; tile += gridDim.x) {
        const uint32_t seg = c.sg.tile_seg ? c.sg.tile_seg[tile] : 0u;
        const uint32_t per = READS ? c.t.rpt : (uint32_t)SP_TILE;
        uint32_t base = tile * per, end = READS ? c.n_reads : c.n;
        if (c.sg.tile_seg) {
            base = c.sg.start[seg] + (tile - c.sg.tile0[seg]) * per;
            end = c.sg.start[seg + 1];
        }
        __syncthreads();  // the tile before is stored
        if (seg != have) {
            have = seg;
            d0 = c.seg_bin0[seg];
            nd = c.seg_bin0[seg + 1] - d0;
            for (uint32_t d = tid; d < nd; d += SP_THREADS) sm.b0[d] = c.bb0[d0 + d] & (NB - 1);
            for (uint32_t d = tid; d < CELLS_1; d += SP_THREADS) sm.cells[d] = c.cells[(size_t)seg * CELLS_1 + d];
        }
        uint64_t key[SP_ITEMS];
        uint32_t rd[SP_ITEMS];
        if constexpr (READS) {
            uint32_t *packed = reinterpret_cast<uint32_t *>(sm.key);
            const uint32_t r1 = min(end, base + per);
            if (c.check_many) many[tid] = 0;
            rt_pack(c.t, base, r1, packed);
            __syncthreads();
#pragma unroll
            for (int j = 0; j < SP_ITEMS; j++) rd[j] = 0xFFFFu;
            const uint32_t rr = tid / c.t.spr, i0 = (tid - rr * c.t.spr) * c.t.P, r = base + rr;
            const uint32_t L = rr < per && r < r1 ? c.t.seq_len[r] : 0u;
            uint32_t id = r;
            if (L > (uint32_t)c.t.k && i0 <= L - (uint32_t)c.t.k) {
                if (c.label) {
                    const uint32_t p = c.label[r];
                    id = p == BAD ? r : p;  // findRoot after full compression (metapart.c:543-568)
                }
                KmerRoll s;
                kr_init(s, c.t, packed + rr * rt_stride(c.t), L, i0);
                const uint32_t m = min(c.t.P, s.last + 1 - i0);
                uint32_t got = 0;
#pragma unroll
                for (int j = 0; j < SP_ITEMS; j++) {
                    if (j < m) {
                        uint64_t km;
                        const bool v = kr_get(s, c.t.k, km);
                        const uint32_t b = (uint32_t)(km >> c.bsh);
                        if (v && b >= c.b_lo && b < c.b_hi) {
                            const uint32_t d = cell_digit(sm.cells, sm.b0, c.shift, b - c.b_lo, b);
                            key[j] = ((((uint64_t)(b - sm.b0[d]) << c.bsh) | (km & lowmask)) << 6) | kr_adj6(s);
                            rd[j] = d;
                            got++;
                        }
                        kr_next(s, c.t.k);
                    }
                }
                // the reference counts a read's k-mers of one scan in 8 bits (enumerateKmers.c:152)
                if (c.check_many && atomicAdd(&many[rr], got) + got > 255u) atomicOr(c.err, 4u);
            }
            split_tile<BinSmem, GP_MAX_BINS>(sm, key, rd, c.bcur + d0, nd, [&](int) { return id; }, c.out_k, c.out_id, c.n);
        } else {
            const uint32_t nv = min((uint32_t)SP_TILE, end - base);
            __syncthreads();
#pragma unroll
            for (int j = 0; j < SP_ITEMS; j++) {
                const uint32_t e = j * SP_THREADS + tid;
                rd[j] = 0xFFFFu;
                if (e < nv) {
                    const uint64_t v = c.lo[base + e], km = (v >> 8) | (c.hi ? (uint64_t)c.hi[base + e] << 56 : 0ull);
                    const uint32_t b = min(max((uint32_t)(km >> c.bsh), c.b_lo), c.b_hi - 1);
                    const uint32_t d = cell_digit(sm.cells, sm.b0, c.shift, b - c.b_lo, b);
                    key[j] = ((((uint64_t)(b - sm.b0[d]) << c.bsh) | (km & lowmask)) << 6) | (v & 63u);
                    rd[j] = d;
                }
            }
            split_tile<BinSmem, GP_MAX_BINS>(
                sm, key, rd, c.bcur + d0, nd,
                [&](int j) { const uint32_t e = j * SP_THREADS + tid; return e < nv ? c.id[base + e] : 0u; }, c.out_k, c.out_id, c.n);
        }
    }
}

// Second pass: a bin's tuples into its units.  A block takes consecutive tiles, so it sets up a bin's digits once.
template <int DIGITS, int BLOCKS>
__global__ void __launch_bounds__(SP_THREADS, BLOCKS) k_split_units(const uint64_t *__restrict__ kk, const uint32_t *__restrict__ id,
                                                                    uint32_t n, int bsh, const uint32_t *__restrict__ ctr,
                                                                    const uint32_t *__restrict__ bstart,
                                                                    const uint32_t *__restrict__ bb0,
                                                                    const uint32_t *__restrict__ bu0,
                                                                    const uint32_t *__restrict__ bcur,
                                                                    const uint32_t *__restrict__ ub0, uint32_t *ucur,
                                                                    const uint32_t *__restrict__ tile_bin,
                                                                    const uint32_t *__restrict__ tile_first, uint64_t *out_k,
                                                                    uint32_t *out_id)
{
    extern __shared__ __align__(16) unsigned char smraw[];
    UnitSmem<DIGITS> &sm = *reinterpret_cast<UnitSmem<DIGITS> *>(smraw);
    const int tid = threadIdx.x;
    const uint32_t tiles = ctr[GC_TILES], per = (tiles + gridDim.x - 1) / gridDim.x;
    const uint32_t t0 = blockIdx.x * per, t1 = min(tiles, t0 + per);
    uint32_t have = ~0u, d0 = 0, nd = 0, bin_start = 0, bin_end = 0, first_tile = 0;
    int shift = 0;
    bool whole = false;
    for (uint32_t d = tid; d < DIGITS; d += SP_THREADS) sm.hist[d] = 0;
    for (uint32_t tile = t0; tile < t1; tile++) {
        const uint32_t bin = tile_bin[tile];
        __syncthreads();  // the tile before is stored
        if (bin != have) {
            have = bin;
            bin_start = bstart[bin];
            bin_end = bstart[bin + 1];
            whole = bcur[bin] == bin_end;  // else the histogram is not the tuples' (the bin's units stay short: k_group)
            first_tile = tile_first[bin];
            d0 = bu0[bin];
            nd = min(bu0[bin + 1] - d0, (uint32_t)DIGITS);
            const uint32_t first = bb0[bin];
            for (uint32_t d = tid; d < nd; d += SP_THREADS) sm.b0[d] = (uint16_t)((ub0[d0 + d] & 0x7FFFFFFFu) - first);
            __syncthreads();
            const uint32_t span = (uint32_t)sm.b0[nd - 1] + 1;  // buckets from the last unit's first on are its own
            shift = cell_shift(span, CELLS_2);
            for (uint32_t c = tid; c < CELLS_2; c += SP_THREADS) {
                uint32_t v[2];
#pragma unroll
                for (int q = 0; q < 2; q++) {
                    const uint32_t x = ((c + q) << shift) - q;
                    uint32_t a = 0, z = nd - 1;
                    while (a < z) {
                        const uint32_t m = (a + z + 1) >> 1;
                        if (sm.b0[m] <= x) a = m; else z = m - 1;
                    }
                    v[q] = a;
                }
                sm.cells[c] = v[0] | (v[1] << 16);
            }
            __syncthreads();
        }
        if (!whole) continue;
        const uint32_t base = bin_start + (tile - first_tile) * SP_TILE, nv = min((uint32_t)SP_TILE, bin_end - base);
        const uint32_t top = (uint32_t)sm.b0[nd - 1];
        uint64_t key[SP_ITEMS];
        uint32_t rd[SP_ITEMS];
#pragma unroll
        for (int j = 0; j < SP_ITEMS; j++) {
            const uint32_t e = j * SP_THREADS + tid;
            key[j] = e < nv ? kk[base + e] : 0ull;
        }
#pragma unroll
        for (int j = 0; j < SP_ITEMS; j++) {
            const uint32_t b = min((uint32_t)(key[j] >> (bsh + 6)), top);
            rd[j] = j * SP_THREADS + tid < nv ? cell_digit(sm.cells, sm.b0, shift, b, b) : 0xFFFFu;
        }
        split_tile<UnitSmem<DIGITS>, DIGITS>(
            sm, key, rd, ucur + d0, nd, [&](int j) { const uint32_t e = j * SP_THREADS + tid; return e < nv ? id[base + e] : 0u; },
            out_k, out_id, n);
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
    uint32_t cap_lo, cap_hi;  // takes units of cap_lo < tuples <= cap_hi
    uint32_t *out, *parent;
    uint8_t *filtered;
};

// Bound by shared memory (random accesses and atomics: about five per tuple) and the block's barriers; two
// 512-thread blocks per SM overlap each other's.  20M x 150 bp, 2 scans (2.39 G tuples): 31.4 ms for both block
// shapes, where sorting the units (66.8 ms) and judging the sorted runs (31.9 ms) took 98.7.
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
__global__ void __launch_bounds__(THREADS, 1024 / THREADS) k_group(GroupCtx c)
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
        const bool ends = last || (nextb >> 31), seg_last = last || ((nextb & 0x7FFFFFFFu) / NB != b0 / NB);
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
        // ---- every tuple's slot and its number within the slot (sr: slot 0-13, number 16-29), codes in ac
        uint32_t sr[ITEMS], ac[ITEMS];
#pragma unroll
        for (int j = 0; j < ITEMS; j++) {
            sr[j] = 0;
            ac[j] = (uint32_t)key[j] & 63u;
            if (j * THREADS + tid < cnt) {
                const unsigned long long k = key[j] >> 6;
                uint32_t h = key_hash(k) >> (32 - SLOT_BITS);
                for (;;) {
                    unsigned long long v = vkey[h];
                    if (v == EMPTY) {
                        v = atomicCAS(&sm.u.key[h], EMPTY, k);
                        if (v == EMPTY) v = k;
                    }
                    if (v == k) break;
                    h = (h + 1) & SMASK;
                }
                const uint32_t bi = ac[j] & 7u, ai = ac[j] >> 3;
                const uint32_t m = (bi < 7u ? 0x10000u << bi : 0u) | (ai < 7u ? 0x800000u << ai : 0u);
                const uint32_t old = atomicAdd(&sm.info[h], 1u);
                if (m & ~old) atomicOr(&sm.info[h], m);
                sr[j] = h | ((old & 0xFFFFu) << 16);
                if (k == 0) ac[j] |= 64u;
                if (ends && k == sm.maxkey) sm.slot_ex = h;
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
        const bool zero_bucket = (b0 & (NB - 1)) == 0;
        uint32_t kept = 0;
#pragma unroll
        for (int j = 0; j < ITEMS; j++) {
            if (j * THREADS + tid < cnt && (sr[j] >> 16) == 0) {
                const uint32_t h = sr[j], inf = sm.info[h], n = inf & 0xFFFFu;
                uint32_t side = 0;
                if (h != ex) side = (__popc(inf & 0x7F0000u) > 1 ? 1u : 0u) | (__popc(inf & 0x3F800000u) > 1 ? 2u : 0u);
                uint32_t ni = n | (side << 14);
                if (side == 1u || side == 2u) {
                    const uint32_t p = atomicAdd(&sm.npool, 1u);
                    reinterpret_cast<uint4 *>(sm.u.b.pool)[p] = make_uint4(0, 0, 0, h << 16);
                    ni |= p << 16;
                }
                if (side != 3u && !(zero_bucket && (ac[j] & 64u)) && (n >= 2u || singles)) {
                    ni |= GI_KEPT;
                    kept += n;
                    ac[j] |= 128u;
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
        uint32_t at = x - kept, total = 0;
        for (int q = 0; q < THREADS / 32; q++) {
            const uint32_t t = sm.ws[q];
            at += q < warp ? t : 0u;
            total += t;
        }
        if (tid == 0) sm.base = atomicAdd(&c.ctr[GC_OUT], total);
#pragma unroll
        for (int j = 0; j < ITEMS; j++) {
            if (ac[j] & 128u) {
                const uint32_t h = sr[j] & 0xFFFFu;
                sm.u.b.off[h] = (uint16_t)at;
                at += sm.info[h] & 0x3FFFu;
            }
        }
        // ---- code counts of the runs branching on one side
#pragma unroll
        for (int j = 0; j < ITEMS; j++) {
            if (j * THREADS + tid < cnt) {
                const uint32_t inf = sm.info[sr[j] & 0xFFFFu], side = (inf >> 14) & 3u;
                const uint32_t code = side == 1u ? ac[j] & 7u : (ac[j] >> 3) & 7u;
                if ((side == 1u || side == 2u) && code < 7u)
                    atomicAdd(&sm.u.b.pool[((inf >> 16) & 0x1FFFu) * 4 + (code >> 1)], 1u << (16 * (code & 1)));
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
                const uint32_t h = sr[j] & 0xFFFFu, inf = sm.info[h], side = (inf >> 14) & 3u;
                const uint32_t code = side == 1u ? ac[j] & 7u : (ac[j] >> 3) & 7u;
                if ((side == 1u || side == 2u) && (code != ((inf >> 16) & 7u) || (inf & (1u << 19)))) {
                    c.parent[id[j]] = BAD;
                    c.filtered[id[j]] = 1;
                }
                if (inf & GI_KEPT) stage[sm.u.b.off[h] + (sr[j] >> 16)] = id[j] | ((sr[j] >> 16) == 0 ? 0x80000000u : 0u);
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
typedef GroupSmem<512, 12, 13> GroupSmemS;
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
                            const uint32_t *fill, uint32_t *err, uint32_t *out)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nb) return;
    const uint32_t u = big[i];
    out[4 * i] = u;
    out[4 * i + 1] = ustart[u];
    out[4 * i + 2] = ustart[u + 1] - ustart[u];
    out[4 * i + 3] = (u + 1 == nunits || (ub0[u + 1] >> 31)) ? 1u : 0u;  // ends a thread range
    if (fill[u] != ustart[u + 1]) {  // the histogram is not the tuples'
        atomicOr(err, 2u);
        out[4 * i + 2] = 0;
    }
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

// The sorted units' ids into out, as k_group leaves them (a zeroed tuple or the zero k-mer's stands for no read).
__global__ void k_gbig_emit(const BigUnit *bu, const uint32_t *base, const uint64_t *tk, const uint32_t *tid, const uint32_t *z,
                            const uint32_t *ub0, uint32_t nunits, const uint32_t *lrs, int bsh, uint32_t *ctr, uint32_t *qlist,
                            uint32_t *quirk, uint32_t *out)
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
        out[o + e] = (none ? GP_NONE : tid[i]) | (head ? 0x80000000u : 0u);
    }
    if (blockIdx.y == 0 && threadIdx.x == 0 && b.start >= lrs[seg]) {
        uint32_t *q = qlist + 3 * (size_t)atomicAdd(&ctr[GC_QLIST], 1u);
        q[0] = o;
        q[1] = b.cnt;
        q[2] = seg;
        if (b.u + 1 == nunits || (ub0[b.u + 1] & 0x7FFFFFFFu) / NB != seg) {  // the segment's last run
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

__global__ void k_gbig_reserve(uint32_t *ctr, uint32_t n, uint32_t *base) { *base = atomicAdd(&ctr[GC_OUT], n); }

// ------------------------------------------------------------------ unions

// The sweeps' initial state (metapart.c:2539-2548): a thread range's first valid tuple joins the scan's first
// read when it carries the scan's last k-mer, which only the last range with tuples can hold and only if no
// smaller k-mer of that range has a read that is not BAD.  Per segment, over the grouped stretches of its last
// range: [0] a read outside the last run, [1] one inside, [2] its id.
__global__ void __launch_bounds__(256) k_gp_quirk(const uint32_t *ctr, const uint32_t *qlist, const uint32_t *out,
                                                  const uint8_t *filtered, uint32_t *quirk)
{
    volatile uint32_t *vq = quirk;
    const uint32_t nq = ctr[GC_QLIST];
    for (uint32_t q = blockIdx.x; q < nq; q += gridDim.x) {
        const uint32_t o = qlist[3 * (size_t)q], len = qlist[3 * (size_t)q + 1], seg = qlist[3 * (size_t)q + 2];
        const uint32_t l0 = quirk[seg * QW + 3], l1 = l0 + quirk[seg * QW + 4];
        for (uint32_t i = threadIdx.x; i < len; i += blockDim.x) {
            if (vq[seg * QW]) break;
            const uint32_t id = out[o + i] & 0x7FFFFFFFu;
            if (id == GP_NONE || filtered[id]) continue;
            if (o + i >= l0 && o + i < l1) {
                quirk[seg * QW + 2] = id;
                quirk[seg * QW + 1] = 1;
            } else {
                quirk[seg * QW] = 1;
            }
        }
    }
}

constexpr uint32_t GE_SEG = 1024;  // grouped ids per warp and turn

// Bound by the random reads of the BAD flags and parents in L2.  It reads 4 bytes per joining tuple where the
// sweep over sorted tuples read 13 per tuple: 6.7 ms against 21.0 at 20M x 150 bp, 2 scans.
//
// The unions of every k-mer's reads (metapart.c:2537-2727): each read that is not BAD joins its k-mer's first one
// of the stretch.  A stretch that starts inside a run looks back for one read of it, so long runs are shared by
// many warps.
__global__ void __launch_bounds__(256) k_gp_union(const uint32_t *ctr, const uint32_t *__restrict__ out, uint32_t *parent,
                                                  const uint8_t *__restrict__ filtered, uint32_t *err, uint32_t uf_cap)
{
    const uint32_t m = ctr[GC_OUT];
    const int lane = threadIdx.x & 31;
    const uint32_t le = (lane == 31) ? FULLG : ((2u << lane) - 1);
    const uint32_t nw = (gridDim.x * blockDim.x) >> 5, nseg = (m + GE_SEG - 1) / GE_SEG;
    for (uint32_t sgm = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; sgm < nseg; sgm += nw) {
        const uint32_t p0 = sgm * GE_SEG, p1 = min(m, p0 + GE_SEG);
        bool has = false;
        uint32_t anchor = 0;
        if (!(out[p0] >> 31)) {  // the run's reads before the stretch, a window at a time
            for (uint32_t q = p0; q >= 32;) {
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

static uint32_t bins_bound(uint64_t n, int nseg, int shift) { return (uint32_t)(n >> shift) + 18u * (uint32_t)nseg + 1u; }

// A scan takes the grouped path when its positions fit 32 bits, its read ids 31, and the split's digits suffice.
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
        cudaFuncSetAttribute(k_split_bins<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(BinSmem));
        cudaFuncSetAttribute(k_split_bins<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(BinSmem));
        cudaFuncSetAttribute(k_split_units<GP_MAX_UNITS, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)sizeof(UnitSmem<GP_MAX_UNITS>));
        cudaFuncSetAttribute(k_split_units<GP_MAX_UNITS_L, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)sizeof(UnitSmem<GP_MAX_UNITS_L>));
        cudaFuncSetAttribute(k_group<512, 12, 13>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(GroupSmemS));
        cudaFuncSetAttribute(k_group<1024, 12, 14>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(GroupSmemL));
    });
}

int group_plan(GroupScan &g, DeviceArena &arena, cudaStream_t st)
{
    const int nseg = (int)g.seg_tstart.size() - 1;
    const uint32_t nbounds = (uint32_t)g.bounds.size();
    const uint64_t nbk = g.hi - g.lo;
    uint64_t seg_max = 0;  // a segment's units and bins bound the digits of a pass
    for (int q = 0; q < nseg; q++) seg_max = std::max<uint64_t>(seg_max, g.seg_tstart[q + 1] - g.seg_tstart[q]);
    g.unit_shift = GP_UNIT_SHIFT;
    // units per segment: a start per thread range, per 2^16 buckets, and at most two per 2^unit_shift tuples
    const uint64_t units_seg = 2 * (seg_max >> g.unit_shift) + nbounds + 20;
    g.two_level = units_seg > GP_MAX_BINS;
    // two levels: about as many bins as units per bin
    int lg = 0;
    while ((seg_max >> lg) > 1) lg++;
    g.bin_shift = (g.unit_shift + lg + 1) / 2;
    while ((seg_max >> g.bin_shift) + 20 > GP_MAX_BINS) g.bin_shift++;
    g.max_units = 2 * (uint32_t)(g.n >> g.unit_shift) + nbounds + 20u * (uint32_t)nseg + 8;
    g.max_bins = g.two_level ? bins_bound(g.n, nseg, g.bin_shift) : g.max_units;
    if (g.two_level) g.max_units += g.max_bins;
    g.max_tiles = (uint32_t)(g.n / SP_TILE) + g.max_bins + 1;
    g.cell_shift = cell_shift(nseg > 1 ? (uint64_t)NB : nbk, CELLS_1);
    g.cells = arena.alloc<uint32_t>((size_t)nseg * CELLS_1);
    const uint32_t nblk = blocks_of(nbk, GP_COUNT_BLOCK);
    const size_t brk_words = nbk / 32 + 1;
    uint32_t *brk = arena.alloc<uint32_t>(brk_words + GC_N + (size_t)nseg * QW);
    uint64_t *blk = arena.alloc<uint64_t>(nblk), *d_bounds = arena.alloc<uint64_t>(nbounds);
    g.ustart = arena.alloc<uint32_t>(3 * (size_t)(g.max_units + 1));
    g.bstart = arena.alloc<uint32_t>(4 * (size_t)(g.max_bins + 1));
    g.seg_bin0 = arena.alloc<uint32_t>(2 * (size_t)nseg + 1);
    g.tile_bin = arena.alloc<uint32_t>((size_t)g.max_tiles + g.max_bins);
    g.mid = arena.alloc<uint32_t>(2 * (size_t)(g.n / GP_CAP_S + 1));
    g.qlist = arena.alloc<uint32_t>(3 * (size_t)(g.max_units + 1));
    if (!brk || !blk || !d_bounds || !g.ustart || !g.bstart || !g.seg_bin0 || !g.tile_bin || !g.mid || !g.qlist || !g.cells)
        return set_error(MP_ENOMEM, "device memory for the scan's plan");
    g.ub0 = g.ustart + g.max_units + 1;
    g.ucur = g.ub0 + g.max_units + 1;
    g.bb0 = g.bstart + g.max_bins + 1;
    g.bu0 = g.bb0 + g.max_bins + 1;
    g.bcur = g.bu0 + g.max_bins + 1;
    g.lrs = g.seg_bin0 + nseg + 1;
    g.tile_first = g.tile_bin + g.max_tiles;
    g.big = g.mid + g.n / GP_CAP_S + 1;
    g.ctr = brk + brk_words;
    g.quirk = g.ctr + GC_N;
    std::vector<uint32_t> &lrs = g.h_lrs;
    lrs.assign(nseg, 0);
    for (int q = 0, t = 0; q < nseg; q++) {  // the last range bound inside the segment's tuples
        uint64_t b = g.seg_tstart[q];
        for (; t < (int)nbounds && g.bounds[t] < g.seg_tstart[q + 1]; t++) b = std::max(b, g.bounds[t]);
        lrs[q] = (uint32_t)b;
    }
    MP_CUDA(cudaMemsetAsync(brk, 0, (brk_words + GC_N + (size_t)nseg * QW) * 4, st));
    MP_CUDA(cudaMemcpyAsync(d_bounds, g.bounds.data(), nbounds * 8, cudaMemcpyHostToDevice, st));
    MP_CUDA(cudaMemcpyAsync(g.lrs, lrs.data(), nseg * 4, cudaMemcpyHostToDevice, st));
    PlanCtx c{g.d_hist, g.lo, g.hi, brk, g.unit_shift, g.bin_shift, g.two_level};
    (count_launch(), k_gp_marks<<<blocks_of(nbounds, 64), 64, 0, st>>>(g.d_hist, g.lo, g.hi, d_bounds, (int)nbounds, brk));
    (count_launch(), k_gp_count<<<nblk, GP_COUNT_THREADS, 0, st>>>(c, blk));
    (count_launch(), k_gp_scan<<<1, 1024, 0, st>>>(blk, nblk, (uint32_t)g.n, nseg, g.ctr, g.ustart, g.bstart, g.bu0, g.seg_bin0));
    (count_launch(), k_gp_write<<<nblk, GP_COUNT_THREADS, 0, st>>>(c, blk, g.ctr, g.ustart, g.ub0, g.ucur, g.bstart, g.bb0, g.bu0,
                                                                  g.bcur, g.seg_bin0, g.mid, g.big));
    (count_launch(), k_gp_cells<<<dim3(CELLS_1 / 256, nseg), 256, 0, st>>>(g.bb0, g.seg_bin0, nseg > 1 ? 0u : (uint32_t)g.lo,
                                                                          nseg > 1 ? NB : (uint32_t)g.hi, g.cell_shift, g.cells));
    if (g.two_level) (count_launch(), k_gp_tiles<<<1, 1024, 0, st>>>(g.bstart, g.ctr, g.tile_first, g.tile_bin));
    MP_CUDA(cudaMemcpyAsync(g.hctr, g.ctr, GC_N * 4, cudaMemcpyDeviceToHost, st));
    MP_CUDA(cudaGetLastError());
    return 0;
}

static int launch_bins(GroupScan &g, BinCtx &c, const std::vector<uint64_t> &seg_start, DeviceArena &arena, cudaStream_t st)
{
    group_kernel_attrs();
    const int nseg = (int)g.seg_tstart.size() - 1;
    const bool reads = c.lo == nullptr;
    const uint32_t per = reads ? c.t.rpt : (uint32_t)SP_TILE;
    c.tiles = blocks_of(reads ? c.n_reads : g.n, (int)per);
    if (nseg > 1) {
        std::vector<uint32_t> &h = g.h_tiles;
        h.assign(2 * (size_t)nseg + 2, 0);
        c.tiles = 0;
        for (int q = 0; q <= nseg; q++) {
            h[q] = c.tiles;
            h[nseg + 1 + q] = (uint32_t)seg_start[q];
            if (q < nseg) c.tiles += blocks_of(seg_start[q + 1] - seg_start[q], (int)per);
        }
        uint32_t *d = arena.alloc<uint32_t>(h.size() + c.tiles);
        if (!d) return set_error(MP_ENOMEM, "device memory for the scan's tiles");
        MP_CUDA(cudaMemcpyAsync(d, h.data(), h.size() * 4, cudaMemcpyHostToDevice, st));
        c.sg.tile0 = d;
        c.sg.start = d + nseg + 1;
        c.sg.tile_seg = d + h.size();
        (count_launch(), k_gp_segtiles<<<nseg, 256, 0, st>>>(d, nseg, d + h.size()));
    }
    c.n = (uint32_t)g.n;
    c.b_lo = nseg > 1 ? 0u : (uint32_t)g.lo;
    c.b_hi = nseg > 1 ? NB : (uint32_t)g.hi;
    c.bsh = 2 * (g.k - 10);
    c.shift = g.cell_shift;
    c.bb0 = g.bb0;
    c.seg_bin0 = g.seg_bin0;
    c.cells = g.cells;
    c.bcur = g.bcur;
    c.err = g.ctr + GC_ERR;
    const unsigned blocks = std::min<unsigned>(c.tiles, 2u * (unsigned)sm_count());
    if (blocks)
        (count_launch(), (reads ? k_split_bins<true> : k_split_bins<false>)<<<blocks, SP_THREADS, sizeof(BinSmem), st>>>(c));
    MP_CUDA(cudaGetLastError());
    return 0;
}

int group_bins_reads(GroupScan &g, const uint8_t *fq, const ParsedReads &pr, const std::vector<uint64_t> &seg_reads,
                     const uint32_t *label, uint64_t *k1, uint32_t *id1, DeviceArena &arena, cudaStream_t st)
{
    BinCtx c;
    c.t = read_tiles(fq, pr, g.k, pr.max_len, SP_THREADS);
    c.n_reads = (uint32_t)pr.n_reads;
    c.check_many = pr.max_len > (uint32_t)g.k + 254u;  // a read with 256 positions or more
    c.label = label;
    c.out_k = k1;
    c.out_id = id1;
    return launch_bins(g, c, seg_reads, arena, st);
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
    return launch_bins(g, c, g.seg_tstart, arena, st);
}

int group_units(GroupScan &g, const uint64_t *k1, const uint32_t *id1, uint64_t *k2, uint32_t *id2, cudaStream_t st)
{
    if (!g.two_level) return 0;
    const int bsh = 2 * (g.k - 10);
    const unsigned sms = (unsigned)sm_count();
    if (g.bin_shift <= 21)
        (count_launch(), k_split_units<GP_MAX_UNITS, 2><<<std::min(g.max_tiles, 2 * sms), SP_THREADS, sizeof(UnitSmem<GP_MAX_UNITS>), st>>>(
            k1, id1, (uint32_t)g.n, bsh, g.ctr, g.bstart, g.bb0, g.bu0, g.bcur, g.ub0, g.ucur, g.tile_bin, g.tile_first, k2, id2));
    else
        (count_launch(), k_split_units<GP_MAX_UNITS_L, 1><<<std::min(g.max_tiles, sms), SP_THREADS, sizeof(UnitSmem<GP_MAX_UNITS_L>), st>>>(
            k1, id1, (uint32_t)g.n, bsh, g.ctr, g.bstart, g.bb0, g.bu0, g.bcur, g.ub0, g.ucur, g.tile_bin, g.tile_first, k2, id2));
    MP_CUDA(cudaGetLastError());
    return 0;
}

int group_filter(GroupScan &g, const uint64_t *kk, const uint32_t *ids, uint32_t *out, uint32_t *parent, uint8_t *filtered,
                 DeviceArena &arena, cudaStream_t st)
{
    group_kernel_attrs();
    const uint32_t *fill = g.two_level ? g.ucur : g.bcur;
    GroupCtx c{kk, ids, g.ustart, g.ub0, fill, g.lrs, nullptr, g.ctr, g.qlist, g.quirk, GC_WORK_S, GC_UNITS, 0, (uint32_t)GP_CAP_S,
               out, parent, filtered};
    const unsigned sms = (unsigned)sm_count();
    (count_launch(), k_group<512, 12, 13><<<std::min(2 * sms, std::max(1u, g.hctr[GC_UNITS])), 512, sizeof(GroupSmemS), st>>>(c));
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
                                                                        g.ctr + GC_ERR, d_l));
        std::vector<uint32_t> hl(4 * (size_t)nb);
        MP_CUDA(cudaMemcpyAsync(hl.data(), d_l, hl.size() * 4, cudaMemcpyDeviceToHost, st));
        MP_CUDA(cudaStreamSynchronize(st));
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
            (count_launch(), k_gbig_reserve<<<1, 1, 0, st>>>(g.ctr, (uint32_t)acc, d_base));
            (count_launch(), k_gbig_emit<<<grid, 256, 0, st>>>(d_b + b0, d_base, tp.lo, tp.id, tp.z, g.ub0, g.hctr[GC_UNITS], g.lrs,
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
    (count_launch(), k_gp_quirk<<<64, 256, 0, st>>>(g.ctr, g.qlist, out, filtered, g.quirk));
    const unsigned blocks = std::min<unsigned>(8u * (unsigned)sm_count(), blocks_of(g.n, (int)GE_SEG * 8));
    uint32_t *err = arena.alloc<uint32_t>(1);
    if (!err) return set_error(MP_ENOMEM, "device memory");
    MP_CUDA(cudaMemsetAsync(err, 0, 4, st));
    (count_launch(), k_gp_union<<<blocks, 256, 0, st>>>(g.ctr, out, parent, filtered, err, arena.lim.union_retries));
    compress_parents(parent, n_reads, st);
    std::vector<uint32_t> h(GC_N + (size_t)nseg * QW);
    uint32_t herr = 0;
    MP_CUDA(cudaMemcpyAsync(h.data(), g.ctr, h.size() * 4, cudaMemcpyDeviceToHost, st));
    MP_CUDA(cudaMemcpyAsync(&herr, err, 4, cudaMemcpyDeviceToHost, st));
    MP_CUDA(cudaStreamSynchronize(st));
    MP_CUDA(cudaGetLastError());
    if (h[GC_ERR] & 4u)
        return set_error(MP_EUNSUP, "a read has 256 or more k-mers in one scan (the reference counts them in 8 bits, "
                                    "enumerateKmers.c:152)");
    if (h[GC_ERR] & 2u) return set_error(MP_EFMT, "the histogram does not match the scan's tuples");
    if (herr) return set_error(MP_EDEVICE, "union-find retry limit reached (flags 0x%x)", herr);
    for (int q = 0; q < nseg; q++) {
        const uint32_t *w = h.data() + GC_N + (size_t)q * QW;
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
