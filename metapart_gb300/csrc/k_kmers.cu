// K1 (m-mer histogram) and K2 (tuple enumeration) kernels.
//
// Counting (plain variant) takes the reads in tiles (k_readtile.cuh), as the grouped scans' enumeration does.  The
// enumeration in read order, for the sorted scans: one warp per read.  Each round of 32 bases is loaded with one
// coalesced byte load per lane; two warp OR-reductions pack the 2-bit base codes
// most-significant-first into a 64-bit word and a ballot gives the N mask.  Lane j
// of round t then owns k-mer position 32t+j: its forward code is a funnel shift of
// two packed words, its reverse complement a bit reversal, and the neighbouring
// characters of the adjacency byte come by shuffle (countMmers.c:83-217,
// enumerateKmers.c:127-371 compute the same codes with a rolling update).
//
// 3-minimizer variant: one thread per read running the reference's window logic
// (countMmers_3minimizers.c:83-271, enumerateKmers_3minimizers.c:129-470); it
// emits about three k-mers per read, so the base scan dominates either way.
#include <algorithm>

#include "k_kmers.cuh"
#include "k_readtile.cuh"

namespace mp {

constexpr unsigned FULL = 0xFFFFFFFFu;

struct Round {
    uint64_t W;  // codes of positions 32t..32t+31, position 32t in bits 63..62
    uint32_t N;  // bit j: position 32t+j is 'N'
    uint32_t c;  // this lane's character (position 32t+lane); the adjacency bytes take neighbours by shuffle
};

__device__ __forceinline__ void load_round(const uint8_t *s, uint32_t L, int t, int lane, Round &r)
{
    const uint32_t p = 32u * (uint32_t)t + (uint32_t)lane;
    const uint32_t c = p < L ? (uint32_t)s[p] : 0x41u;
    // lane j's code goes to bits 63-2j..62-2j of W: two warp OR-reductions build the halves
    const uint32_t f = fcode(c) << (30 - 2 * (lane & 15));
    const uint32_t hi = __reduce_or_sync(FULL, lane < 16 ? f : 0u), lo = __reduce_or_sync(FULL, lane < 16 ? 0u : f);
    r.W = ((uint64_t)hi << 32) | lo;
    r.N = __ballot_sync(FULL, p < L && c == 'N');
    r.c = c;
}

// Forward code, validity (no N in the window) of the k-mer at lane's position of round t.
__device__ __forceinline__ bool kmer_at(int lane, int k, const Round &c, const Round &n, uint64_t &fwd)
{
    const uint64_t x = lane ? ((c.W << (2 * lane)) | (n.W >> (64 - 2 * lane))) : c.W;
    fwd = x >> (64 - 2 * k);
    const uint64_t n64 = (uint64_t)c.N | ((uint64_t)n.N << 32);
    return ((n64 >> lane) & ((1ull << k) - 1)) == 0;
}

__device__ __forceinline__ uint32_t chunk_of(const uint64_t *chunk_rec, int nchunks, uint64_t r)
{
    int lo = 0, hi = nchunks - 1;  // largest c with chunk_rec[c] <= r
    while (lo < hi) {
        int mid = (lo + hi + 1) >> 1;
        if (chunk_rec[mid] <= r) lo = mid; else hi = mid - 1;
    }
    return (uint32_t)lo;
}

// ------------------------------------------------------------ K1 plain

constexpr int CT_THREADS = 256;
// Where a read is longer than CT_SPLIT, those above CT_LONG are counted by themselves, a block each: the longest sets the tiling
// of all, and from about 1,540 bases a tile is one read (600,000 reads of 100 bases and one of 4,000: counting 1.8 ms, apart
// 0.5; and one of 1,000: 0.7.  Apart wherever a read is above 512, a tenth of 900 bases 0.9 -> 1.15).
constexpr uint32_t CT_LONG = 512, CT_SPLIT = 1536;

struct CountOut {
    const uint64_t *chunk_rec;
    int nchunks;
    uint32_t *cc;
    unsigned long long *glob;
    uint32_t *err;
};

// The k-mers of the reads [r0, r0 + n) by one block; of those of at most `most` bases.  One reduction per k-mer: neighbouring
// positions almost never share a bucket, so grouping equal buckets first costs more than it saves.  ODD: a byte other
// than A, C, G, T, N sets DERR_NONACGT.
template <bool ODD, bool HI>
__device__ __forceinline__ void count_tile(const ReadTiles &t, uint64_t r0, uint32_t n, uint32_t most, const CountOut &o, uint32_t *packed)
{
    const uint32_t stride = rt_stride(t);
    const int sh = 2 * (t.k - 10);
    if (rt_pack<ODD>(t, r0, n, packed)) atomicOr(o.err, DERR_NONACGT);
    __syncthreads();
    for (uint32_t x = threadIdx.x; x < n * t.spr; x += CT_THREADS) {
        const uint32_t rr = x / t.spr, i0 = (x - rr * t.spr) * t.P, L = t.seq_len[r0 + rr];
        if (L <= (uint32_t)t.k || L > most || i0 > L - (uint32_t)t.k) continue;
        uint32_t *ccc = o.cc ? o.cc + (size_t)chunk_of(o.chunk_rec, o.nchunks, r0 + rr) * NB : nullptr;
        KmerRoll<HI> s;
        s.template init<false>(t, packed + rr * stride, L, i0);
#pragma unroll
        for (int j = 0; j < RT_P; j++) {
            if ((s.vm >> j) & 1u) {
                const uint64_t f = s.fwd(), r = s.rc();
                const uint32_t b = (uint32_t)((f < r ? f : r) >> sh);
                if (ccc) atomicAdd(&ccc[b], 1u);
                else atomicAdd(&o.glob[b], 1ull);
            }
            s.next();
        }
    }
    __syncthreads();
}

// m-mer counts of the reads of at most `most` bases, a tile of reads per block and turn (k_readtile.cuh).
template <bool ODD, bool HI>
__global__ void __launch_bounds__(CT_THREADS) k_count_tiles(ReadTiles t, uint64_t n_reads, uint32_t most, CountOut o)
{
    extern __shared__ __align__(16) uint32_t packed[];
    const uint64_t tiles = (n_reads + t.rpt - 1) / t.rpt;
    for (uint64_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        const uint64_t r0 = tile * t.rpt;
        count_tile<ODD, HI>(t, r0, (uint32_t)(min(n_reads, r0 + t.rpt) - r0), most, o, packed);
    }
}

// And of the longer ones, found among CT_THREADS reads at a time.
template <bool ODD, bool HI>
__global__ void __launch_bounds__(CT_THREADS) k_count_long(ReadTiles t, uint64_t n_reads, CountOut o)
{
    extern __shared__ __align__(16) uint32_t packed[];
    __shared__ uint16_t list[CT_THREADS];
    __shared__ uint32_t nl;
    for (uint64_t r0 = (uint64_t)blockIdx.x * CT_THREADS; r0 < n_reads; r0 += (uint64_t)gridDim.x * CT_THREADS) {
        const bool is_long = r0 + threadIdx.x < n_reads && t.seq_len[r0 + threadIdx.x] > CT_LONG;
        if (threadIdx.x == 0) nl = 0;
        if (!__syncthreads_or(is_long)) continue;
        if (is_long) list[atomicAdd(&nl, 1u)] = (uint16_t)threadIdx.x;
        __syncthreads();
        const uint32_t n = nl;
        for (uint32_t q = 0; q < n; q++) count_tile<ODD, HI>(t, r0 + list[q], 1, ~0u, o, packed);
    }
}

// ------------------------------------------------------- 3-minimizer core

// The adjacency byte of a minimum: at = 4 position + 2 its strand + the strand of the k-mer that ended its window.
__device__ __forceinline__ uint32_t min3_adj(const uint8_t *s, int L, int k, uint32_t at)
{
    const int m = (int)(at >> 2);
    uint32_t pa = m == 0 ? 7u : a5_of(s[m - 1]), na = m == L - k ? 7u : a5_of(s[m + k]);
    if (!(at & 2u)) {
        pa = a5_cmpl(pa);
        na = a5_cmpl(na);
    }
    return at & 1u ? ((pa << 3) | (na & 7)) : ((na << 3) | (pa & 7));
}

// One read, thread-sequential: emit(k-mer, at) for every window's minimum, at as min3_adj takes it.  ENUM: apply the scan
// range.  HI: 2k >= 34 (KmerRoll).
//
// Bound by its integer instructions (41 a character when every character was loaded, tested for N and for the window's end,
// and the minimum's neighbours kept along): eight characters are loaded and decoded at once, and eight k-mers of one window
// take only the roll and the comparison, about twenty.  3 million reads of 250 bases: counting 1.25 -> 0.92 ms,
// enumeration 3.5 (a counting and a writing pass) -> 1.43 ms.
template <bool ENUM, bool HI, class Emit>
__device__ __forceinline__ void min3_read(const uint8_t *s, int L, int k, uint32_t lo, uint32_t hi, Emit emit)
{
    if (L <= k) return;
    const int last = L - k, sh = 2 * (k - 10), win = last / 3;
    const uint64_t mask = kmer_mask(k);
    const uint32_t mh = (uint32_t)(mask >> 32);
    const int top = HI ? 2 * k - 34 : 2 * k - 2;
    uint32_t fl = 0, fh = 0, rl = 0, rh = 0;
    uint64_t mn1 = ~0ull;  // the current minimum less one: none, and the k-mer of code 0, give way to any (all ones)
    uint32_t mpf = 0;      // its position and strand
    int lastN = -1, next_win = win;
    const bool all = lo == 0 && hi >= NB;
    auto roll = [&](uint32_t fc) {
        if constexpr (HI) {
            fh = __funnelshift_l(fl, fh, 2) & mh;
            fl = (fl << 2) | fc;
            rl = __funnelshift_r(rl, rh, 2);
            rh = (rh >> 2) | ((fc ^ 3u) << top);
        } else {
            const uint64_t f = (((((uint64_t)fh << 32) | fl) << 2) | fc) & mask;
            const uint64_t r = ((((uint64_t)rh << 32) | rl) >> 2) | ((uint64_t)(fc ^ 3u) << top);
            fl = (uint32_t)f, fh = (uint32_t)(f >> 32), rl = (uint32_t)r, rh = (uint32_t)(r >> 32);
        }
    };
    auto flush = [&](bool f) {  // f: the strand of the k-mer that ends the window
        if (mn1 != ~0ull) emit(mn1 + 1, 2 * mpf + f);
    };
    const uint64_t *w = reinterpret_cast<const uint64_t *>(reinterpret_cast<uintptr_t>(s) & ~(uintptr_t)7);
    const uint32_t ws = (uint32_t)(reinterpret_cast<uintptr_t>(s) & 7) * 8;
    uint64_t w0 = w[0], w1 = w[1];
    for (int t0 = 0; t0 < L; t0 += 8) {
        const uint64_t c8 = ws ? (w0 >> ws) | (w1 << (64 - ws)) : w0;
        w0 = w1;
        w1 = w[t0 / 8 + 2];  // a turn ahead: at most 23 bytes past the read, inside the buffer's spare bytes
        const int i0 = t0 - (k - 1);  // the position whose last character is the first of these
        const uint32_t cl = (uint32_t)c8, ch = (uint32_t)(c8 >> 32);
        const bool plain = !(pack_n4(cl) | pack_n4(ch)) && t0 + 8 <= L;
        if (plain && (i0 < -7 || (i0 > lastN && i0 + 7 <= next_win && (!ENUM || all)))) {
            // eight characters of no k-mer yet, or eight k-mers of one window
            uint32_t x[2] = {(cl >> 1) & 0x03030303u, (ch >> 1) & 0x03030303u};
            x[0] ^= (x[0] >> 1) & 0x01010101u;
            x[1] ^= (x[1] >> 1) & 0x01010101u;
            if (i0 < -7) {
#pragma unroll
                for (int q = 0; q < 8; q++) roll((x[q >> 2] >> (8 * (q & 3))) & 3u);
            } else {
#pragma unroll
                for (int q = 0; q < 8; q++) {
                    roll((x[q >> 2] >> (8 * (q & 3))) & 3u);
                    const uint64_t fwd = ((uint64_t)fh << 32) | fl, rc = ((uint64_t)rh << 32) | rl;
                    const bool f = fwd < rc;
                    const uint64_t v = f ? fwd : rc;
                    if (v <= mn1) {
                        mn1 = v - 1;
                        mpf = 2 * (uint32_t)(i0 + q) + f;
                    }
                }
            }
            continue;
        }
        const int e = min(8, L - t0);
#pragma unroll 1
        for (int q = 0; q < e; q++) {
            const uint32_t c = (uint32_t)(c8 >> (8 * q)) & 0xFFu;
            const int i = i0 + q;
            roll(fcode(c));
            if (c == 'N') lastN = t0 + q;
            if (!(i > lastN && i >= 0)) continue;
            const uint64_t fwd = ((uint64_t)fh << 32) | fl, rc = ((uint64_t)rh << 32) | rl;
            const bool f = fwd < rc;
            const uint64_t v = f ? fwd : rc;
            if (ENUM && !all) {
                const uint32_t b = (uint32_t)(v >> sh);
                if (!(b >= lo && b < hi)) continue;
            }
            if (i > next_win) {
                flush(f);
                mn1 = ~0ull;
                next_win += win;
                if (next_win + win > last) next_win = last;
            }
            if (v <= mn1) {
                mn1 = v - 1;
                mpf = 2 * (uint32_t)i + f;
            }
        }
    }
    flush(false);
}

template <bool HI>
__global__ void k_count_min3(const uint8_t *fq, const uint64_t *seq_off, const uint32_t *seq_len, uint64_t r0, uint64_t r1,
                             int k, const uint64_t *chunk_rec, int nchunks, uint32_t *cc, unsigned long long *glob,
                             uint32_t *err)
{
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    const int sh = 2 * (k - 10);
    for (uint64_t r = r0 + (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; r < r1; r += stride) {
        const uint32_t L = seq_len[r];
        if (L > (uint32_t)MAX_READ_COUNT) { atomicOr(err, DERR_LONG_READ); continue; }
        uint32_t *ccc = cc ? cc + (size_t)chunk_of(chunk_rec, nchunks, r) * NB : nullptr;
        min3_read<false, HI>(fq + seq_off[r], (int)L, k, 0, 0, [&](uint64_t v, uint32_t) {
            const uint32_t b = (uint32_t)(v >> sh);
            if (ccc) atomicAdd(&ccc[b], 1u); else atomicAdd(&glob[b], 1ull);
        });
    }
}

// Global histogram from per-chunk counts: hist_cnt[b] = sum over chunks.
__global__ void k_sum_chunks(const uint32_t *cc, int nchunks, unsigned long long *glob)
{
    const uint32_t b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= NB) return;
    unsigned long long s = 0;
    for (int c = 0; c < nchunks; c++) s += cc[(size_t)c * NB + b];
    glob[b] = s;
}

// ------------------------------------------------------------ K2 plain

template <bool WRITE>
__global__ void __launch_bounds__(256) k_enum_plain(const uint8_t *fq, const uint64_t *seq_off, const uint32_t *seq_len,
                                                    uint64_t n_reads, int k, uint32_t lo, uint32_t hi,
                                                    const uint32_t *label, const uint64_t *out_off, uint32_t *cnt,
                                                    uint64_t *o_lo, uint8_t *o_hi, uint32_t *o_id, uint32_t *err)
{
    const int lane = threadIdx.x & 31;
    const uint64_t nw = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    const int sh = 2 * (k - 10);
    for (uint64_t r = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; r < n_reads; r += nw) {
        const uint32_t L = seq_len[r];
        if (L <= (uint32_t)k) {
            if (!WRITE && lane == 0) cnt[r] = 0;
            continue;
        }
        if (L > 32u * MAX_ROUNDS_ENUM || L - (uint32_t)k >= 300u) {
            if (lane == 0) { atomicOr(err, DERR_LONG_READ); if (!WRITE) cnt[r] = 0; }
            continue;
        }
        const uint8_t *s = fq + seq_off[r];
        auto load = [&](int t, Round &x) { load_round(s, L, t, lane, x); };
        const int last = (int)L - k;
        uint64_t base = WRITE ? out_off[r] : 0;
        uint32_t id = (uint32_t)r;
        if (WRITE && label) {
            const uint32_t p = label[r];
            id = (p == BAD) ? (uint32_t)r : p;  // findRoot after full compression (metapart.c:543-568)
        }
        Round prv, cur, nxt;
        load(0, cur);
        load(1, nxt);
        prv = cur;
        uint32_t total = 0;
        for (int t = 0; 32 * t <= last; t++) {
            const int i = 32 * t + lane;
            uint64_t fwd;
            const bool v0 = kmer_at(lane, k, cur, nxt, fwd) && i <= last;
            const uint64_t rc = revcomp(fwd, k);
            const bool f = fwd < rc;
            const uint64_t canon = f ? fwd : rc;
            const uint32_t b = (uint32_t)(canon >> sh);
            const bool v = v0 && b >= lo && b < hi;
            const uint32_t bal = __ballot_sync(FULL, v);
            uint32_t pc = 0, nc = 0;  // characters before and after this lane's k-mer
            if (WRITE) {
                const uint32_t x = __shfl_sync(FULL, cur.c, (lane + 31) & 31), y = __shfl_sync(FULL, prv.c, 31);
                pc = lane ? x : y;
                const int q = lane + k;
                const uint32_t u = __shfl_sync(FULL, cur.c, q & 31), w = __shfl_sync(FULL, nxt.c, q & 31);
                nc = q < 32 ? u : w;
            }
            if (WRITE && v) {
                // 'N' at the read ends (enumerateKmers.c:177, 252-255)
                const uint32_t pa = i > 0 ? a5_of(pc) : 7u, na = i < last ? a5_of(nc) : 7u;
                const uint32_t adj = f ? adj_fwd(pa, na) : adj_rc(pa, na);
                const uint64_t pos = base + __popc(bal & ((1u << lane) - 1));
                o_lo[pos] = (canon << 8) | adj;
                if (o_hi) o_hi[pos] = (uint8_t)(canon >> 56);
                o_id[pos] = id;
            }
            base += __popc(bal);
            total += __popc(bal);
            prv = cur;
            cur = nxt;
            load(t + 2, nxt);
        }
        if (!WRITE && lane == 0) {
            cnt[r] = total;
            if (total > 255) atomicOr(err, DERR_TOO_MANY);  // the reference's per-read counter is a uint8_t
        }
    }
}

// Tuples per read of every scan in one pass: scan s holds buckets [bounds[s], bounds[s+1]).
// cnt[s * stride + r]; S <= MAX_SCAN_COUNT.
constexpr int MAX_SCAN_COUNT = 8;

__global__ void __launch_bounds__(256) k_enum_count_scans(const uint8_t *fq, const uint64_t *seq_off,
                                                          const uint32_t *seq_len, uint64_t n_reads, int k,
                                                          const uint32_t *bounds, int S, uint32_t *cnt, uint64_t stride,
                                                          uint32_t *err)
{
    __shared__ uint32_t sb[MAX_SCAN_COUNT + 1];
    if (threadIdx.x <= (unsigned)S) sb[threadIdx.x] = bounds[threadIdx.x];
    __syncthreads();
    const int lane = threadIdx.x & 31;
    const uint64_t nw = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    const int sh = 2 * (k - 10);
    const uint32_t b_lo = sb[0], b_hi = sb[S];
    for (uint64_t r = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; r < n_reads; r += nw) {
        const uint32_t L = seq_len[r];
        uint32_t c[MAX_SCAN_COUNT];
#pragma unroll
        for (int q = 0; q < MAX_SCAN_COUNT; q++) c[q] = 0;
        if (L > (uint32_t)k && (L > 32u * MAX_ROUNDS_ENUM || L - (uint32_t)k >= 300u)) {
            if (lane == 0) atomicOr(err, DERR_LONG_READ);
        } else if (L > (uint32_t)k) {
            const uint8_t *s = fq + seq_off[r];
            auto load = [&](int t, Round &x) { load_round(s, L, t, lane, x); };
            const int last = (int)L - k;
            Round cur, nxt;
            load(0, cur);
            load(1, nxt);
            for (int t = 0; 32 * t <= last; t++) {
                const int i = 32 * t + lane;
                uint64_t fwd;
                const bool v0 = kmer_at(lane, k, cur, nxt, fwd) && i <= last;
                const uint64_t rc = revcomp(fwd, k);
                const uint32_t b = (uint32_t)((fwd < rc ? fwd : rc) >> sh);
                if (v0 && b >= b_lo && b < b_hi) {
                    int sc = 0;
#pragma unroll
                    for (int q = 1; q < MAX_SCAN_COUNT; q++) sc += (q < S && b >= sb[q]) ? 1 : 0;
#pragma unroll
                    for (int q = 0; q < MAX_SCAN_COUNT; q++) c[q] += (sc == q) ? 1u : 0u;
                }
                cur = nxt;
                load(t + 2, nxt);
            }
        }
        for (int q = 0; q < S; q++) {
            uint32_t x = c[q];
#pragma unroll
            for (int o = 16; o; o >>= 1) x += __shfl_xor_sync(FULL, x, o);
            if (lane == 0) {
                cnt[(uint64_t)q * stride + r] = x;
                if (x > 255) atomicOr(err, DERR_TOO_MANY);  // the reference's per-read counter is a uint8_t
            }
        }
    }
}

// ------------------------------------------------------------- K2 3-min

template <bool WRITE, bool HI>
__global__ void k_enum_min3(const uint8_t *fq, const uint64_t *seq_off, const uint32_t *seq_len, uint64_t n_reads, int k,
                            uint32_t lo, uint32_t hi, const uint32_t *label, const uint64_t *out_off, uint32_t *cnt,
                            uint64_t *o_lo, uint8_t *o_hi, uint32_t *o_id, uint32_t *err)
{
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t r = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; r < n_reads; r += stride) {
        const uint32_t L = seq_len[r];
        if (L > (uint32_t)k && L - (uint32_t)k >= 300u) {
            atomicOr(err, DERR_LONG_READ);
            if (!WRITE) cnt[r] = 0;
            continue;
        }
        uint32_t id = (uint32_t)r;
        if (WRITE && label) { const uint32_t p = label[r]; id = (p == BAD) ? (uint32_t)r : p; }
        uint64_t pos = WRITE ? out_off[r] : 0;
        const uint64_t end = WRITE ? out_off[r + 1] : 0;
        uint32_t c = 0;
        min3_read<true, HI>(fq + seq_off[r], (int)L, k, lo, hi, [&](uint64_t v, uint32_t at) {
            if constexpr (WRITE) {
                if (pos < end) {
                    o_lo[pos] = (v << 8) | min3_adj(fq + seq_off[r], (int)L, k, at);
                    if (o_hi) o_hi[pos] = (uint8_t)(v >> 56);
                    o_id[pos] = id;
                } else {
                    atomicOr(err, DERR_OVERFLOW);
                }
                pos++;
            }
            c++;
        });
        if (!WRITE) {
            cnt[r] = c;
            if (c > 255) atomicOr(err, DERR_TOO_MANY);
        }
    }
}

// The same in one pass and no order: a block's reads keep their tuples in shared memory (three each, as a rule) and take
// their places with one addition a block -- one a warp and window was bound by the additions to one address (1.8 ms for 3
// million reads).  Tuples past n are counted and not written.
constexpr int EM_THREADS = 128, EM_KEEP = 4;

template <bool HI>
__global__ void __launch_bounds__(EM_THREADS) k_enum_min3_any(const uint8_t *fq, const uint64_t *seq_off, const uint32_t *seq_len,
                                                              uint64_t n_reads, int k, uint32_t lo, uint32_t hi, const uint32_t *label,
                                                              unsigned long long *total, uint64_t n, uint64_t *o_lo, uint8_t *o_hi,
                                                              uint32_t *o_id, uint32_t *err)
{
    __shared__ uint64_t kv[EM_KEEP][EM_THREADS];
    __shared__ uint32_t ka[EM_KEEP][EM_THREADS];
    __shared__ uint32_t ws[EM_THREADS / 32];
    __shared__ unsigned long long place;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (uint64_t r0 = (uint64_t)blockIdx.x * EM_THREADS; r0 < n_reads; r0 += (uint64_t)gridDim.x * EM_THREADS) {
        const uint64_t r = r0 + threadIdx.x;
        const uint32_t L = r < n_reads ? seq_len[r] : 0u;
        uint32_t id = (uint32_t)r, c = 0;
        if (L > (uint32_t)k && L - (uint32_t)k >= 300u) {
            atomicOr(err, DERR_LONG_READ);
        } else if (L > (uint32_t)k) {
            if (label && label[r] != BAD) id = label[r];
            min3_read<true, HI>(fq + seq_off[r], (int)L, k, lo, hi, [&](uint64_t v, uint32_t at) {
                if (c < (uint32_t)EM_KEEP) {
                    kv[c][threadIdx.x] = v;
                    ka[c][threadIdx.x] = at;
                } else {  // (windows of no position: a short read)
                    const unsigned long long pos = atomicAdd(total, 1ull);
                    if (pos < n) {
                        o_lo[pos] = (v << 8) | min3_adj(fq + seq_off[r], (int)L, k, at);
                        if (o_hi) o_hi[pos] = (uint8_t)(v >> 56);
                        o_id[pos] = id;
                    }
                }
                c++;
            });
            if (c > 255) atomicOr(err, DERR_TOO_MANY);
        }
        const uint32_t m = min(c, (uint32_t)EM_KEEP);
        uint32_t x = m;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(FULL, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) ws[warp] = x;
        __syncthreads();
        uint32_t before = x - m, all = 0;
#pragma unroll
        for (int q = 0; q < EM_THREADS / 32; q++) {
            if (q < warp) before += ws[q];
            all += ws[q];
        }
        if (threadIdx.x == 0) place = atomicAdd(total, (unsigned long long)all);
        __syncthreads();
#pragma unroll
        for (uint32_t q = 0; q < (uint32_t)EM_KEEP; q++) {
            const unsigned long long pos = place + before + q;
            if (q >= m || pos >= n) continue;
            const uint64_t v = kv[q][threadIdx.x];
            o_lo[pos] = (v << 8) | min3_adj(fq + seq_off[r], (int)L, k, ka[q][threadIdx.x]);
            if (o_hi) o_hi[pos] = (uint8_t)(v >> 56);
            o_id[pos] = id;
        }
        __syncthreads();
    }
}

// ------------------------------------------------------------- host side

// Blocks for `work` items at per_block each, at most `waves` blocks per SM.
static unsigned grid_for(uint64_t work, int per_block, int waves = 16)
{
    const uint64_t max_blocks = (uint64_t)waves * (uint64_t)sm_count();
    uint64_t g = (work + per_block - 1) / per_block;
    if (g < 1) g = 1;
    if (g > max_blocks) g = max_blocks;
    return (unsigned)g;
}

void launch_count(const uint8_t *fq, const ParsedReads &pr, int k, int min3, const uint64_t *chunk_rec, int nchunks,
                  uint32_t *cc, unsigned long long *glob, uint32_t *err, cudaStream_t st, bool odd)
{
    if (min3)
        (mp::count_launch(), (k >= 17 ? k_count_min3<true> : k_count_min3<false>)<<<grid_for(pr.n_reads, 128, 32), 128, 0, st>>>(fq, pr.seq_off, pr.seq_len, 0, pr.n_reads, k,
                                                                          chunk_rec, nchunks, cc, glob, err));
    else if (pr.max_len > (uint32_t)k) {
        const CountOut o{chunk_rec, nchunks, cc, glob, err};
        const uint32_t most = pr.max_len > CT_SPLIT ? CT_LONG : pr.max_len;
        const ReadTiles t = read_tiles(fq, pr, k, most, CT_THREADS, 4096);
        auto kern = odd ? (k >= 17 ? k_count_tiles<true, true> : k_count_tiles<true, false>)
                        : (k >= 17 ? k_count_tiles<false, true> : k_count_tiles<false, false>);
        (mp::count_launch(), kern<<<grid_for(pr.n_reads, (int)t.rpt, 16), CT_THREADS, t.words() * 4, st>>>(t, pr.n_reads, most, o));
        if (pr.max_len > CT_SPLIT) {
            ReadTiles l = read_tiles(fq, pr, k, std::min<uint32_t>(pr.max_len, (uint32_t)MAX_READ_COUNT), CT_THREADS, 4096);
            l.rpt = 1;
            auto kern_long = odd ? (k >= 17 ? k_count_long<true, true> : k_count_long<true, false>)
                                 : (k >= 17 ? k_count_long<false, true> : k_count_long<false, false>);
            (mp::count_launch(), kern_long<<<grid_for(pr.n_reads, CT_THREADS, 8), CT_THREADS, l.words() * 4, st>>>(l, pr.n_reads, o));
        }
    }
    if (cc && glob) (mp::count_launch(), k_sum_chunks<<<NB / 256, 256, 0, st>>>(cc, nchunks, glob));
}

void launch_enum_count(const uint8_t *fq, const ParsedReads &pr, int k, int min3, uint32_t lo, uint32_t hi,
                       uint32_t *cnt, uint32_t *err, cudaStream_t st)
{
    if (min3)
        (mp::count_launch(), (k >= 17 ? k_enum_min3<false, true> : k_enum_min3<false, false>)<<<grid_for(pr.n_reads, 128, 32), 128, 0,
                                                                                               st>>>(
            fq, pr.seq_off, pr.seq_len, pr.n_reads, k, lo, hi, nullptr, nullptr, cnt, nullptr, nullptr, nullptr, err));
    else
        (mp::count_launch(), k_enum_plain<false><<<grid_for(pr.n_reads, 8), 256, 0, st>>>(fq, pr.seq_off, pr.seq_len, pr.n_reads, k, lo, hi,
                                                                     nullptr, nullptr, cnt, nullptr, nullptr, nullptr, err));
}

int launch_enum_count_scans(const uint8_t *fq, const ParsedReads &pr, int k, const uint32_t *bounds, int S,
                            uint32_t *cnt, uint64_t stride, uint32_t *err, cudaStream_t st)
{
    if (S < 1 || S > MAX_SCAN_COUNT) return -1;
    (mp::count_launch(), k_enum_count_scans<<<grid_for(pr.n_reads, 8), 256, 0, st>>>(
        fq, pr.seq_off, pr.seq_len, pr.n_reads, k, bounds, S, cnt, stride, err));
    return 0;
}

void launch_enum_write(const uint8_t *fq, const ParsedReads &pr, int k, int min3, uint32_t lo, uint32_t hi,
                       const uint32_t *label, const uint64_t *off, uint64_t *o_lo, uint8_t *o_hi, uint32_t *o_id,
                       uint32_t *err, cudaStream_t st)
{
    if (min3)
        (mp::count_launch(), (k >= 17 ? k_enum_min3<true, true> : k_enum_min3<true, false>)<<<grid_for(pr.n_reads, 128, 32), 128, 0,
                                                                                             st>>>(
            fq, pr.seq_off, pr.seq_len, pr.n_reads, k, lo, hi, label, off, nullptr, o_lo, o_hi, o_id, err));
    else
        (mp::count_launch(), k_enum_plain<true><<<grid_for(pr.n_reads, 8), 256, 0, st>>>(fq, pr.seq_off, pr.seq_len, pr.n_reads, k, lo, hi,
                                                                    label, off, nullptr, o_lo, o_hi, o_id, err));
}

void launch_enum_min3(const uint8_t *fq, const ParsedReads &pr, int k, uint32_t lo, uint32_t hi, const uint32_t *label,
                      unsigned long long *total, uint64_t n, uint64_t *o_lo, uint8_t *o_hi, uint32_t *o_id, uint32_t *err,
                      cudaStream_t st)
{
    (mp::count_launch(), (k >= 17 ? k_enum_min3_any<true> : k_enum_min3_any<false>)<<<grid_for(pr.n_reads, EM_THREADS, 64), EM_THREADS,
                                                                                     0, st>>>(
        fq, pr.seq_off, pr.seq_len, pr.n_reads, k, lo, hi, label, total, n, o_lo, o_hi, o_id, err));
}

}  // namespace mp
