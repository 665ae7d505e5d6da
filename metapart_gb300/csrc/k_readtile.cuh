// Canonical k-mers of a tile of reads, straight from the FASTQ bytes.
//
// A block takes `rpt` consecutive reads.  Their bases are packed into shared memory, 32 per thread and turn with byte
// arithmetic on whole words, as three streams: 2-bit codes (first base in the top bits), bit 3 of every byte (with
// the code it is all that the filter reads of a neighbouring character) and N flags.  Then every thread takes P consecutive
// positions of one read: its first k-mer is a funnel shift of the packed codes, its reverse complement a bit reversal,
// and the next ones roll (countMmers.c:83-217, enumerateKmers.c:127-371 roll the same way over a whole read).
//
// Per position that is about 35 instructions of one thread; a warp per read with one position per lane (two warp
// reductions, a ballot, two 64-bit shifts and a bit reversal per 32 positions, and idle lanes at each read's end)
// took about three times as long.
#pragma once
#include "k_reads.cuh"

namespace mp {

constexpr int RT_P = 12;  // most positions per thread

struct ReadTiles {
    const uint8_t *fq = nullptr;
    const uint64_t *seq_off = nullptr;
    const uint32_t *seq_len = nullptr;
    int k = 0;
    uint32_t P = 1, spr = 1;      // positions per thread; threads per read
    uint32_t rpt = 1, rounds = 1; // reads per tile; rounds of 32 bases per read
    uint32_t words() const { return rpt * (4 * rounds + 8); }  // shared-memory words of a tile's packed reads
};

// The tiling of reads of at most max_len bases (longer than k) for blocks of `threads`.
inline ReadTiles read_tiles(const uint8_t *fq, const ParsedReads &pr, int k, uint32_t max_len, uint32_t threads)
{
    ReadTiles t;
    t.fq = fq;
    t.seq_off = pr.seq_off;
    t.seq_len = pr.seq_len;
    t.k = k;
    const uint32_t pos = max_len > (uint32_t)k ? max_len - (uint32_t)k + 1 : 1;
    t.spr = (pos + RT_P - 1) / RT_P;
    t.P = (pos + t.spr - 1) / t.spr;
    t.rpt = threads / t.spr ? threads / t.spr : 1;
    t.rounds = (max_len + 31) / 32;
    return t;
}

// Layout of a tile in shared memory: per read 2 * rounds + 4 code words, rounds + 2 bit-3 words, rounds + 2 N words
// (the last ones are read past the end, never used).
__device__ __forceinline__ uint32_t rt_stride(const ReadTiles &t) { return 4 * t.rounds + 8; }

__device__ __forceinline__ uint32_t pack_codes4(uint32_t w)  // four bytes' codes, the first in bits 7-6
{
    const uint32_t x = (w >> 1) & 0x03030303u;
    return ((x ^ ((x >> 1) & 0x01010101u)) * 0x40100401u) >> 24;
}
__device__ __forceinline__ uint32_t pack_bits4(uint32_t b)  // bit 0 of four bytes, the first in bit 0
{
    return ((b * 0x01020408u) >> 24) & 15u;
}

// Packs the reads [r0, r1) (at most rpt) into sm.  ODD: returns whether this thread saw a sequence byte other than A, C,
// G, T, N in a read with a k-mer.
template <bool ODD = false>
__device__ __forceinline__ bool rt_pack(const ReadTiles &t, uint64_t r0, uint64_t r1, uint32_t *sm)
{
    uint32_t odd = 0;
    const uint32_t n = (uint32_t)(r1 - r0), stride = rt_stride(t);
    for (uint32_t i = threadIdx.x; i < n * t.rounds; i += blockDim.x) {
        const uint32_t rr = i / t.rounds, rd = i - rr * t.rounds;
        const uint32_t L = t.seq_len[r0 + rr];
        if (32 * rd >= L) continue;
        const uint64_t a = t.seq_off[r0 + rr] + 32 * rd;
        const uintptr_t base = reinterpret_cast<uintptr_t>(t.fq) + a;
        const uint32_t *p = reinterpret_cast<const uint32_t *>(base & ~(uintptr_t)3);  // words of the buffer, its first byte included
        const uint32_t sh = (uint32_t)(base & 3) * 8;
        uint32_t w[9];
#pragma unroll
        for (int q = 0; q < 9; q++) w[q] = p[q];  // at most 35 bytes past the read's last round: inside the buffer's 64 spare bytes
        uint32_t c0 = 0, c1 = 0, b3 = 0, nn = 0;
#pragma unroll
        for (int q = 0; q < 8; q++) {
            const uint32_t v = __funnelshift_r(w[q], w[q + 1], sh);
            const uint32_t c = pack_codes4(v);
            if (q < 4) c0 |= c << (24 - 8 * q);
            else c1 |= c << (24 - 8 * (q - 4));
            b3 |= pack_bits4((v >> 3) & 0x01010101u) << (4 * q);
            const uint32_t z = v ^ 0x4E4E4E4Eu;  // zero bytes where the base is 'N'
            const uint32_t y = ~(((z & 0x7F7F7F7Fu) + 0x7F7F7F7Fu) | z | 0x7F7F7F7Fu);
            nn |= pack_bits4((y >> 7) & 0x01010101u) << (4 * q);
            if constexpr (ODD) {  // the letters of the codes against the bytes, the bytes past the read and N aside
                const uint32_t f = ((v >> 1) & 0x03030303u) ^ ((v >> 2) & 0x01010101u);
                const uint32_t sel = (f & 3u) | ((f >> 4) & 0x30u) | ((f >> 8) & 0x300u) | ((f >> 12) & 0x3000u);
                const uint32_t left = L > 32 * rd + 4 * q ? L - (32 * rd + 4 * q) : 0u;
                const uint32_t in = left >= 4 ? ~0u : (1u << (8 * left)) - 1;
                if (L > (uint32_t)t.k) odd |= (v ^ __byte_perm(0x54474341u, 0u, sel)) & in & ~((y >> 7) * 255u);
            }
        }
        uint32_t *s = sm + rr * stride;
        s[2 * rd] = c0;
        s[2 * rd + 1] = c1;
        s[2 * t.rounds + 4 + rd] = b3;
        s[3 * t.rounds + 6 + rd] = nn;
    }
    return odd != 0;
}

// A thread's positions [i0, i0 + n) of one packed read.
struct KmerRoll {
    uint64_t fwd, rc, nmask;   // nmask: N flags of the bases from the current position on
    uint32_t nx, pv, b3n, b3p; // the next characters' and the previous characters' codes and bits 3
    uint32_t i, last;          // current position, the read's last one
};

__device__ __forceinline__ void kr_init(KmerRoll &s, const ReadTiles &t, const uint32_t *w, uint32_t L, uint32_t i0)
{
    const uint32_t *b3 = w + 2 * t.rounds + 4, *nw = w + 3 * t.rounds + 6;
    const int k = t.k;
    {
        const uint32_t q = i0 >> 4, sh = 2 * (i0 & 15);
        const uint32_t a = w[q], b = w[q + 1], c = w[q + 2];
        s.fwd = (((uint64_t)__funnelshift_l(b, a, sh) << 32) | __funnelshift_l(c, b, sh)) >> (64 - 2 * k);
    }
    s.rc = revcomp(s.fwd, k);
    const uint32_t j = i0 + (uint32_t)k;
    s.nx = __funnelshift_l(w[(j >> 4) + 1], w[j >> 4], 2 * (j & 15));
    s.b3n = __funnelshift_r(b3[j >> 5], b3[(j >> 5) + 1], j & 31);
    if (i0) {
        const uint32_t p = i0 - 1;
        s.pv = __funnelshift_l(w[(p >> 4) + 1], w[p >> 4], 2 * (p & 15));
        s.b3p = __funnelshift_r(b3[p >> 5], b3[(p >> 5) + 1], p & 31);
    } else {
        s.pv = w[0] >> 2;
        s.b3p = b3[0] << 1;
    }
    const uint32_t q = i0 >> 5, sh = i0 & 31;
    s.nmask = __funnelshift_r(nw[q], nw[q + 1], sh) | ((uint64_t)__funnelshift_r(nw[q + 1], nw[q + 2], sh) << 32);
    s.i = i0;
    s.last = L - (uint32_t)k;
}

// The canonical k-mer at the current position; false when its window holds an N.
__device__ __forceinline__ bool kr_get(const KmerRoll &s, int k, uint64_t &canon)
{
    canon = s.fwd < s.rc ? s.fwd : s.rc;
    return (s.nmask & ((1ull << k) - 1)) == 0;
}

// The six adjacency bits the filter reads (the adjacency byte's low ones: after-code << 0, before-code << 3, complemented
// and exchanged when the reverse complement is the canonical one; 'N', code 7, at the read's ends).
__device__ __forceinline__ uint32_t kr_adj6(const KmerRoll &s)
{
    const uint32_t cn = s.nx >> 30, cp = s.pv >> 30;
    const uint32_t na = s.i < s.last ? (cn ^ (cn >> 1)) | ((s.b3n & 1u) << 2) : 7u;
    const uint32_t pa = s.i ? (cp ^ (cp >> 1)) | ((s.b3p & 1u) << 2) : 7u;
    if (s.fwd < s.rc) return (pa << 3) | na;
    return (((0x70001032u >> (4 * na)) & 7u) << 3) | ((0x70001032u >> (4 * pa)) & 7u);  // "TGAC   N" by character bits 1-3
}

__device__ __forceinline__ void kr_next(KmerRoll &s, int k)
{
    const uint32_t c = s.nx >> 30;
    s.fwd = ((s.fwd << 2) | c) & ((1ull << (2 * k)) - 1);
    s.rc = (s.rc >> 2) | ((uint64_t)(3u - c) << (2 * (k - 1)));
    s.nx <<= 2;
    s.pv <<= 2;
    s.b3n >>= 1;
    s.b3p >>= 1;
    s.nmask >>= 1;
    s.i++;
}

}  // namespace mp
