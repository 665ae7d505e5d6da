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
// (at most max_words of shared memory a tile, a read at least).
inline ReadTiles read_tiles(const uint8_t *fq, const ParsedReads &pr, int k, uint32_t max_len, uint32_t threads, uint32_t max_words)
{
    ReadTiles t;
    t.fq = fq;
    t.seq_off = pr.seq_off;
    t.seq_len = pr.seq_len;
    t.k = k;
    const uint32_t pos = max_len > (uint32_t)k ? max_len - (uint32_t)k + 1 : 1;
    t.spr = (pos + RT_P - 1) / RT_P;
    t.P = (pos + t.spr - 1) / t.spr;
    t.rounds = (max_len + 31) / 32;
    t.rpt = threads / t.spr;
    if (t.rpt > max_words / (4 * t.rounds + 8)) t.rpt = max_words / (4 * t.rounds + 8);
    if (t.rpt < 1) t.rpt = 1;
    return t;
}

// Layout of a tile in shared memory: per read 2 * rounds + 4 code words, rounds + 2 bit-3 words, rounds + 2 N words
// (the last ones are read past the end, never used).
__device__ __forceinline__ uint32_t rt_stride(const ReadTiles &t) { return 4 * t.rounds + 8; }

__device__ __forceinline__ uint32_t pack_codes4(uint32_t w)  // four bytes' codes in bits 31-24, the first in 31-30
{
    const uint32_t x = (w >> 1) & 0x03030303u;
    return (x ^ ((x >> 1) & 0x01010101u)) * 0x40100401u;
}
__device__ __forceinline__ uint32_t pack_bit3(uint32_t w)  // bit 3 of four bytes in bits 31-28, the first in 28
{
    return (w & 0x08080808u) * 0x02040810u;
}
__device__ __forceinline__ uint32_t pack_n4(uint32_t w)  // the same for the bytes that are 'N'
{
    const uint32_t z = w ^ 0x4E4E4E4Eu;
    return ((~(((z & 0x7F7F7F7Fu) + 0x7F7F7F7Fu) | z | 0x7F7F7F7Fu) >> 4) & 0x08080808u) * 0x02040810u;
}

// One round of 32 bases of a tile's read: fetch takes its bytes into registers, pack leaves it in shared memory.
struct RoundFetch {
    uint32_t w[9], sh, L;  // L: the read's length, 0 when there is nothing to pack
    uint32_t rr, rd;
};

__device__ __forceinline__ void rt_fetch(const ReadTiles &t, uint64_t r0, uint32_t n, uint32_t i, RoundFetch &f)
{
    f.L = 0;
    if (i >= n * t.rounds) return;
    f.rr = i / t.rounds;
    f.rd = i - f.rr * t.rounds;
    const uint32_t L = t.seq_len[r0 + f.rr];
    const uint64_t a = t.seq_off[r0 + f.rr] + 32 * f.rd;
    if (32 * f.rd >= L) return;
    f.L = L;
    const uintptr_t base = reinterpret_cast<uintptr_t>(t.fq) + a;
    const uint32_t *p = reinterpret_cast<const uint32_t *>(base & ~(uintptr_t)3);  // words of the buffer, its first byte included
    f.sh = (uint32_t)(base & 3) * 8;
#pragma unroll
    for (int q = 0; q < 9; q++) f.w[q] = p[q];  // at most 35 bytes past the read's last round: inside the buffer's 64 spare bytes
}

// ODD: returns whether the round holds a sequence byte other than A, C, G, T, N of a read with a k-mer.
template <bool ODD = false>
__device__ __forceinline__ bool rt_pack_round(const ReadTiles &t, const RoundFetch &f, uint32_t *sm)
{
    if (f.L == 0) return false;
    uint32_t odd = 0, w[8], c0 = 0, c1 = 0, b3 = 0, nn = 0;
#pragma unroll
    for (int q = 0; q < 8; q++) w[q] = __funnelshift_r(f.w[q], f.w[q + 1], f.sh);
#pragma unroll
    for (int q = 0; q < 4; q++) {
        c0 = __funnelshift_l(pack_codes4(w[q]), c0, 8);
        c1 = __funnelshift_l(pack_codes4(w[q + 4]), c1, 8);
    }
#pragma unroll
    for (int q = 7; q >= 0; q--) b3 = __funnelshift_l(pack_bit3(w[q]), b3, 4);
    const uint32_t left = f.L - 32 * f.rd, in = left >= 32 ? ~0u : (1u << left) - 1;
    if (b3 & in) {  // 'N' has bit 3 set, A, C, G and T have not
#pragma unroll
        for (int q = 7; q >= 0; q--) nn = __funnelshift_l(pack_n4(w[q]), nn, 4);
    }
    if constexpr (ODD) {  // the letters of the codes against the bytes, the bytes past the read and N aside
#pragma unroll
        for (int q = 0; q < 8; q++) {
            const uint32_t g = ((w[q] >> 1) & 0x03030303u) ^ ((w[q] >> 2) & 0x01010101u);
            const uint32_t sel = (g & 3u) | ((g >> 4) & 0x30u) | ((g >> 8) & 0x300u) | ((g >> 12) & 0x3000u);
            const uint32_t d = w[q] ^ __byte_perm(0x54474341u, 0u, sel);
#pragma unroll
            for (int x = 0; x < 4; x++)
                if ((d >> (8 * x)) & 0xFFu) odd |= in & ~nn & (1u << (4 * q + x));
        }
        if (f.L <= (uint32_t)t.k) odd = 0;
    }
    uint32_t *s = sm + f.rr * rt_stride(t);
    s[2 * f.rd] = c0;
    s[2 * f.rd + 1] = c1;
    s[2 * t.rounds + 4 + f.rd] = b3;
    s[3 * t.rounds + 6 + f.rd] = nn;
    return odd != 0;
}

// Packs the reads [r0, r0 + n) (at most rpt) into sm.
template <bool ODD = false>
__device__ __forceinline__ bool rt_pack(const ReadTiles &t, uint64_t r0, uint32_t n, uint32_t *sm)
{
    bool odd = false;
    for (uint32_t i = threadIdx.x; i < n * t.rounds; i += blockDim.x) {
        RoundFetch f;
        rt_fetch(t, r0, n, i, f);
        odd |= rt_pack_round<ODD>(t, f, sm);
    }
    return odd;
}

// A thread's positions [i0, i0 + P) of one packed read.  HI: 2k >= 34, so the rolling touches the high words only where
// it has to (half the instructions of 64-bit shifts by a runtime k).
template <bool HI> struct KmerRoll {
    uint32_t fl, fh, rl, rh;    // forward code and reverse complement, low and high words
    uint32_t nx;                // the next characters' codes
    uint32_t an[2], ap[2];      // character bits 1-3 of the next and the previous characters, a nibble each (position j in
                                // nibble j; 7, 'N', at the read's ends)
    uint32_t vm;                // bit j: position i0 + j holds a k-mer (inside the read, no N in its window)
    uint32_t mh, sh;            // HI: mask of the high word, place of a base in it; else 2 (k - 1)
    uint64_t mask;

    __device__ __forceinline__ uint64_t fwd() const { return ((uint64_t)fh << 32) | fl; }
    __device__ __forceinline__ uint64_t rc() const { return ((uint64_t)rh << 32) | rl; }

    // ADJ: with the neighbouring characters (adj6).
    template <bool ADJ = true> __device__ __forceinline__ void init(const ReadTiles &t, const uint32_t *w, uint32_t L, uint32_t i0)
    {
        const uint32_t *b3 = w + 2 * t.rounds + 4, *nw = w + 3 * t.rounds + 6;
        const int k = t.k;
        {
            const uint32_t q = i0 >> 4, s = 2 * (i0 & 15);
            const uint32_t a = w[q], b = w[q + 1], c = w[q + 2];
            const uint64_t f = (((uint64_t)__funnelshift_l(b, a, s) << 32) | __funnelshift_l(c, b, s)) >> (64 - 2 * k);
            const uint64_t r = revcomp(f, k);
            fl = (uint32_t)f;
            fh = (uint32_t)(f >> 32);
            rl = (uint32_t)r;
            rh = (uint32_t)(r >> 32);
        }
        mask = (1ull << (2 * k)) - 1;
        mh = (uint32_t)(mask >> 32);
        sh = HI ? 2 * k - 34 : 2 * k - 2;
        const uint32_t j = i0 + (uint32_t)k, last = L - (uint32_t)k, e = last - i0;
        nx = __funnelshift_l(w[(j >> 4) + 1], w[j >> 4], 2 * (j & 15));
        if constexpr (ADJ) {
            nibbles(an, nx, __funnelshift_r(b3[j >> 5], b3[(j >> 5) + 1], j & 31));
            if (e < 8) an[0] |= 7u << (4 * e);  // no character after the read's last k-mer
            else if (e < 16) an[1] |= 7u << (4 * (e - 8));
            const uint32_t p = i0 ? i0 - 1 : 0;
            nibbles(ap, __funnelshift_l(w[(p >> 4) + 1], w[p >> 4], 2 * (p & 15)), __funnelshift_r(b3[p >> 5], b3[(p >> 5) + 1], p & 31));
            if (i0 == 0) {  // nor before its first one
                ap[1] = (ap[1] << 4) | (ap[0] >> 28);
                ap[0] = (ap[0] << 4) | 7u;
            }
        }
        const uint32_t m = min(t.P, e + 1);
        vm = (1u << m) - 1;
        const uint32_t q = i0 >> 5, s = i0 & 31;
        const uint64_t nm = __funnelshift_r(nw[q], nw[q + 1], s) | ((uint64_t)__funnelshift_r(nw[q + 1], nw[q + 2], s) << 32);
        if (nm)
            for (uint32_t x = 0; x < m; x++)
                if ((nm >> x) & ((1ull << k) - 1)) vm &= ~(1u << x);
    }

    // Sixteen characters' bits 1-3 (bits 1-2 from the codes, first code in the top bits; bit 3 from b, first in bit 0) as
    // nibbles, the first in the lowest.
    static __device__ __forceinline__ void nibbles(uint32_t (&o)[2], uint32_t codes, uint32_t b)
    {
        const uint32_t rev = __brev(codes);  // first code in bits 1-0, its two bits exchanged
#pragma unroll
        for (int q = 0; q < 2; q++) {
            uint32_t v = (rev >> (16 * q)) & 0xFFFFu, y = (b >> (8 * q)) & 0xFFu;
            v = (v | (v << 8)) & 0x00FF00FFu;
            v = (v | (v << 4)) & 0x0F0F0F0Fu;
            v = (v | (v << 2)) & 0x33333333u;
            v = ((v << 1) & 0x22222222u) | (((v >> 1) ^ v) & 0x11111111u);  // the code's gray form, its bits in place
            y = (y | (y << 12)) & 0x000F000Fu;
            y = (y | (y << 6)) & 0x03030303u;
            y = (y | (y << 3)) & 0x11111111u;
            o[q] = v | (y << 2);
        }
    }

    // "TGAC   N" by character bits 1-3, eight nibbles at a time: 0-3 with bit 1 flipped, 7 itself, 4-6 none.
    static __device__ __forceinline__ uint32_t compl_nibbles(uint32_t v)
    {
        const uint32_t h = (v >> 2) & 0x11111111u, h7 = h & (v >> 1) & v;
        return ((v ^ 0x22222222u) & ~(h * 7u)) | (h7 * 7u);
    }

    // The six adjacency bits the filter reads of position J (the adjacency byte's low ones: code of the character after the
    // k-mer in bits 0-2, of the one before in 3-5, complemented and exchanged when the reverse complement is the
    // canonical one; cn and cp: compl_nibbles of an and ap).
    template <int J> __device__ __forceinline__ uint32_t adj6(bool f, const uint32_t (&cn)[2], const uint32_t (&cp)[2]) const
    {
        const uint32_t b = f ? ap[J / 8] : cn[J / 8], a = f ? an[J / 8] : cp[J / 8];
        constexpr int s = 4 * (J % 8);
        return ((s >= 3 ? b >> (s - 3) : b << 3) & 0x38u) | ((a >> s) & 7u);
    }

    __device__ __forceinline__ void next()
    {
        const uint32_t c = nx >> 30;
        nx <<= 2;
        if constexpr (HI) {
            fh = __funnelshift_l(fl, fh, 2) & mh;
            fl = (fl << 2) | c;
            rl = __funnelshift_r(rl, rh, 2);
            rh = (rh >> 2) | ((c ^ 3u) << sh);
        } else {
            const uint64_t f = ((fwd() << 2) | c) & mask, r = (rc() >> 2) | ((uint64_t)(c ^ 3u) << sh);
            fl = (uint32_t)f;
            fh = (uint32_t)(f >> 32);
            rl = (uint32_t)r;
            rh = (uint32_t)(r >> 32);
        }
    }
};

}  // namespace mp
