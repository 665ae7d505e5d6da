// K0: FASTQ parsing on the GPU, plus the device-wide exclusive scans every stage uses.
//
// A record is four '\n'-terminated lines (header, sequence, '+', quality) with the
// quality as long as the sequence -- the walk getNextRead does (genHistograms.c:60-80,
// metapart.c:296-369).  The parser finds every newline with coalesced 16-byte loads,
// compacts their positions in order, and derives the record table from every fourth one.
#include <algorithm>
#include <cstdio>

#include "k_reads.cuh"

namespace mp {

// ------------------------------------------------------------------ scans

constexpr int SCAN_THREADS = 256;
constexpr int SCAN_ITEMS = 16;
constexpr int SCAN_TILE = SCAN_THREADS * SCAN_ITEMS;

template <typename T>
__device__ __forceinline__ uint64_t load_or_zero(const T *in, uint64_t i, uint64_t n)
{
    return i < n ? (uint64_t)in[i] : 0ull;
}

// Block-wide exclusive scan of one value per thread; returns the exclusive prefix, *total = block sum.
__device__ __forceinline__ uint64_t block_excl_scan(uint64_t v, uint64_t *total)
{
    __shared__ uint64_t warp_sums[SCAN_THREADS / 32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    uint64_t x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        uint64_t y = __shfl_up_sync(0xFFFFFFFFu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) warp_sums[wid] = x;
    __syncthreads();
    if (wid == 0) {
        uint64_t w = lane < SCAN_THREADS / 32 ? warp_sums[lane] : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            uint64_t y = __shfl_up_sync(0xFFFFFFFFu, w, o);
            if (lane >= o) w += y;
        }
        if (lane < SCAN_THREADS / 32) warp_sums[lane] = w;
    }
    __syncthreads();
    uint64_t before = wid ? warp_sums[wid - 1] : 0;
    *total = warp_sums[SCAN_THREADS / 32 - 1];
    __syncthreads();
    return before + x - v;
}

template <typename T>
__global__ void __launch_bounds__(SCAN_THREADS) k_tile_sums(const T *in, uint64_t n, uint64_t *sums)
{
    const uint64_t base = (uint64_t)blockIdx.x * SCAN_TILE;
    uint64_t s = 0;
#pragma unroll
    for (int j = 0; j < SCAN_ITEMS; j++) s += load_or_zero(in, base + (uint64_t)j * SCAN_THREADS + threadIdx.x, n);
    uint64_t tot;
    block_excl_scan(s, &tot);
    if (threadIdx.x == 0) sums[blockIdx.x] = tot;
}

template <typename T>
__global__ void __launch_bounds__(SCAN_THREADS) k_tile_scan(const T *in, uint64_t *out, uint64_t n,
                                                            const uint64_t *offsets, uint64_t *total)
{
    __shared__ uint64_t tile[SCAN_TILE];
    const uint64_t base = (uint64_t)blockIdx.x * SCAN_TILE;
#pragma unroll
    for (int j = 0; j < SCAN_ITEMS; j++) {
        int idx = j * SCAN_THREADS + threadIdx.x;
        tile[idx] = load_or_zero(in, base + idx, n);
    }
    __syncthreads();
    uint64_t v[SCAN_ITEMS], s = 0;
#pragma unroll
    for (int j = 0; j < SCAN_ITEMS; j++) { v[j] = tile[threadIdx.x * SCAN_ITEMS + j]; s += v[j]; }
    uint64_t tot;
    uint64_t run = block_excl_scan(s, &tot) + (offsets ? offsets[blockIdx.x] : 0ull);
#pragma unroll
    for (int j = 0; j < SCAN_ITEMS; j++) { tile[threadIdx.x * SCAN_ITEMS + j] = run; run += v[j]; }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < SCAN_ITEMS; j++) {
        int idx = j * SCAN_THREADS + threadIdx.x;
        if (base + idx < n) out[base + idx] = tile[idx];
    }
    if (total && blockIdx.x == gridDim.x - 1 && threadIdx.x == SCAN_THREADS - 1) *total = run;
}

size_t scan_tmp_bytes(uint64_t n)
{
    size_t b = 0;
    while (n > (uint64_t)SCAN_TILE) {
        n = (n + SCAN_TILE - 1) / SCAN_TILE;
        b += n * sizeof(uint64_t) + 256;
    }
    return b + 256;
}

template <typename T>
static void scan_impl(const T *in, uint64_t *out, uint64_t n, uint64_t *total_dev, void *tmp, size_t tmp_bytes,
                      cudaStream_t st)
{
    if (n == 0) {
        if (total_dev) cudaMemsetAsync(total_dev, 0, sizeof(uint64_t), st);
        return;
    }
    uint64_t tiles = (n + SCAN_TILE - 1) / SCAN_TILE;
    if (tiles == 1) {
        (mp::count_launch(), k_tile_scan<T><<<1, SCAN_THREADS, 0, st>>>(in, out, n, nullptr, total_dev));
        return;
    }
    uint64_t *sums = (uint64_t *)tmp;
    size_t used = (tiles * sizeof(uint64_t) + 255) & ~(size_t)255;
    (mp::count_launch(), k_tile_sums<T><<<(unsigned)tiles, SCAN_THREADS, 0, st>>>(in, n, sums));
    scan_impl<uint64_t>(sums, sums, tiles, nullptr, (char *)tmp + used, tmp_bytes - used, st);
    (mp::count_launch(), k_tile_scan<T><<<(unsigned)tiles, SCAN_THREADS, 0, st>>>(in, out, n, sums, total_dev));
}

void scan_u32_to_u64(const uint32_t *in, uint64_t *out, uint64_t n, uint64_t *total_dev, void *tmp,
                     size_t tmp_bytes, cudaStream_t st)
{
    scan_impl<uint32_t>(in, out, n, total_dev, tmp, tmp_bytes, st);
}
void scan_u64(const uint64_t *in, uint64_t *out, uint64_t n, uint64_t *total_dev, void *tmp, size_t tmp_bytes,
              cudaStream_t st)
{
    scan_impl<uint64_t>(in, out, n, total_dev, tmp, tmp_bytes, st);
}

// ---------------------------------------------------------------- newlines

constexpr int NL_THREADS = 256;
constexpr uint64_t NL_SEG = 65536;  // bytes per block; a multiple of 16 * NL_THREADS

__device__ __forceinline__ uint32_t nl_in_word(uint32_t w)
{
    // 0x80 in exactly the bytes equal to '\n' (0x0A): exact zero-byte test of w ^ 0x0A0A0A0A
    // (no carry crosses a byte: (x & 0x7F) + 0x7F <= 0xFE)
    const uint32_t x = w ^ 0x0A0A0A0Au;
    const uint32_t y = (x & 0x7F7F7F7Fu) + 0x7F7F7F7Fu;
    return ~(y | x | 0x7F7F7F7Fu);
}

// Bit q: byte q of the sixteen at p is a newline of the parsed range.
__device__ __forceinline__ uint32_t nl_mask16(const uint8_t *buf, uint64_t p, uint64_t end, uint32_t skip)
{
    if (p + 16 <= end && p >= skip) {
        const uint4 v = *reinterpret_cast<const uint4 *>(buf + p);
        const uint32_t w[4] = {v.x, v.y, v.z, v.w};
        uint32_t m = 0;
#pragma unroll
        for (int q = 0; q < 4; q++) m |= ((((nl_in_word(w[q]) >> 7) * 0x01020408u) >> 24) & 0xFu) << (4 * q);
        return m;
    }
    uint32_t m = 0;
    for (uint32_t q = 0; q < 16; q++)
        if (p + q < end && p + q >= skip && buf[p + q] == '\n') m |= 1u << q;
    return m;
}

// buf is 16-byte aligned; its first `skip` (< 16) bytes are not part of the parsed range, whose byte 0 is
// buf[skip] (newline positions are written relative to it).  mask (nullable): a bit per byte of the blocks, for k_nl_place.
__global__ void __launch_bounds__(NL_THREADS) k_nl_count(const uint8_t *buf, uint64_t n, uint32_t skip, uint32_t *seg_counts,
                                                         uint16_t *mask)
{
    const uint64_t s0 = (uint64_t)blockIdx.x * NL_SEG, s1 = min(n, s0 + NL_SEG);
    uint32_t c = 0;
#pragma unroll 4
    for (uint64_t p = s0 + (uint64_t)threadIdx.x * 16; p < s0 + NL_SEG; p += NL_THREADS * 16) {
        const uint32_t m = p < s1 ? nl_mask16(buf, p, s1, skip) : 0u;
        if (mask) mask[p >> 4] = (uint16_t)m;
        c += (uint32_t)__popc(m);
    }
    uint64_t tot;
    uint64_t x = c;
    for (int o = 16; o; o >>= 1) x += __shfl_xor_sync(0xFFFFFFFFu, x, o);
    __shared__ uint64_t ws[NL_THREADS / 32];
    if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = x;
    __syncthreads();
    if (threadIdx.x == 0) {
        tot = 0;
        for (int w = 0; w < NL_THREADS / 32; w++) tot += ws[w];
        seg_counts[blockIdx.x] = (uint32_t)tot;
    }
}

// A warp takes an eighth of the block's bytes and keeps its newlines as bits, so the block meets once, for the warps' counts.
// Bound by its instructions, about 60 per 16 bytes (220 with every byte compared and a block scan every 4 KB): 6.2 GB
// 2.73 -> 2.30 ms.
__global__ void __launch_bounds__(NL_THREADS) k_nl_write(const uint8_t *buf, uint64_t n, uint32_t skip,
                                                         const uint64_t *seg_off, uint64_t *nl_pos, unsigned long long *stat)
{
    if (blockIdx.x == 0 && threadIdx.x == 0) {  // k_records' results
        stat[0] = ~0ull;
        stat[1] = 0;
    }
    constexpr int WARPS = NL_THREADS / 32, TURNS = (int)(NL_SEG / (NL_THREADS * 16));
    __shared__ uint32_t ws[WARPS];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint64_t end = min(n, ((uint64_t)blockIdx.x + 1) * NL_SEG);
    const uint64_t p0 = (uint64_t)blockIdx.x * NL_SEG + (uint64_t)warp * (NL_SEG / WARPS) + (uint64_t)lane * 16;
    uint32_t m[TURNS], c = 0;
#pragma unroll
    for (int i = 0; i < TURNS; i++) {
        const uint64_t p = p0 + (uint64_t)i * 512;
        m[i] = p < end ? nl_mask16(buf, p, end, skip) : 0u;
        c += (uint32_t)__popc(m[i]);
    }
    c = __reduce_add_sync(0xFFFFFFFFu, c);
    if (lane == 0) ws[warp] = c;
    __syncthreads();
    uint64_t out = seg_off[blockIdx.x];
    for (int w = 0; w < warp; w++) out += ws[w];
#pragma unroll
    for (int i = 0; i < TURNS; i++) {
        const uint32_t cnt = (uint32_t)__popc(m[i]);
        uint32_t x = cnt;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, o);
            if (lane >= o) x += y;
        }
        uint64_t o = out + x - cnt;
        for (uint32_t b = m[i]; b; b &= b - 1) nl_pos[o++] = p0 + (uint64_t)i * 512 + (uint32_t)(__ffs((int)b) - 1) - skip;
        out += __shfl_sync(0xFFFFFFFFu, x, 31);
    }
}

// The same from the count's bits: a lane takes 256 bytes, so a warp's counts meet once.  6.2 GB: 0.33 ms where the bytes read
// again took 2.29, and the bits cost the count 0.36.
__global__ void __launch_bounds__(NL_THREADS) k_nl_place(const uint16_t *mask, uint32_t skip, const uint64_t *seg_off, uint64_t *nl_pos,
                                                         unsigned long long *stat)
{
    if (blockIdx.x == 0 && threadIdx.x == 0) {  // k_records' results
        stat[0] = ~0ull;
        stat[1] = 0;
    }
    static_assert(NL_SEG == (uint64_t)NL_THREADS * 256, "256 bytes per thread");
    __shared__ uint32_t ws[NL_THREADS / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint64_t p0 = (uint64_t)blockIdx.x * NL_SEG + (uint64_t)threadIdx.x * 256;
    const ulonglong2 *mp = reinterpret_cast<const ulonglong2 *>(mask + (p0 >> 4));
    const ulonglong2 a = mp[0], b = mp[1];
    const unsigned long long w[4] = {a.x, a.y, b.x, b.y};
    const uint32_t c = (uint32_t)(__popcll(w[0]) + __popcll(w[1]) + __popcll(w[2]) + __popcll(w[3]));
    uint32_t x = c;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) ws[warp] = x;
    __syncthreads();
    uint64_t o = seg_off[blockIdx.x] + x - c;
    for (int v = 0; v < warp; v++) o += ws[v];
#pragma unroll
    for (int q = 0; q < 4; q++)
        for (unsigned long long m = w[q]; m; m &= m - 1) nl_pos[o++] = p0 + (uint32_t)(64 * q + __ffsll((long long)m) - 1) - skip;
}

// Record table from the newline positions; flags quality/sequence length mismatches.
// stat: [0] first record with a mismatch, [1] the longest sequence (both set before), [2] the end of the last record.
__global__ void k_records(const uint64_t *nl, uint64_t n_rec, uint64_t *rec_start, uint64_t *seq_off, uint32_t *seq_len,
                          unsigned long long *stat)
{
    uint64_t r = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t here = r < n_rec ? (uint32_t)min(nl[4 * r + 1] - nl[4 * r] - 1, (uint64_t)0xFFFFFFFFull) : 0u;
    const uint32_t most = __reduce_max_sync(0xFFFFFFFFu, here);
    if ((threadIdx.x & 31) == 0 && most > (uint32_t)*(volatile unsigned long long *)&stat[1])
        atomicMax(&stat[1], (unsigned long long)most);
    if (r >= n_rec) return;
    uint64_t s = r ? nl[4 * r - 1] + 1 : 0;
    uint64_t sq = nl[4 * r] + 1;
    uint64_t sl = nl[4 * r + 1] - sq;
    uint64_t q = nl[4 * r + 2] + 1;
    uint64_t ql = nl[4 * r + 3] - q;
    rec_start[r] = s;
    seq_off[r] = sq;
    seq_len[r] = (uint32_t)sl;
    if (ql != sl || sl > 0xFFFFFFFFull) atomicMin(&stat[0], (unsigned long long)r);
    if (r == n_rec - 1) stat[2] = rec_start[n_rec] = nl[4 * r + 3] + 1;
}

// For each query offset: the record whose start equals it, or ~0 when no record starts there.
__global__ void k_record_of_offset(const uint64_t *rec_start, uint64_t n_rec, const uint64_t *queries, int nq,
                                   uint64_t *out)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nq) return;
    uint64_t x = queries[i], lo = 0, hi = n_rec + 1;  // search rec_start[0..n_rec]
    while (lo < hi) {
        uint64_t mid = (lo + hi) / 2;
        if (rec_start[mid] < x) lo = mid + 1; else hi = mid;
    }
    out[i] = (lo <= n_rec && rec_start[lo] == x) ? lo : ~0ull;
}

int parse_fastq(const uint8_t *d_buf, uint64_t n, ParsedReads *pr, DeviceArena &arena, cudaStream_t st)
{
    return parse_fastq_range(d_buf, 0, n, pr, arena, st);
}

int parse_fastq_range(const uint8_t *d_base, uint64_t begin, uint64_t end, ParsedReads *pr, DeviceArena &arena,
                      cudaStream_t st)
{
    const uint64_t n = end - begin;
    if (n == 0 || end < begin) return set_error(MP_EFMT, "empty FASTQ input");
    // the kernels read 16-byte words from the 16-byte boundary at or below begin and skip the bytes before it
    const uint64_t a0 = begin & ~15ull;
    const uint32_t skip = (uint32_t)(begin - a0);
    const uint8_t *d_buf = d_base + a0;
    const uint64_t na = end - a0;
    const uint64_t segs = (na + NL_SEG - 1) / NL_SEG;
    uint32_t *seg_counts = arena.alloc<uint32_t>(segs);
    uint64_t *seg_off = arena.alloc<uint64_t>(segs + 1);
    uint64_t *total = arena.alloc<uint64_t>(1);
    size_t tb = scan_tmp_bytes(segs);
    void *tmp = arena.alloc<uint8_t>(tb);
    if (!seg_counts || !seg_off || !total || !tmp) return set_error(MP_ENOMEM, "device memory for the FASTQ parse");
    // the newlines as bits, where there is room for them beside what has to be held
    uint16_t *mask = arena.alloc<uint16_t>(segs * (NL_SEG / 16));
    auto without_mask = [&] {
        const bool had = mask != nullptr;
        if (had) arena.free_scratch(mask);
        mask = nullptr;
        return had;
    };
    (mp::count_launch(), k_nl_count<<<(unsigned)segs, NL_THREADS, 0, st>>>(d_buf, na, skip, seg_counts, mask));
    scan_u32_to_u64(seg_counts, seg_off, segs, total, tmp, tb, st);
    ReadBack<uint64_t> rb(arena, 4);
    MP_CUDA(cudaMemcpyAsync(&rb[0], total, sizeof(uint64_t), cudaMemcpyDeviceToHost, st));
    MP_CUDA(cudaStreamSynchronize(st));
    const uint64_t n_nl = rb[0];
    if (n_nl == 0 || n_nl % 4) return set_error(MP_EFMT, "FASTQ line count %llu is not a multiple of 4", (unsigned long long)n_nl);
    uint64_t *nl = arena.alloc<uint64_t>(n_nl);
    if (!nl && without_mask()) nl = arena.alloc<uint64_t>(n_nl);
    if (!nl) return set_error(MP_ENOMEM, "device memory for newline positions");
    const uint64_t n_rec = n_nl / 4;
    pr->n_reads = n_rec;
    pr->rec_start = arena.alloc_persistent<uint64_t>(n_rec + 1);
    pr->seq_off = arena.alloc_persistent<uint64_t>(n_rec);
    pr->seq_len = arena.alloc_persistent<uint32_t>(n_rec);
    if (!(pr->rec_start && pr->seq_off && pr->seq_len) && without_mask()) {
        if (!pr->rec_start) pr->rec_start = arena.alloc_persistent<uint64_t>(n_rec + 1);
        if (!pr->seq_off) pr->seq_off = arena.alloc_persistent<uint64_t>(n_rec);
        if (!pr->seq_len) pr->seq_len = arena.alloc_persistent<uint32_t>(n_rec);
    }
    unsigned long long *bad = arena.alloc<unsigned long long>(3);
    if (!bad && without_mask()) bad = arena.alloc<unsigned long long>(3);
    if (!pr->rec_start || !pr->seq_off || !pr->seq_len || !bad) return set_error(MP_ENOMEM, "device memory for the record table");
    if (mask) (mp::count_launch(), k_nl_place<<<(unsigned)segs, NL_THREADS, 0, st>>>(mask, skip, seg_off, nl, bad));
    else (mp::count_launch(), k_nl_write<<<(unsigned)segs, NL_THREADS, 0, st>>>(d_buf, na, skip, seg_off, nl, bad));
    (mp::count_launch(), k_records<<<(unsigned)((n_rec + 255) / 256), 256, 0, st>>>(nl, n_rec, pr->rec_start, pr->seq_off, pr->seq_len, bad));
    MP_CUDA(cudaMemcpyAsync(&rb[1], bad, 3 * sizeof(uint64_t), cudaMemcpyDeviceToHost, st));
    MP_CUDA(cudaStreamSynchronize(st));
    const uint64_t hb[2] = {rb[1], rb[2]}, last_end = rb[3];
    MP_CUDA(cudaGetLastError());
    if (hb[0] != ~0ull) return set_error(MP_EFMT, "FASTQ record %llu: quality length differs from the sequence length",
                                          (unsigned long long)hb[0]);
    pr->max_len = (uint32_t)hb[1];
    if (last_end != n) return set_error(MP_EFMT, "FASTQ input does not end with a complete record");
    arena.release_scratch();
    return 0;
}

// Record table of one input segment (offsets relative to the segment) into the job's table at read r0,
// offsets moved by the segment's byte offset; n + 1 start entries (the last is the next segment's first).
__global__ void k_concat_records(const uint64_t *rs, const uint64_t *so, const uint32_t *sl, uint64_t n, uint64_t base,
                                 uint64_t *drs, uint64_t *dso, uint32_t *dsl)
{
    const uint64_t r = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (r > n) return;
    drs[r] = rs[r] + base;
    if (r < n) {
        dso[r] = so[r] + base;
        dsl[r] = sl[r];
    }
}

void concat_records(const ParsedReads &seg, uint64_t byte_base, ParsedReads &dst, uint64_t r0, cudaStream_t st)
{
    (mp::count_launch(), k_concat_records<<<(unsigned)((seg.n_reads + 1 + 255) / 256), 256, 0, st>>>(
        seg.rec_start, seg.seq_off, seg.seq_len, seg.n_reads, byte_base, dst.rec_start + r0, dst.seq_off + r0,
        dst.seq_len + r0));
}

int records_at_offsets(const ParsedReads *pr, const uint64_t *h_offsets, int nq, uint64_t *h_rec, DeviceArena &arena,
                       cudaStream_t st)
{
    uint64_t *dq = arena.alloc<uint64_t>(nq), *dr = arena.alloc<uint64_t>(nq);
    if (!dq || !dr) return set_error(MP_ENOMEM, "device memory");
    MP_CUDA(cudaMemcpyAsync(dq, h_offsets, nq * sizeof(uint64_t), cudaMemcpyHostToDevice, st));
    (mp::count_launch(), k_record_of_offset<<<(nq + 127) / 128, 128, 0, st>>>(pr->rec_start, pr->n_reads, dq, nq, dr));
    ReadBack<uint64_t> rb(arena, nq);
    MP_CUDA(cudaMemcpyAsync(rb.p, dr, nq * sizeof(uint64_t), cudaMemcpyDeviceToHost, st));
    MP_CUDA(cudaStreamSynchronize(st));
    std::copy(rb.p, rb.p + nq, h_rec);
    arena.release_scratch();
    for (int i = 0; i < nq; i++)
        if (h_rec[i] == ~0ull)
            return set_error(MP_EFMT, "offset %llu is not the start of a FASTQ record", (unsigned long long)h_offsets[i]);
    return 0;
}

}  // namespace mp
