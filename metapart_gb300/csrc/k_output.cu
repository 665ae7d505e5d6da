// K7: partition FASTQ output (writeOutput3, metapart.c:956-1066).
//
// Output file j = partition * T + tid holds, in input order, every record whose
// component root falls in the partition's read-id range, written by thread tid (the
// thread owning the record's chunk).  An interleaved pair is written to the partition of
// mate 1's root and, when mate 2's root differs, again to mate 2's (:1006-1047).  On the
// GPU the entries take their places by one stable partition into the 16 parts (OutBlock), and a warp
// copies each record.
#include <algorithm>

#include "k_output.cuh"

namespace mp {

__device__ __forceinline__ uint32_t part_of(const uint64_t *bounds, uint32_t root)
{
    uint32_t p = 0;
    while (p < 16 && !((uint64_t)root < bounds[p + 1])) p++;
    return p;
}

struct OutCtx {
    const uint64_t *rec_start;
    int interleaved;
};

// The plan's input: samples one after another in the reads (one for a job); sample q's files are the global files
// file0[q] + part * T[q] + tid, its blocks (of OP_UNITS units, a unit being a read or an interleaved pair) blk0[q] on.
struct OutPlanCtx {
    const uint64_t *rec_start;
    const uint32_t *label;
    const uint64_t *srec;       // nseg + 1 read offsets
    const uint64_t *bounds;     // nseg x 17, each sample's own read ids
    const uint64_t *chunk_rec;  // every sample's nchunks + 1 chunk record starts (its own read ids), one after another
    const uint32_t *chunk0;     // nseg + 1: where each sample's chunk records start in chunk_rec
    const uint32_t *T, *per_thread, *file0, *blk0;  // per sample (blk0: nseg + 1)
    int nseg, interleaved;
};

constexpr int OP_THREADS = 256, OP_ROUNDS = 4, OP_UNITS = OP_THREADS * OP_ROUNDS;

// The file order is part, then thread, then input order, and a record's thread never falls as the records go on (threads
// own consecutive chunks): the entries of a file are the part's entries in input order, cut at the threads' first
// records.  So the layout is one stable partition into 16 parts: the blocks' entries and bytes per part, scanned in (part,
// block) order, and then every entry's place.  (Sorted by file with the radix sort: 10 launches and a host wait more.)
struct OutBlock {
    uint64_t len[OP_ROUNDS];             // bytes of this lane's unit of every round
    uint32_t p0[OP_ROUNDS], p1[OP_ROUNDS];  // its parts: one (p1 = 16) or, mates in two components, two
    uint32_t seg, blk, nblk;             // the block's sample, its number in the sample and the sample's blocks
    uint64_t u0;                         // lane's first unit (round r: u0 + 32 r) in all reads' units
};

__device__ __forceinline__ uint32_t tid_of(const OutPlanCtx &c, uint32_t q, uint64_t lr)
{
    const uint64_t *cr = c.chunk_rec + c.chunk0[q];
    int lo = 0, hi = (int)(c.chunk0[q + 1] - c.chunk0[q]) - 2;  // the sample's chunk holding lr
    while (lo < hi) {
        const int m = (lo + hi + 1) >> 1;
        if (cr[m] <= lr) lo = m; else hi = m - 1;
    }
    return (uint32_t)lo / c.per_thread[q];
}

__device__ __forceinline__ void out_block(const OutPlanCtx &c, OutBlock &o)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int lo = 0, hi = c.nseg - 1;  // the last sample whose blocks start at or below this one
    while (lo < hi) {
        const int m = (lo + hi + 1) >> 1;
        if (c.blk0[m] <= blockIdx.x) lo = m; else hi = m - 1;
    }
    o.seg = (uint32_t)lo;
    o.blk = blockIdx.x - c.blk0[lo];
    o.nblk = c.blk0[lo + 1] - c.blk0[lo];
    const int il = c.interleaved ? 1 : 0;
    const uint64_t R = c.srec[lo], units = (c.srec[lo + 1] - R) >> il, first = (uint64_t)o.blk * OP_UNITS + warp * (32 * OP_ROUNDS) + lane;
    const uint64_t *b = c.bounds + (uint64_t)lo * 17;
    o.u0 = (R >> il) + first;
#pragma unroll
    for (int r = 0; r < OP_ROUNDS; r++) {
        o.len[r] = 0;
        o.p0[r] = o.p1[r] = 16;
        if (first + 32 * r >= units) continue;
        const uint64_t u = R + ((first + 32 * r) << il);
        o.len[r] = c.rec_start[u + 1 + il] - c.rec_start[u];
        const uint32_t pu = c.label[u];
        o.p0[r] = part_of(b, (uint32_t)(pu - R));
        if (il) {
            const uint32_t pv = c.label[u + 1];
            if (pu != pv) o.p1[r] = part_of(b, (uint32_t)(pv - R));
        }
    }
}

// Sums over the lanes up to and including this one.
__device__ __forceinline__ uint64_t lanes_scan(uint64_t x, bool small)
{
    const int lane = threadIdx.x & 31;
    if (small) {
        uint32_t v = (uint32_t)x;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, v, o);
            if (lane >= o) v += y;
        }
        return v;
    }
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint64_t y = __shfl_up_sync(0xFFFFFFFFu, x, o);
        if (lane >= o) x += y;
    }
    return x;
}

// Walks a warp's units part by part: f(round, part, lane's entries, entries before the lane, bytes before it, the warp's
// entries and bytes) with the counts of one round.
template <class F> __device__ __forceinline__ void out_walk(const OutBlock &o, F f)
{
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int r = 0; r < OP_ROUNDS; r++) {
        const bool small = !__any_sync(0xFFFFFFFFu, o.len[r] >= (1ull << 25));
        const bool two = __any_sync(0xFFFFFFFFu, o.p1[r] < 16);
        uint32_t left = __reduce_or_sync(0xFFFFFFFFu, (1u << o.p0[r]) | (1u << o.p1[r])) & 0xFFFFu;
        while (left) {
            const uint32_t p = __ffs(left) - 1;
            left &= left - 1;
            const uint32_t n = (o.p0[r] == p ? 1u : 0u) + (o.p1[r] == p ? 1u : 0u);
            const uint64_t b = lanes_scan(n * o.len[r], small);
            uint32_t e;
            if (two) {
                e = (uint32_t)lanes_scan(n, true);
            } else {
                e = (uint32_t)__popc(__ballot_sync(0xFFFFFFFFu, n) & ((2u << lane) - 1));
            }
            f(r, p, n, e - n, b - n * o.len[r], __shfl_sync(0xFFFFFFFFu, e, 31), __shfl_sync(0xFFFFFFFFu, b, 31));
        }
    }
}

// Entries and bytes of every (part, block), and the files' sizes.
__global__ void __launch_bounds__(OP_THREADS) k_out_count(OutPlanCtx c, uint32_t *cnt, uint64_t *bytes, unsigned long long *file_bytes)
{
    __shared__ uint32_t se[OP_THREADS / 32][16];
    __shared__ uint64_t sb[OP_THREADS / 32][16];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int i = threadIdx.x; i < (OP_THREADS / 32) * 16; i += OP_THREADS) {
        (&se[0][0])[i] = 0;
        (&sb[0][0])[i] = 0;
    }
    __syncthreads();
    OutBlock o;
    out_block(c, o);
    const uint64_t units = (c.srec[o.seg + 1] - c.srec[o.seg]) >> (c.interleaved ? 1 : 0), b0 = (uint64_t)o.blk * OP_UNITS;
    const uint32_t T = c.T[o.seg];
    const uint32_t ta = tid_of(c, o.seg, b0 << c.interleaved), tz = tid_of(c, o.seg, (min(units, b0 + OP_UNITS) - 1) << c.interleaved);
    out_walk(o, [&](int, uint32_t p, uint32_t, uint32_t, uint64_t, uint32_t e, uint64_t b) {
        if (lane == 0) {
            se[warp][p] += e;
            sb[warp][p] += b;
        }
    });
    if (ta != tz) {  // a thread's first record lies in the block: its files' bytes unit by unit
#pragma unroll
        for (int r = 0; r < OP_ROUNDS; r++) {
            if (o.p0[r] == 16) continue;
            const uint32_t f = c.file0[o.seg] + tid_of(c, o.seg, (o.u0 + 32 * r - (c.srec[o.seg] >> c.interleaved)) << c.interleaved);
            atomicAdd(&file_bytes[f + o.p0[r] * T], (unsigned long long)o.len[r]);
            if (o.p1[r] < 16) atomicAdd(&file_bytes[f + o.p1[r] * T], (unsigned long long)o.len[r]);
        }
    }
    __syncthreads();
    if (threadIdx.x < 16) {
        const uint32_t p = threadIdx.x;
        uint32_t e = 0;
        uint64_t b = 0;
        for (int w = 0; w < OP_THREADS / 32; w++) {
            e += se[w][p];
            b += sb[w][p];
        }
        const size_t cell = 16 * (size_t)c.blk0[o.seg] + (size_t)p * o.nblk + o.blk;
        cnt[cell] = e;
        bytes[cell] = b;
        if (ta == tz && b) atomicAdd(&file_bytes[c.file0[o.seg] + p * T + ta], (unsigned long long)b);
    }
}

// Every entry's unit and byte offset at its place.
__global__ void __launch_bounds__(OP_THREADS) k_out_place(OutPlanCtx c, const uint64_t *cell_e, const uint64_t *cell_b, uint32_t *val,
                                                          uint64_t *off)
{
    __shared__ uint32_t se[OP_THREADS / 32][16];
    __shared__ uint64_t sb[OP_THREADS / 32][16], be[16];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int i = threadIdx.x; i < (OP_THREADS / 32) * 16; i += OP_THREADS) {
        (&se[0][0])[i] = 0;
        (&sb[0][0])[i] = 0;
    }
    __syncthreads();
    OutBlock o;
    out_block(c, o);
    out_walk(o, [&](int, uint32_t p, uint32_t, uint32_t, uint64_t, uint32_t e, uint64_t b) {
        if (lane == 0) {
            se[warp][p] += e;
            sb[warp][p] += b;
        }
    });
    __syncthreads();
    if (threadIdx.x < 16) {  // the warps' first places
        const uint32_t p = threadIdx.x;
        const size_t cell = 16 * (size_t)c.blk0[o.seg] + (size_t)p * o.nblk + o.blk;
        uint32_t e = 0;
        uint64_t b = cell_b[cell];
        be[p] = cell_e[cell];
        for (int w = 0; w < OP_THREADS / 32; w++) {
            const uint32_t x = se[w][p];
            const uint64_t y = sb[w][p];
            se[w][p] = e;
            sb[w][p] = b;
            e += x;
            b += y;
        }
    }
    __syncthreads();
    out_walk(o, [&](int r, uint32_t p, uint32_t n, uint32_t e, uint64_t b, uint32_t we, uint64_t wb) {
        const uint64_t ew = be[p] + se[warp][p], bw = sb[warp][p];
        for (uint32_t q = 0; q < n; q++) {
            val[ew + e + q] = (uint32_t)(o.u0 + 32 * r);
            off[ew + e + q] = bw + b + q * o.len[r];
        }
        __syncwarp();
        if (lane == 0) {
            se[warp][p] += we;
            sb[warp][p] += wb;
        }
        __syncwarp();
    });
}

// One record (l bytes at src) to dst by a warp, lanes 16 bytes each: an aligned 16-byte load, the bytes that follow from the
// next lane, a 16-byte store; the bytes before dst's first 16-byte boundary and after its last by lanes 0-15 and 16-31.
// load takes the record's first 512 bytes into registers, store writes them and copies what is left.
struct RecordCopy {
    const uint8_t *src;
    uint8_t *dst;
    uint32_t l, head, chunks;  // bytes before the boundary, 16-byte chunks
    uint4 v;

    __device__ __forceinline__ const uint4 *block(uint32_t j) const
    {
        return reinterpret_cast<const uint4 *>(reinterpret_cast<uintptr_t>(src + head + 16ull * j) & ~(uintptr_t)15);
    }
    __device__ __forceinline__ uint32_t end_at(int lane) const  // l: no byte
    {
        const uint32_t i = lane < 16 ? (uint32_t)lane : head + 16 * chunks + lane - 16;
        return lane < 16 && i >= head ? l : min(i, l);
    }
    __device__ __forceinline__ void load(const uint8_t *s, uint32_t len, uint8_t *d, int lane)
    {
        src = s;
        dst = d;
        l = len;
        head = min(l, (uint32_t)(-reinterpret_cast<uintptr_t>(d) & 15));
        chunks = (l - head) >> 4;
        // (at most 31 bytes past the record: the buffer carries 64 bytes of padding)
        if ((uint32_t)lane <= chunks) v = *block((uint32_t)lane);
    }
    __device__ __forceinline__ void store(int lane)
    {
        const uint32_t sh = (uint32_t)(reinterpret_cast<uintptr_t>(src + head) & 15), bs = (sh & 3) * 8;
        const uint32_t i = end_at(lane), end = i < l ? src[i] : 0u;  // (its line came with the chunks, or nearly)
        for (uint32_t c0 = 0; c0 < chunks; c0 += 32) {
            const uint32_t j = c0 + lane;
            if (c0 && j <= chunks) v = *block(j);
            uint4 n = make_uint4(__shfl_down_sync(0xFFFFFFFFu, v.x, 1), __shfl_down_sync(0xFFFFFFFFu, v.y, 1),
                                 __shfl_down_sync(0xFFFFFFFFu, v.z, 1), __shfl_down_sync(0xFFFFFFFFu, v.w, 1));
            if (lane == 31 && j < chunks) n = *block(j + 1);
            uint4 r;
            switch (sh >> 2) {  // the same in every lane
            case 0: r = shifted(v.x, v.y, v.z, v.w, n.x, bs); break;
            case 1: r = shifted(v.y, v.z, v.w, n.x, n.y, bs); break;
            case 2: r = shifted(v.z, v.w, n.x, n.y, n.z, bs); break;
            default: r = shifted(v.w, n.x, n.y, n.z, n.w, bs); break;
            }
            if (j < chunks) *reinterpret_cast<uint4 *>(dst + head + 16ull * j) = r;
        }
        if (i < l) dst[i] = (uint8_t)end;
    }
    static __device__ __forceinline__ uint4 shifted(uint32_t a, uint32_t b, uint32_t c, uint32_t d, uint32_t e, uint32_t bs)
    {
        return make_uint4(__funnelshift_r(a, b, bs), __funnelshift_r(b, c, bs), __funnelshift_r(c, d, bs), __funnelshift_r(d, e, bs));
    }
};

// A warp copies OC_PER_WARP records: lanes fetch the records' source ranges and destinations in one round, then OC_FLY
// records at a time are loaded before the first is stored.  With 4-byte words, one record after another, the loads'
// latency bound it: 20M x 150 bp (6.2 GB) 4.5 -> 3.5 ms, 3M x 250 bp 0.98 -> 0.62 ms.
// 64 registers a thread: with 79 (three blocks an SM) 4.2 and 0.71 ms.
constexpr int OC_PER_WARP = 8, OC_FLY = 4;
static_assert(OC_PER_WARP % OC_FLY == 0, "whole turns");

__global__ void __launch_bounds__(256, 4) k_out_copy(OutCtx c, const uint8_t *__restrict__ fq, const uint32_t *val, const uint64_t *off, uint64_t n,
                           uint8_t *__restrict__ out)
{
    const uint64_t w0 = (((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5) * OC_PER_WARP;
    const int lane = threadIdx.x & 31;
    if (w0 >= n) return;
    uint64_t my_s = 0, my_l = 0, my_o = 0;  // lane q < OC_PER_WARP: record w0 + q
    if (lane < OC_PER_WARP && w0 + lane < n) {
        const uint64_t u = val[w0 + lane];
        const uint64_t r0 = c.interleaved ? 2 * u : u, r1 = c.interleaved ? 2 * u + 2 : u + 1;
        my_s = c.rec_start[r0];
        my_l = c.rec_start[r1] - my_s;
        my_o = off[w0 + lane];
    }
    const int nrec = (int)min((uint64_t)OC_PER_WARP, n - w0);
    for (int q = 0; q < nrec; q += OC_FLY) {
        RecordCopy r[OC_FLY];
#pragma unroll
        for (int x = 0; x < OC_FLY; x++) {  // (past the last record: no bytes)
            uint64_t s = __shfl_sync(0xFFFFFFFFu, my_s, q + x), l = __shfl_sync(0xFFFFFFFFu, my_l, q + x),
                     o = __shfl_sync(0xFFFFFFFFu, my_o, q + x);
            for (; l > 1ull << 30; s += 1ull << 30, o += 1ull << 30, l -= 1ull << 30) {
                r[x].load(fq + s, 1u << 30, out + o, lane);
                r[x].store(lane);
            }
            r[x].load(fq + s, (uint32_t)l, out + o, lane);
        }
#pragma unroll
        for (int x = 0; x < OC_FLY; x++) r[x].store(lane);
    }
}

int plan_output(const uint8_t *d_fq, const ParsedReads &pr, const uint32_t *d_label, const uint64_t *bounds_host,
                const uint64_t *chunk_rec_host, int nchunks, int T, int interleaved, OutputPlan *plan,
                std::vector<uint64_t> &file_sizes, DeviceArena &arena, cudaStream_t st)
{
    (void)d_fq;
    std::vector<uint64_t> file0;
    return plan_output_batch(pr, d_label, interleaved, {0, pr.n_reads}, std::vector<uint64_t>(bounds_host, bounds_host + 17),
                             {std::vector<uint64_t>(chunk_rec_host, chunk_rec_host + nchunks + 1)}, {T}, plan, file_sizes, file0,
                             arena, st);
}

int plan_output_batch(const ParsedReads &pr, const uint32_t *d_label, int interleaved, const std::vector<uint64_t> &seg_reads,
                      const std::vector<uint64_t> &bounds_host, const std::vector<std::vector<uint64_t>> &chunk_rec_host,
                      const std::vector<int> &T, OutputPlan *plan, std::vector<uint64_t> &file_sizes,
                      std::vector<uint64_t> &file0, DeviceArena &arena, cudaStream_t st)
{
    const int nseg = (int)seg_reads.size() - 1;
    // 64-bit words, then 32-bit ones, in one upload: read offsets, bounds, chunk records; chunk0, blk0, T, per_thread, file0
    std::vector<uint64_t> w(seg_reads.begin(), seg_reads.end());
    w.insert(w.end(), bounds_host.begin(), bounds_host.end());
    const size_t at_cr = w.size();
    std::vector<uint32_t> v(5 * (size_t)nseg + 2);
    uint32_t *c0 = v.data(), *blk0 = c0 + nseg + 1, *hT = blk0 + nseg + 1, *hpt = hT + nseg, *hf0 = hpt + nseg;
    file0.assign(nseg + 1, 0);
    uint64_t blocks = 0, ncr = 0;
    for (int q = 0; q < nseg; q++) {
        const int nch = (int)chunk_rec_host[q].size() - 1;
        if (nch < 1 || T[q] < 1 || nch % T[q]) return set_error(MP_EARG, "sample %d: numThreads must divide its chunks", q);
        c0[q] = (uint32_t)ncr;
        ncr += chunk_rec_host[q].size();
        w.insert(w.end(), chunk_rec_host[q].begin(), chunk_rec_host[q].end());
        blk0[q] = (uint32_t)blocks;
        blocks += ((seg_reads[q + 1] - seg_reads[q]) / (interleaved ? 2 : 1) + OP_UNITS - 1) / OP_UNITS;
        hT[q] = (uint32_t)T[q];
        hpt[q] = (uint32_t)(nch / T[q]);
        hf0[q] = (uint32_t)file0[q];
        file0[q + 1] = file0[q] + 16ull * (uint64_t)T[q];
    }
    c0[nseg] = (uint32_t)ncr;
    blk0[nseg] = (uint32_t)blocks;
    const uint64_t nf = file0[nseg], cells = 16 * blocks, units = seg_reads[nseg] / (interleaved ? 2 : 1);
    file_sizes.assign(nf, 0);
    const size_t n64 = w.size();
    w.resize(n64 + (v.size() + 1) / 2);
    std::copy(v.begin(), v.end(), reinterpret_cast<uint32_t *>(w.data() + n64));
    uint64_t *dw = arena.alloc<uint64_t>(w.size());
    uint32_t *cnt = arena.alloc<uint32_t>(cells + 1);
    uint64_t *bytes = arena.alloc<uint64_t>(cells + 1), *cell_e = arena.alloc<uint64_t>(cells + 1), *cell_b = arena.alloc<uint64_t>(cells + 1);
    unsigned long long *tail = arena.alloc<unsigned long long>(nf + 2);  // total entries and bytes, then the file sizes
    const size_t tb = scan_tmp_bytes(cells + 1);
    void *tmp = arena.alloc<uint8_t>(tb);
    const uint64_t most = units * (interleaved ? 2 : 1);  // entries at most
    plan->val = arena.alloc_persistent<uint32_t>(most + 1);
    plan->off = arena.alloc_persistent<uint64_t>(most + 1);
    if (!dw || !cnt || !bytes || !cell_e || !cell_b || !tail || !tmp || !plan->val || !plan->off)
        return set_error(MP_ENOMEM, "device memory for the output plan");
    MP_CUDA(cudaMemcpyAsync(dw, w.data(), w.size() * 8, cudaMemcpyHostToDevice, st));
    MP_CUDA(cudaMemsetAsync(tail, 0, (nf + 2) * sizeof(unsigned long long), st));
    OutPlanCtx c;
    c.rec_start = pr.rec_start;
    c.label = d_label;
    c.srec = dw;
    c.bounds = dw + nseg + 1;
    c.chunk_rec = dw + at_cr;
    c.chunk0 = reinterpret_cast<uint32_t *>(dw + n64);
    c.blk0 = c.chunk0 + nseg + 1;
    c.T = c.blk0 + nseg + 1;
    c.per_thread = c.T + nseg;
    c.file0 = c.per_thread + nseg;
    c.nseg = nseg;
    c.interleaved = interleaved ? 1 : 0;
    if (blocks) {
        (mp::count_launch(), k_out_count<<<(unsigned)blocks, OP_THREADS, 0, st>>>(c, cnt, bytes, tail + 2));
        scan_u32_to_u64(cnt, cell_e, cells, (uint64_t *)tail, tmp, tb, st);
        scan_u64(bytes, cell_b, cells, (uint64_t *)tail + 1, tmp, tb, st);
        (mp::count_launch(), k_out_place<<<(unsigned)blocks, OP_THREADS, 0, st>>>(c, cell_e, cell_b, plan->val, plan->off));
    }
    ReadBack<uint64_t> rb(arena, nf + 2);
    MP_CUDA(cudaMemcpyAsync(rb.p, tail, (nf + 2) * sizeof(uint64_t), cudaMemcpyDeviceToHost, st));
    MP_CUDA(cudaStreamSynchronize(st));
    MP_CUDA(cudaGetLastError());
    std::copy(rb.p + 2, rb.p + 2 + nf, file_sizes.begin());
    plan->n = rb[0];
    plan->total = rb[1];
    plan->rec_start = pr.rec_start;
    plan->interleaved = interleaved;
    return 0;
}

int copy_output_range(const OutputPlan &plan, uint64_t e0, uint64_t e1, const uint8_t *d_fq, uint8_t *dst,
                      cudaStream_t st)
{
    if (e1 <= e0) return 0;
    OutCtx c{};
    c.rec_start = plan.rec_start;
    c.interleaved = plan.interleaved;
    const uint64_t warps = (e1 - e0 + OC_PER_WARP - 1) / OC_PER_WARP;
    (mp::count_launch(), k_out_copy<<<(unsigned)((warps * 32 + 255) / 256), 256, 0, st>>>(
        c, d_fq, plan.val + e0, plan.off + e0, e1 - e0, dst));
    MP_CUDA(cudaGetLastError());
    return 0;
}

int copy_output(const OutputPlan &plan, const uint8_t *d_fq, uint8_t *dst, cudaStream_t st)
{
    return copy_output_range(plan, 0, plan.n, d_fq, dst, st);
}

}  // namespace mp
