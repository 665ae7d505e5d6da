#pragma once
#include <vector>

#include "k_graph.cuh"
#include "k_sort.cuh"

namespace mp {

// A scan without the order of its tuples: what the mischief filter and the unions need of the sorted scan is
// only which tuples share a k-mer, so the tuples are split into units of consecutive m-mer buckets (two
// unstable multi-split passes) and grouped by k-mer in shared-memory hash tables.  Results equal filter_scan +
// union_scan over the sorted scan: the same BAD marks, the same components.
//
// A tuple between the passes is K = (bucket - first bucket of its bin) << (2 (k - 10) + 6) | low k-mer bits << 6 |
// the six adjacency bits the filter reads, and the read id.

constexpr uint64_t GROUP_MAX_TUPLES = 4000000000ull;  // tuple positions are 32 bits
constexpr uint64_t GROUP_MAX_READS = 0x7FFFFFFFull;   // a grouped id keeps its top bit for the group's first tuple

// The first split pass of all scans of a job at once: the reads are packed and rolled through once.  Needs the tuples of
// every scan at once, so it is for the callers whose memory holds them, and the components of later scans are looked up in
// the second pass.  The scans' bins count from the first scan's first bucket, in the same widths; a bin that a scan's
// bounds cut is two.
// Up to three scans: a scan more is a comparison per k-mer and a digit above a thread's two in the reorder, and all scans'
// tuples are held at once (12 bytes each), while who asks for many scans asks for little memory.  4M x 150 bp, partition:
// 3 scans 16.0 ms (19.8 with a pass per scan), 4 scans 22.7.
constexpr int GROUP_MAX_MERGED = 3;
struct MergedScans {
    std::vector<uint32_t> scan;  // the scans' buckets, consecutive
    uint64_t n = 0;              // their tuples
    int sh = 0;                  // bins of 2^sh buckets
    uint32_t digits = 0;         // bins
    uint32_t *cur = nullptr;     // the bins' fill (digits words, the caller's), from the first scan's first tuple
    uint64_t *k1 = nullptr;      // the split tuples (n, the caller's)
    uint32_t *id1 = nullptr;
};

// One scan (or every sample's scan of a batch, as segments) to split and group.
struct GroupScan {
    int k = 0;
    uint64_t n = 0;                    // tuples
    const uint64_t *d_hist = nullptr;  // bucket prefix; the scan's buckets are [lo, hi), nseg * NB with segments
    uint64_t lo = 0, hi = 0;
    std::vector<uint64_t> bounds;      // thread ranges' tuple bounds, every segment's after the other (ascending)
    std::vector<uint64_t> seg_tstart;  // nseg + 1 tuple offsets ({0, n} for one scan)

    // a bucket-range piece of a scan: whether a thread range ends with its last tuple, whether it holds the scan's last tuple, and
    // its first tuple of the scan's last range with tuples (~0: none)
    bool part = false, ends_range = true, ends_scan = true;
    uint32_t last_range = 0;
    // after group_union, of a scan or piece: the last range's reads that are not BAD, outside and inside the scan's last run
    bool outside = false, inside = false;
    uint32_t anchor_read = 0;

    // a scan of merged ones (group_take)
    const MergedScans *merged = nullptr;
    uint64_t anchor = 0;                     // where its bins count from
    uint32_t digit0 = 0, tuple0 = 0;         // its first bin's digit and its first tuple among the merged
    const uint32_t *late_label = nullptr;    // the reads' components, for the second pass

    // the plan (device), from group_plan
    uint32_t bins = 0, seg_lo = 0, max_units = 0, max_tiles = 0;
    uint32_t *ustart = nullptr, *ub0 = nullptr, *ucur = nullptr;  // units: first tuple, first bucket | range start << 31, fill
    uint32_t *bstart = nullptr, *bu0 = nullptr, *bcur = nullptr, *bin_sh = nullptr, *bfirst = nullptr;  // bins: first tuple, unit;
                                                                                  // fill; width; first bucket
    uint32_t *unit_of = nullptr;  // every bucket's unit
    uint32_t *seg_bin0 = nullptr, *seg_sh = nullptr;
    uint4 *tiles = nullptr;       // of the second pass
    uint32_t *mid = nullptr, *big = nullptr;  // units above a small block's and above a large block's capacity
    uint32_t *lrs = nullptr;                  // per segment: first tuple of its last range with tuples
    uint32_t *ctr = nullptr;                  // GC_* counters
    uint32_t *qlist = nullptr;                // grouped stretches of the segments' last ranges
    uint32_t *quirk = nullptr;                // per segment: QW words (see k_gp_quirk)
    uint32_t hctr[16] = {};                   // the plan's counters on the host, from group_counts on
    std::vector<uint32_t> h_ctr;              // (where they arrive without a mailbox)
    cudaEvent_t planned = nullptr;            // after the counters' copy
    GroupScan() = default;
    GroupScan(const GroupScan &) = delete;
    GroupScan &operator=(const GroupScan &) = delete;
    ~GroupScan() { if (planned) cudaEventDestroy(planned); }
    std::vector<uint32_t> h_plan, h_tiles;     // sources of uploads still queued
};

enum GroupCounter : int {
    GC_UNITS = 0, GC_TILES, GC_MID, GC_BIG, GC_BIG_TUPLES,  // the plan's counts
    GC_WORK_S, GC_WORK_L, GC_OUT, GC_QLIST, GC_ERR, GC_LONG, GC_N = 16
};

// What a scan's unions left open, per segment: the segment's last run is to be united with the segment's first
// read (the sweeps' initial state, metapart.c:2539-2548); anchor is a read of that run.
struct GroupQuirk {
    int seg;
    uint32_t anchor;
};

bool group_fits(uint64_t n, uint64_t n_reads, const SortSegments *segs);
// Plans g (its inputs set) on the device; its counts are on their way to the host (group_filter takes them).
int group_plan(GroupScan &g, DeviceArena &arena, cudaStream_t st);
// First split pass, into bins, of n tuples to (k1, id1): enumerated from the reads (seg_reads: nseg + 1 read offsets; label:
// the reads' components, null in the first scan; every read at most 300 positions; seg_len: with several segments, each
// one's longest read, else empty), or of tuples enumerated before, segment-major.
int group_bins_reads(GroupScan &g, const uint8_t *fq, const ParsedReads &pr, const std::vector<uint64_t> &seg_reads,
                     const uint32_t *label, uint64_t *k1, uint32_t *id1, DeviceArena &arena, cudaStream_t st,
                     const std::vector<uint32_t> &seg_len = {});
int group_bins_tuples(GroupScan &g, const uint64_t *lo, const uint8_t *hi, const uint32_t *id, uint64_t *k1, uint32_t *id1,
                      DeviceArena &arena, cudaStream_t st);
// Whether the scans [scan[s], scan[s + 1]) can be split together, and how (m's arrays are then the caller's to set).
bool group_merge(MergedScans &m, const uint64_t *hist, const std::vector<uint32_t> &scan, uint32_t max_len, int k);
// Their first split pass, from the reads; ids are the reads'.
int group_bins_scans(MergedScans &m, const uint64_t *d_hist, int k, const uint8_t *fq, const ParsedReads &pr, cudaStream_t st);
// Before group_plan: g is scan s of m (tuple0: every scan's first tuple among the merged).
void group_take(GroupScan &g, const MergedScans &m, int s, const uint32_t *label, const std::vector<uint64_t> &tuple0);
// Second pass: the bins' tuples into units.
int group_units(GroupScan &g, const uint64_t *k1, const uint32_t *id1, uint64_t *k2, uint32_t *id2, cudaStream_t st);
// The mischief filter over the split tuples (kk, ids), and every k-mer's reads side by side in out (n ids).
int group_filter(GroupScan &g, const uint64_t *kk, const uint32_t *ids, uint32_t *out, uint32_t *parent, uint8_t *filtered,
                 DeviceArena &arena, cudaStream_t st);
// The unions over the grouped ids and the compression; open: what the caller has to finish (group_finish).
int group_union(GroupScan &g, const uint32_t *out, uint32_t *parent, const uint8_t *filtered, uint64_t n_reads,
                DeviceArena &arena, cudaStream_t st, std::vector<GroupQuirk> &open);
// The first of the tuples (lo, hi, id)[0, n) by (k-mer, adjacency, position): its id.
int first_tuple_id(const uint64_t *lo, const uint8_t *hi, const uint32_t *id, uint64_t n, DeviceArena &arena, cudaStream_t st,
                   uint32_t *out);
// Unites a segment's last run (a read of it: anchor) with the segment's first read (or hooks that read below it
// when it is BAD, as union_scan does; *hooked as there) and compresses again.
int group_finish(uint32_t *parent, uint64_t n_reads, uint32_t first, uint32_t anchor, DeviceArena &arena, cudaStream_t st,
                 uint32_t *hooked);

}  // namespace mp
