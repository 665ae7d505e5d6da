#pragma once
#include "k_reads.cuh"

namespace mp {

// K1: bucket counts.  cc (nullable): per-chunk u32 counts [nchunks][NB]; glob: u64 counts [NB]
// (summed from cc when cc is given; nullable with cc).  Reads longer than MAX_READ_COUNT are the caller's to refuse
// (plain variant: pr.max_len; 3-minimizer variant: DERR_LONG_READ in err).  odd (plain variant): a sequence byte other
// than A, C, G, T, N sets DERR_NONACGT in err.
void launch_count(const uint8_t *fq, const ParsedReads &pr, int k, int min3, const uint64_t *chunk_rec, int nchunks,
                  uint32_t *cc, unsigned long long *glob, uint32_t *err, cudaStream_t st, bool odd = false);

// K2a: tuples per read in the bucket range [lo, hi).
void launch_enum_count(const uint8_t *fq, const ParsedReads &pr, int k, int min3, uint32_t lo, uint32_t hi,
                       uint32_t *cnt, uint32_t *err, cudaStream_t st);

// K2a for all scans at once (plain variant, at most 8 scans): cnt[s * stride + read] for the buckets
// [bounds[s], bounds[s+1]) (bounds: S + 1 device words).  Returns -1 (nothing launched) for other S.
int launch_enum_count_scans(const uint8_t *fq, const ParsedReads &pr, int k, const uint32_t *bounds, int S,
                            uint32_t *cnt, uint64_t stride, uint32_t *err, cudaStream_t st);

// K2b: tuples at off[read]: o_lo = kmer << 8 | adj, o_hi = kmer >> 56 (nullable when k <= 28),
// o_id = read id (scan 0, label == nullptr) or its component label.
void launch_enum_write(const uint8_t *fq, const ParsedReads &pr, int k, int min3, uint32_t lo, uint32_t hi,
                       const uint32_t *label, const uint64_t *off, uint64_t *o_lo, uint8_t *o_hi, uint32_t *o_id,
                       uint32_t *err, cudaStream_t st);

// K2 of the 3-minimizer variant in one pass, for readers that need no order: the tuples (as launch_enum_write's) at places
// counted in *total (zero before); those past n are counted and not written.
void launch_enum_min3(const uint8_t *fq, const ParsedReads &pr, int k, uint32_t lo, uint32_t hi, const uint32_t *label,
                      unsigned long long *total, uint64_t n, uint64_t *o_lo, uint8_t *o_hi, uint32_t *o_id, uint32_t *err,
                      cudaStream_t st);

}  // namespace mp
