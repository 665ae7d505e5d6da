// Host-side pieces shared by the job driver (mp_api.cu) and the batch driver (mp_batch.cu).
#pragma once
#include <nvtx3/nvToolsExt.h>
#include "k_reads.cuh"

namespace mp {

// Read stores of a job (mp_job_set_read_store).
constexpr int STORE_FASTQ = MP_STORE_FASTQ, STORE_KMER_CACHE = MP_STORE_KMER_CACHE, STORE_PACKED = MP_STORE_PACKED;

// The context's device and its HBM budget accounting (shared by every job and batch of the context).
int ctx_device(const mp_ctx *ctx);
void ctx_budget(mp_ctx *ctx, std::atomic<uint64_t> **used, uint64_t *limit);

// parent[x] = x for every read.
void launch_init_parent(uint32_t *parent, uint64_t n, cudaStream_t st);

// Device time of the work queued on a stream while the timer lives, added to *slot (ms).
// The stages of a job or batch, in the order of their time slots (mp_job_stage_ms, mp_batch_stage_ms).
constexpr const char *STAGE_NAMES[8] = {"parse", "count", "enumerate", "sort", "filter", "union_find",
                                        "mate_union_plan", "output"};

// A stage's device time (CUDA events on its stream, added to its slot) and an NVTX range of the stage's
// name for a profiler's timeline (a no-op without one attached).
struct StageTimer {
    cudaEvent_t a, b;
    cudaStream_t st;
    double *acc;
    StageTimer(cudaStream_t s, double *slots, int stage) : st(s), acc(slots + stage)
    {
        nvtxRangePushA(STAGE_NAMES[stage]);
        cudaEventCreate(&a);
        cudaEventCreate(&b);
        cudaEventRecord(a, st);
    }
    ~StageTimer()
    {
        cudaEventRecord(b, st);
        cudaEventSynchronize(b);
        float ms = 0;
        cudaEventElapsedTime(&ms, a, b);
        *acc += ms;
        cudaEventDestroy(a);
        cudaEventDestroy(b);
        nvtxRangePop();
    }
    StageTimer(const StageTimer &) = delete;
    StageTimer &operator=(const StageTimer &) = delete;
};

}  // namespace mp
