// Host-side pieces shared by the job driver (mp_api.cu) and the batch driver (mp_batch.cu).
#pragma once
#include <nvtx3/nvToolsExt.h>

#include <vector>

#include "k_reads.cuh"

namespace mp {

// Read stores of a job (mp_job_set_read_store).
constexpr int STORE_FASTQ = MP_STORE_FASTQ, STORE_KMER_CACHE = MP_STORE_KMER_CACHE, STORE_PACKED = MP_STORE_PACKED;

// The context's device and its HBM budget accounting (shared by every job and batch of the context).
int ctx_device(const mp_ctx *ctx);
void ctx_budget(mp_ctx *ctx, std::atomic<uint64_t> **used, uint64_t *limit);

// The device bytes that are set aside for a job's input (a request's footprint): it takes no more than these by choice.
void job_set_share(mp_job *job, uint64_t bytes);

// parent[x] = x for every read.
void launch_init_parent(uint32_t *parent, uint64_t n, cudaStream_t st);

// The stages of a job or batch, in the order of their time slots (mp_job_stage_ms, mp_batch_stage_ms).
constexpr const char *STAGE_NAMES[8] = {"parse", "count", "enumerate", "sort", "filter", "union_find",
                                        "mate_union_plan", "output"};
constexpr int SPLIT_SLOT = 8;  // the split passes of grouped scans, apart

// Device time per stage in ms, from event pairs that are read when the times are asked for: a stage's end is not waited
// for (eight waits per job, 10-20 us each, kept the host from queueing ahead).
struct StageClock {
    struct Pending {
        cudaEvent_t a, b;
        int slot[2];
    };
    double ms[9] = {0};
    std::vector<Pending> pending;
    std::vector<cudaEvent_t> pool;

    cudaEvent_t take()
    {
        cudaEvent_t e = nullptr;
        if (!pool.empty()) {
            e = pool.back();
            pool.pop_back();
        } else {
            cudaEventCreate(&e);
        }
        return e;
    }
    void clear(int slot)
    {
        ms[slot] = 0;
        for (size_t i = 0; i < pending.size();) {
            Pending &p = pending[i];
            for (int &s : p.slot)
                if (s == slot) s = -1;
            if (p.slot[0] < 0 && p.slot[1] < 0) {
                pool.push_back(p.a);
                pool.push_back(p.b);
                pending.erase(pending.begin() + (long)i);
            } else {
                i++;
            }
        }
    }
    void resolve()
    {
        for (Pending &p : pending) {
            float x = 0;
            cudaEventSynchronize(p.b);
            if (cudaEventElapsedTime(&x, p.a, p.b) != cudaSuccess) cudaGetLastError();
            for (int s : p.slot)
                if (s >= 0) ms[s] += x;
            pool.push_back(p.a);
            pool.push_back(p.b);
        }
        pending.clear();
    }
    ~StageClock()
    {
        for (Pending &p : pending) {
            cudaEventDestroy(p.a);
            cudaEventDestroy(p.b);
        }
        for (auto e : pool) cudaEventDestroy(e);
    }
};

// The device time of the work queued on a stream while the timer lives, for a stage's slot (and another's), and an NVTX
// range of the stage's name for a profiler's timeline (a no-op without one attached).
struct StageTimer {
    StageClock &c;
    StageClock::Pending p;
    cudaStream_t st;
    StageTimer(StageClock &clk, cudaStream_t s, int stage, int also = -1) : c(clk), p{clk.take(), clk.take(), {stage, also}}, st(s)
    {
        nvtxRangePushA(STAGE_NAMES[stage]);
        cudaEventRecord(p.a, st);
    }
    ~StageTimer()
    {
        cudaEventRecord(p.b, st);
        c.pending.push_back(p);
        nvtxRangePop();
    }
    StageTimer(const StageTimer &) = delete;
    StageTimer &operator=(const StageTimer &) = delete;
};

}  // namespace mp
