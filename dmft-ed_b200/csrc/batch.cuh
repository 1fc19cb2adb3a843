// What the batched kernels share (batch.cu, onchip.cu): the job records, the
// work queue and the persistent launch.
#pragma once
#include <cooperative_groups.h>

#include <algorithm>
#include <utility>
#include <vector>

#include "internal.cuh"

namespace dmfted {

template <int CL>
__device__ __forceinline__ int cta_rank() {
    if constexpr (CL == 1) return 0;
    else return (int)cooperative_groups::this_cluster().block_rank();
}

struct QueueSlot {
    int job, jobl;
};

// Next job of the queue for this CTA (CL == 1) or cluster (rank 0 takes it,
// the others read it from rank 0's shared memory).  The closing barrier
// keeps rank 0 from exiting or overwriting the slot before every CTA read it.
template <int CL, typename Slot>
__device__ __forceinline__ int next_job(unsigned *queue, Slot &sm) {
    if constexpr (CL == 1) {
        if (threadIdx.x == 0) sm.job = (int)atomicAdd(queue, 1u);
        __syncthreads();
        const int j = sm.job;
        __syncthreads();
        return j;
    } else {
        cooperative_groups::cluster_group cl = cooperative_groups::this_cluster();
        if (cl.block_rank() == 0 && threadIdx.x == 0) sm.job = (int)atomicAdd(queue, 1u);
        cl.sync();
        if (threadIdx.x == 0) sm.jobl = *cl.map_shared_rank(&sm.job, 0);
        cl.sync();
        return sm.jobl;
    }
}

struct ChainJob {
    int tnup, tndw;        // target sector
    int snup;              // source sector's nup (down-spin sign)
    int ispin, iorb, particle;
    int kmax;
    int slot;              // output slot
    int64_t psi_off;       // FP64 state vector in the eigenspace pool
    int64_t work_off;      // elements of T: three vectors of the job
};

// Chain output slot: alpha[kLzMax+2], beta[kLzMax+2], then nsteps and norm2
// in separate arrays.
constexpr int kChainStride = kLzMax + 2;

// Extents of the buffers a batched launch writes or gathers from, checked
// against every job in a checked build (the checks are uniform over the CTAs
// of a cluster, so a skipped job is skipped by all of them).
struct BatchCaps {
    int64_t work, vec, aux, states, slots, lock;
};

// Where a list of chains keeps its job records and its two queue counters.
struct ChainQueue {
    ChainJob *jobs;
    unsigned *next;
    void fill(dmfted_ctx *c, const std::vector<ChainJob> &list) const {
        DM_CUDA(cudaMemcpyAsync(jobs, list.data(), list.size() * sizeof(ChainJob),
                                cudaMemcpyHostToDevice, c->stream));
        DM_CUDA(cudaMemsetAsync(next, 0, 2 * sizeof(unsigned), c->stream));
    }
};

struct EigsJob {
    int nup, ndw;
    int neigen, kmax;
    int slot;          // output slot: evals, steps
    int64_t basis_off; // elements of T: (kmax + 1) vectors of ld elements
    int64_t vec_off;   // FP64 eigenvectors: neigen x dim
    int64_t aux_off;   // FP64 scratch: Y and coefficients (2 x neigen x kmax)
    int64_t lock_off;  // locked FP64 vectors (dim apart) in the lock pool
    int nlock;         // how many (0: plain run)
    double top;        // probe: eigenvalues above this are not wanted (early stop)
};

// Persistent launch: as many CTAs (CL == 1) or clusters as can be resident,
// at most one per job.
template <typename... KArgs, typename... Args>
inline void launch_persistent(dmfted_ctx *c, void (*kern)(KArgs...), int CL, int njobs,
                              int threads, size_t smem, Args &&...args) {
    cudaLaunchConfig_t cfg = {};
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = c->stream;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = CL;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = CL > 1 ? 1 : 0;
    if (CL > 8) {
        // 16 CTAs per cluster is beyond the portable size: opt in per kernel
        DM_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    }
    int units = std::max(1, num_sms(c) / CL);
    if (CL > 1) {
        cfg.gridDim = dim3(units * CL);
        int ncl = 0;
        if (cudaOccupancyMaxActiveClusters(&ncl, kern, &cfg) == cudaSuccess && ncl > 0)
            units = ncl;
        else
            (void)cudaGetLastError();
    }
    units = std::min(units, njobs);
    cfg.gridDim = dim3(units * CL);
    DM_CUDA(cudaLaunchKernelEx(&cfg, kern, std::forward<Args>(args)...));
    c->launches++;
}

// ---- onchip.cu -------------------------------------------------------------
// CTAs a job needs to keep its vectors on chip (0: it does not fit the largest
// cluster).
int oc_need(dmfted_ctx *c, int nup, int ndw);
// The chains that fit on chip, in one launch; CL: CTAs of the shared ones
// (raised to what the largest needs).
void run_chains_onchip(dmfted_ctx *c, int CL, const ChainQueue &q, std::vector<ChainJob> jobs,
                       double *alpha, double *beta, int *nsteps, double *norm2, int64_t nslots);

}  // namespace dmfted
