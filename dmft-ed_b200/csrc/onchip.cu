// Batched Green's-function chains with their vectors on chip (onchip.cuh).
#include <algorithm>
#include <vector>

#include "batch.cuh"
#include "onchip.cuh"

namespace dmfted {

// ---- a chain (chain_job in batch.cu) with its vectors on chip ---------------
// One Lanczos step: u = sc H x - b_k scp v_prev over v_prev's registers and
// alpha (first barrier), then x -> v_prev, w = u - alpha sc x -> x and |w|
// (second barrier).  Green's-function phase of the two-orbital Ns=10 solve at
// finite temperature (88 to 200 chains of up to 52,920 states, four CTAs for the
// large ones), four baths: 17.3 / 10.0 / 12.9 / 23.0 ms against 24.8 / 18.5 / 18.6 /
// 33.9 with the vectors in L2; of the Ns=8 scan (4,900 and 3,920 states) 1.26
// against 2.1 ms; a chain of 108,900 states on sixteen CTAs 8.4 against 12.2 ms.
template <int CL>
__device__ void chain_job_oc(const BatchTables<double> &tb, OcSums<CL> &sums, unsigned char *dyn,
                             const ChainJob &J, const double *states64, double *alpha,
                             double *beta, int *nsteps, double *norm2, double thr,
                             const BatchCaps &cap) {
    OcView v0;
    oc_setup<CL>(v0, dyn, tb, J.tnup, J.tndw);
    OcView v = v0;  // in registers
    if (!DM_IN(J.slot, cap.slots) || !DM_IN(J.kmax, kChainStride - 1)) return;
    const bool lead = oc_cluster_rank(CL) == 0 && threadIdx.x == 0;
    double *al = alpha + (int64_t)J.slot * kChainStride;
    double *be = beta + (int64_t)J.slot * kChainStride;
    int buf = 0;
    double prev[kOcSlots];
    // start vector: c^+ / c on the state (the k_apply_op rule)
    CSum a;
    a.zero();
    {
        const double *psi = states64 + J.psi_off;
        const uint32_t bit = 1u << J.iorb;
        const int64_t sdimup = tb.binom[J.snup];
        const uint32_t *wu = tb.words + tb.poff[J.tnup], *wd = tb.words + tb.poff[J.tndw];
#pragma unroll
        for (int s = 0; s < kOcSlots; s++) {
            prev[s] = 0.0;
            if (s >= v.nv) continue;
            const uint32_t r = v.r, q = v.c0 + v.g + v.G * s;  // up and down ranks
            const uint32_t wj = J.ispin == 0 ? wu[r] : wd[q];
            double val = 0.0;
            const bool has = (wj & bit) != 0u;
            if (J.particle ? has : !has) {
                const uint32_t w = J.particle ? (wj ^ bit) : (wj | bit);
                const int64_t rs = DM_IN(w, tb.nrank) ? tb.rank[w] : 0;
                uint32_t par = __popc(w & (bit - 1u)) & 1u;
                int64_t src;
                if (J.ispin == 0) {
                    src = rs + sdimup * q;
                } else {
                    par ^= (uint32_t)J.snup & 1u;
                    src = r + sdimup * rs;
                }
                if (DM_IN(J.psi_off + src, cap.states)) val = par ? -psi[src] : psi[src];
            }
            oc_st(v.x0 + s * v.xstep, val);
            a.add_product(val, val);
        }
    }
    const double n2 = oc_sum<CL>(a, sums, buf);
    if (lead) norm2[J.slot] = n2;
    double sc = n2 > 0.0 ? 1.0 / sqrt(n2) : 0.0, scp = 0.0, bk = 0.0;
    int steps = 0;
    for (int k = 0; k < J.kmax; k++) {
        // keeps the slots' addresses from being hoisted out of the loop into
        // registers that prev needs
        asm volatile("" : "+r"(v.xstep), "+r"(v.dhstep), "+r"(v.dcstep), "+r"(v.G));
        const double cprev = k > 0 ? bk * scp : 0.0;
        a.zero();
#pragma unroll
        for (int s = 0; s < kOcSlots; s += kOcCols)
            if (s < v.nmax) {
                double h[kOcCols], x[kOcCols];
                oc_product<CL>(v, s, h, x);
#pragma unroll
                for (int j = 0; j < kOcCols; j++) {
                    if (s + j >= v.nv) continue;
                    const double u = sc * h[j] - cprev * prev[s + j];
                    prev[s + j] = u;
                    a.add_product(x[j], u);
                }
            }
        const double ak = sc * oc_sum<CL>(a, sums, buf);
        const double coef = ak * sc;
        a.zero();
#pragma unroll
        for (int s = 0; s < kOcSlots; s += kOcCols)
            if (s < v.nmax) {
#pragma unroll
                for (int j = 0; j < kOcCols; j++) {
                    if (s + j >= v.nv) continue;
                    const uint32_t xa = v.x0 + (s + j) * v.xstep;
                    const double x = oc_ld(xa), w = prev[s + j] - coef * x;
                    prev[s + j] = x;
                    oc_st(xa, w);
                    a.add_product(w, w);
                }
            }
        const double bn = sqrt(oc_sum<CL>(a, sums, buf));
        if (lead) {
            al[k] = ak;
            be[k + 1] = bn;
        }
        steps = k + 1;
        scp = sc;
        sc = bn > 0.0 ? 1.0 / bn : 0.0;
        bk = bn;
        if (bn < thr) break;
    }
    if (lead) {
        be[0] = 0.0;
        nsteps[J.slot] = steps;
    }
    __syncthreads();  // the next job's tables overwrite this one's
}

// k_batch_chains with on-chip jobs: chains [0, nbig) by the clusters, the rest
// one per CTA.
template <int CL>
__global__ void __launch_bounds__(kOcThreads, 1)
    k_chains_onchip(const __grid_constant__ BatchTables<double> tb, const ChainJob *jobs, int nbig, int njobs,
                    unsigned *queue, const double *states64, double *alpha, double *beta,
                   
                    int *nsteps, double *norm2, double thr, const BatchCaps cap) {
    extern __shared__ __align__(16) unsigned char ocdyn[];
    __shared__ __align__(16) OcSums<CL> sums;
    __shared__ QueueSlot sm;
    if constexpr (CL > 1) {
        for (;;) {
            const int jid = next_job<CL>(queue, sm);
            if (jid >= nbig) break;
            chain_job_oc<CL>(tb, sums, ocdyn, jobs[jid], states64, alpha, beta, nsteps, norm2, thr,
                             cap);
        }
    }
    // one CTA alone uses the first warps' slots of the same sums
    OcSums<1> &one = *reinterpret_cast<OcSums<1> *>(&sums);
    for (;;) {
        const int jid = nbig + next_job<1>(queue + 1, sm);
        if (jid >= njobs) break;
        chain_job_oc<1>(tb, one, ocdyn, jobs[jid], states64, alpha, beta, nsteps, norm2, thr, cap);
    }
}

template <int CL>
static void chains_attr(dmfted_ctx *c) {
    static bool attr[64] = {false};
    if (!attr[c->device & 63]) {
        DM_CUDA(cudaFuncSetAttribute(k_chains_onchip<CL>,
                                     cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)kOcMaxSmem));
        attr[c->device & 63] = true;
    }
}

// Whether the device takes a cluster of 16 CTAs with their full shared memory:
// it is above the portable size, and a device with fewer SMs per GPC (or a
// partition of one) has no room for it.
static bool sixteen_fit(dmfted_ctx *c) {
    if (c->onchip_16 < 0) {
        chains_attr<16>(c);
        DM_CUDA(cudaFuncSetAttribute(k_chains_onchip<16>,
                                     cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
        cudaLaunchConfig_t cfg = {};
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = 16;
        at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
        cfg.gridDim = dim3(16);
        cfg.blockDim = dim3(kOcThreads);
        cfg.dynamicSmemBytes = kOcMaxSmem;
        cfg.attrs = at;
        cfg.numAttrs = 1;
        int n = 0;
        if (cudaOccupancyMaxActiveClusters(&n, k_chains_onchip<16>, &cfg) != cudaSuccess) {
            (void)cudaGetLastError();
            n = 0;
        }
        c->onchip_16 = n > 0;
    }
    return c->onchip_16 != 0;
}

int oc_need(dmfted_ctx *c, int nup, int ndw) {
    const OcShape o = oc_shape(c, nup, ndw);
    for (int cl = 1; cl <= std::min(c->onchip_max, 16); cl *= 2)
        if (oc_fits(o.R, o.D, cl, o.wr, o.wc, 1 << c->norb))
            return cl < 16 || sixteen_fit(c) ? cl : 0;
    return 0;
}

template <int CL>
static void launch_chains(dmfted_ctx *c, const ChainQueue &q, int nbig, int nj, size_t smem,
                          double *alpha, double *beta, int *nsteps, double *norm2, int64_t nslots) {
    chains_attr<CL>(c);
    launch_persistent(c, k_chains_onchip<CL>, CL, nbig + div_up(nj - nbig, CL), kOcThreads, smem,
                      batch_tables<double>(c), (const ChainJob *)q.jobs, nbig, nj, q.next,
                      (const double *)c->states64.p, alpha, beta, nsteps, norm2, c->p.lanc_gf_threshold,
                      BatchCaps{0, 0, 0, (int64_t)c->states64.n, nslots});
}

void run_chains_onchip(dmfted_ctx *c, int CL, const ChainQueue &q, std::vector<ChainJob> jobs,
                       double *alpha, double *beta, int *nsteps, double *norm2, int64_t nslots) {
    auto dims = [&](const ChainJob &J) { return c->binom[J.tnup] * c->binom[J.tndw]; };
    while (CL > 1 && (CL > c->onchip_max || (CL > 8 && !sixteen_fit(c)))) CL /= 2;
    for (const ChainJob &J : jobs) CL = std::max(CL, oc_need(c, J.tnup, J.tndw));
    auto shared = [&](const ChainJob &J) {
        return CL > 1 && (oc_need(c, J.tnup, J.tndw) > 1 || dims(J) >= c->batch_cluster_min * CL);
    };
    const int nbig = (int)(std::stable_partition(jobs.begin(), jobs.end(), shared) - jobs.begin());
    const int nj = (int)jobs.size();
    size_t smem = 0;
    for (int i = 0; i < nj; i++) {
        const OcShape o = oc_shape(c, jobs[i].tnup, jobs[i].tndw);
        smem = std::max(smem, oc_smem(o.R, o.D, i < nbig ? CL : 1, o.wr, o.wc, 1 << c->norb));
    }
    q.fill(c, jobs);
    switch (CL) {
        case 16: launch_chains<16>(c, q, nbig, nj, smem, alpha, beta, nsteps, norm2, nslots); break;
        case 8: launch_chains<8>(c, q, nbig, nj, smem, alpha, beta, nsteps, norm2, nslots); break;
        case 4: launch_chains<4>(c, q, nbig, nj, smem, alpha, beta, nsteps, norm2, nslots); break;
        case 2: launch_chains<2>(c, q, nbig, nj, smem, alpha, beta, nsteps, norm2, nslots); break;
        default: launch_chains<1>(c, q, 0, nj, smem, alpha, beta, nsteps, norm2, nslots); break;
    }
}

}  // namespace dmfted
