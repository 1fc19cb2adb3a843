// H*v of a batched job with the whole vector on chip.
//
// A job (one sector) is run by CL CTAs of kOcThreads threads (one cluster, or
// one CTA).  The vector is the DimUp x DimDw matrix; each CTA keeps a contiguous
// block of columns in shared memory, with the row hop table of the sector and
// the column hop tables of its own columns: a Lanczos step reads nothing from
// L2.  Rows are the up words, columns the down words; up to kOcThreads rows.
// Every element's arithmetic is that of the jobs in batch.cu and the sums hardly
// depend on the split of the elements (CSum::add_product): G(i w_n) of 32 solves
// (4 to 14 sites, one to three orbitals, one to sixteen CTAs) was equal in every
// bit, or to 6e-16, between the two.
//  * Row hops gather from the element's own column in this CTA's shared memory.
//    A thread owns one row and walks over columns, four at a time, so that one
//    table entry and one coupling serve four gathers.
//  * Column hops read whole neighbour columns: from this CTA's shared memory,
//    or through distributed shared memory from the CTA that owns the column; a
//    table entry is the coupling and the neighbour column's shared-window
//    address, one 16-byte broadcast.  The words of a class ascend, so a block
//    of columns shares its high sites and most hops stay inside it (a warp's
//    256-byte read of another CTA's shared memory takes 13.6 cycles of the SM
//    against 2 for its own; copies of the vector in L2, read there instead,
//    took a third longer for their latency).
//  * The previous vector lives in registers: kOcSlots elements per thread.
//  * A sum over the job is one barrier: every warp writes its partial into all
//    CTAs of the cluster, and after the barrier every warp folds the partials
//    in the same (CTA, warp) order, so all threads hold identical numbers.
//    The same barrier separates a step's gathers from the writes of the next
//    vector, and those from the next gathers: two barriers per Lanczos step.
// What bounds it: the shared-memory pipe (2 wavefronts per 8-byte warp load, 3
// for a row gather with its bank conflicts) for sectors of tens of thousands
// of states, the two barriers and sums (1,000 cycles each on one CTA, 1,800 on
// four, of which the cluster barrier is 470) below a few thousand.
#pragma once
#include <cooperative_groups.h>

#include "internal.cuh"
#include "reduce.cuh"
#include "sector.cuh"

namespace dmfted {

constexpr int kOcThreads = 512;               // 128 registers per thread
constexpr int kOcWarps = kOcThreads / 32;
constexpr int kOcCols = 4;                    // columns per thread and pass
constexpr int kOcSlots = 32;                  // elements per thread in registers
constexpr size_t kOcMaxSmem = 216 * 1024;     // dynamic shared memory of a job

// Shared memory of a job of R rows (at most wr hops each) and D columns (wc)
// on CL CTAs, each array padded to 16 bytes, and whether a job fits: its
// tables and columns the shared memory, its elements the registers.
__host__ __device__ inline size_t oc_pad(size_t b) { return (b + 15) / 16 * 16; }
__host__ __device__ inline size_t oc_smem(int64_t R, int64_t D, int CL, int wr, int wc, int ni) {
    const size_t cpr = (size_t)((D + CL - 1) / CL);
    return oc_pad(cpr * wc * 16) + oc_pad(cpr * R * 8) + oc_pad(2 * kMaxParams * 8) +
           oc_pad(cpr * 8) + oc_pad((size_t)ni * ni * 8) + oc_pad((size_t)wr * R * 4) + oc_pad(cpr * 4);
}
inline bool oc_fits(int64_t R, int64_t D, int CL, int wr, int wc, int ni) {
    if (R > kOcThreads) return false;
    const int64_t cpr = (D + CL - 1) / CL, G = kOcThreads / R;
    return (cpr + G - 1) / G <= kOcSlots && oc_smem(R, D, CL, wr, wc, ni) <= kOcMaxSmem;
}

// A sector's on-chip matrix.
struct OcShape {
    int64_t R, D;
    int wr, wc;
};
inline OcShape oc_shape(const dmfted_ctx *c, int nup, int ndw) {
    return {c->binom[nup], c->binom[ndw], c->spin[0].cls_max[nup],
            (c->spin_shared ? c->spin[0] : c->spin[1]).cls_max[ndw]};
}

// Partials of a job's sums, written by every CTA of the cluster into every
// CTA; two buffers, so that a sum never overwrites the one still being read.
template <int CL>
struct OcSums {
    double part[2][CL * kOcWarps][2];
};

// A column hop: the coupling and the shared-window address of the neighbour
// column.
struct __align__(16) OcHop {
    double t;
    uint32_t addr, pad;
};

// A job's geometry and the calling thread's place in it.  Addresses are bytes
// of the shared window.  Thread (g, r) owns row r of the columns g, g + G, ...
// (nv of them, slot s = column g + G*s); a thread without columns has nv = 0.
struct OcView {
    uint32_t R, D, c0, ncl;  // rows, columns; first column and columns of this CTA
    uint32_t G, g, r;
    int nv, nmax;            // columns of this thread, most of any thread (uniform)
    int wc;                  // most hops of a column
    int nr;                  // hops of this thread's row
    double dr;               // bath energies of the row's word
    uint32_t x0;             // address of slot 0 (column g, row r)
    uint32_t xstep;          // bytes from slot to slot: G columns
    uint32_t ut;             // the row's hop table: row byte offset | coupling offset << 16
    uint32_t spv;            // signed couplings of the row hops: +V, -V per parameter
    uint32_t dc, dcstep;     // [ncl] bath energies of the columns' words; slot step
    uint32_t dint;           // impurity diagonal at this row's impurity state
    uint32_t dh, dhstep;     // [ncl][wc] column hops; bytes from slot to slot
    uint32_t dcnt;           // [ncl] column hop counts | offset of the column's impurity state << 8
};

__device__ __forceinline__ uint32_t oc_cluster_rank(int CL) {
    return CL == 1 ? 0u : (uint32_t)cooperative_groups::this_cluster().block_rank();
}

template <int CL>
__device__ __forceinline__ void oc_barrier() {
    if constexpr (CL == 1) __syncthreads();
    else cooperative_groups::this_cluster().sync();
}

__device__ __forceinline__ uint32_t oc_map(uint32_t addr, uint32_t rank) {
    uint32_t out;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(out) : "r"(addr), "r"(rank));
    return out;
}
__device__ __forceinline__ uint32_t oc_addr(const void *p) {
    return (uint32_t)__cvta_generic_to_shared(p);
}
// Shared-memory accesses by window address; volatile, so that they stay
// between the barriers of the step.
__device__ __forceinline__ double oc_ld(uint32_t a) {
    double v;
    asm volatile("ld.shared.f64 %0, [%1];" : "=d"(v) : "r"(a));
    return v;
}
__device__ __forceinline__ void oc_st(uint32_t a, double v) {
    asm volatile("st.shared.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory");
}
__device__ __forceinline__ uint32_t oc_ld32(uint32_t a) {
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a));
    return v;
}
__device__ __forceinline__ OcHop oc_ldhop(uint32_t a) {
    OcHop h;
    double q;
    asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(h.t), "=d"(q) : "r"(a));
    h.addr = (uint32_t)__double2loint(q);
    h.pad = 0;
    return h;
}
// A neighbour column's element: own CTA or cluster.
template <int CL>
__device__ __forceinline__ double oc_ldn(uint32_t a) {
    if constexpr (CL == 1) return oc_ld(a);
    double v;
    asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(a));
    return v;
}

// Sum of this thread's compensated partial over all threads of the job, in
// every thread.  buf alternates between calls.
template <int CL>
__device__ __forceinline__ double oc_sum(CSum s, OcSums<CL> &sums, int &buf) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    warp_reduce(s);
    if constexpr (CL == 1) {
        if (lane == 0) {
            sums.part[buf][warp][0] = s.hi;
            sums.part[buf][warp][1] = s.lo;
        }
    } else {
        s.hi = __shfl_sync(0xffffffffu, s.hi, 0);
        s.lo = __shfl_sync(0xffffffffu, s.lo, 0);
        if (lane < CL) {
            const uint32_t a =
                oc_map(oc_addr(&sums.part[buf][oc_cluster_rank(CL) * kOcWarps + warp][0]), lane);
            asm volatile("st.shared::cluster.v2.f64 [%0], {%1, %2};" ::"r"(a), "d"(s.hi), "d"(s.lo)
                         : "memory");
        }
        __syncwarp();
    }
    oc_barrier<CL>();
    CSum t;
    t.zero();
#pragma unroll
    for (int i = 0; i < (CL * kOcWarps + 31) / 32; i++) {
        const int k = i * 32 + lane;
        if (k < CL * kOcWarps) t.merge(sums.part[buf][k][0], sums.part[buf][k][1]);
    }
    warp_reduce(t);
    buf ^= 1;
    return __shfl_sync(0xffffffffu, t.value(), 0);
}

// Tables of the job's sector in shared memory (dyn: oc_smem bytes).  Ends
// with a block barrier; no other CTA's shared memory is touched.
template <int CL>
__device__ __noinline__ void oc_setup(OcView &v, unsigned char *dyn, const BatchTables<double> &tb,
                                      int nup, int ndw) {
    const int nr = nup, nc = ndw;
    const BatchSpin<double> &sr = tb.sp[0], &sc = tb.sp[1];
    const int wr = tb.hmax[0][nr];
    v.wc = tb.hmax[1][nc];
    const int64_t orow = tb.poff[nr], ocol = tb.poff[nc];
    const uint32_t *er = sr.ell + (int64_t)tb.W * orow, *ec = sc.ell + (int64_t)tb.W * ocol;
    const uint32_t tid = threadIdx.x, bd = blockDim.x, rank = oc_cluster_rank(CL);
    const uint32_t ni = 1u << tb.norb, imask = ni - 1u;
    v.R = (uint32_t)tb.binom[nr];
    v.D = (uint32_t)tb.binom[nc];
    const uint32_t cpr = (v.D + CL - 1) / CL;
    v.c0 = min(rank * cpr, v.D);
    v.ncl = min(cpr, v.D - v.c0);
    v.G = kOcThreads / v.R;
    v.g = tid / v.R;
    v.r = tid - v.g * v.R;
    v.nv = v.g < v.G && v.g < v.ncl ? (int)((v.ncl - v.g + v.G - 1) / v.G) : 0;
    v.nmax = (int)((cpr + v.G - 1) / v.G);
    unsigned char *p = dyn;
    auto take = [&](size_t bytes) {
        unsigned char *q = p;
        p += oc_pad(bytes);
        return q;
    };
    OcHop *dh = (OcHop *)take((size_t)cpr * v.wc * 16);
    double *xs = (double *)take((size_t)cpr * v.R * 8);
    double *spv = (double *)take(2 * kMaxParams * 8);
    double *dc = (double *)take((size_t)cpr * 8);
    double *dint = (double *)take((size_t)ni * ni * 8);
    uint32_t *ut = (uint32_t *)take((size_t)wr * v.R * 4);
    uint32_t *dcnt = (uint32_t *)take((size_t)cpr * 4);
    for (uint32_t i = tid; i < 2u * tb.P; i += bd) {
        const double c = sr.par[i >> 1];
        spv[i] = (i & 1) ? -c : c;
    }
    for (uint32_t r = tid; r < v.R; r += bd) {
        const int n = min((int)sr.cnt[orow + r], wr);
        for (int e = 0; e < n; e++) {
            const uint32_t en = er[(int64_t)e * v.R + r];
            const bool ok = DM_IN(ell_col(en), v.R) && DM_IN(ell_par(en), tb.P);
            const uint32_t cp = (2u * ell_par(en) + (ell_neg(en) ? 1u : 0u)) * 8u;
            ut[e * v.R + r] = ok ? ell_col(en) * 8u | cp << 16 : r * 8u;
        }
    }
    for (uint32_t i = tid; i < ni * ni; i += bd) dint[i] = tb.dint[i];
    const uint32_t xs0 = oc_addr(xs);
    for (uint32_t c = tid; c < v.ncl; c += bd) {
        const uint32_t q = v.c0 + c;
        dc[c] = sc.diag[ocol + q];
        const uint32_t ic = tb.words[ocol + q] & imask;
        const int n = min((int)sc.cnt[ocol + q], v.wc);
        dcnt[c] = (uint32_t)n | (ic * 8u) << 8;
        for (int e = 0; e < n; e++) {
            const uint32_t en = ec[(int64_t)e * v.D + q];
            const bool ok = DM_IN(ell_col(en), v.D) && DM_IN(ell_par(en), tb.P);
            const uint32_t t = ok ? ell_col(en) : q, owner = t / cpr;
            const double cv = ok ? sc.par[ell_par(en)] : 0.0;
            const uint32_t a = xs0 + (t - owner * cpr) * v.R * 8u;
            dh[c * v.wc + e] = OcHop{ell_neg(en) ? -cv : cv, CL == 1 ? a : oc_map(a, owner), 0u};
        }
    }
    const uint32_t rr = min(v.r, v.R - 1), gg = v.nv > 0 ? v.g : 0u;
    v.nr = min((int)sr.cnt[orow + rr], wr);
    v.dr = sr.diag[orow + rr];
    v.x0 = xs0 + (gg * v.R + rr) * 8u;
    v.xstep = v.G * v.R * 8u;
    v.ut = oc_addr(ut) + rr * 4u;
    v.spv = oc_addr(spv);
    v.dc = oc_addr(dc) + gg * 8u;
    v.dcstep = v.G * 8u;
    v.dint = oc_addr(dint) + (tb.words[orow + rr] & imask) * ni * 8u;
    v.dh = oc_addr(dh) + gg * v.wc * 16u;
    v.dhstep = v.G * v.wc * 16u;
    v.dcnt = oc_addr(dcnt) + gg * 4u;
    __syncthreads();
}

// (H x) of the thread's slots s0 .. s0+3 and their own values x (zero for the
// slots beyond nv).
template <int CL>
__device__ __forceinline__ void oc_product(const OcView &v, int s0, double (&h)[kOcCols],
                                           double (&x)[kOcCols]) {
    const uint32_t r8 = v.r * 8u;
    uint32_t col[kOcCols];  // addresses of the columns' row 0
    int nd[kOcCols], ndmax = 0;
#pragma unroll
    for (int j = 0; j < kOcCols; j++) {
        x[j] = h[j] = 0.0;
        nd[j] = 0;
        const uint32_t a = v.x0 + (s0 + j) * v.xstep;
        col[j] = a - r8;
        if (s0 + j < v.nv) {
            x[j] = oc_ld(a);
            nd[j] = (int)oc_ld32(v.dcnt + (s0 + j) * v.G * 4u);
            h[j] = oc_ld(v.dc + (s0 + j) * v.dcstep);
        }
    }
#pragma unroll
    for (int j = 0; j < kOcCols; j++) {
        h[j] = (v.dr + h[j] + oc_ld(v.dint + ((uint32_t)nd[j] >> 8))) * x[j];
        nd[j] &= 0xff;
        ndmax = max(ndmax, nd[j]);
        if (s0 + j >= v.nv) col[j] = col[0];  // gathers of unused slots repeat the first
    }
    const int nr = s0 < v.nv ? v.nr : 0;
    uint32_t ut = v.ut;
#pragma unroll 2
    for (int e = 0; e < nr; e++) {
        const uint32_t en = oc_ld32(ut);
        ut += v.R * 4u;
        const uint32_t ro = en & 0xffffu;
        const double t = oc_ld(v.spv + (en >> 16));
#pragma unroll
        for (int j = 0; j < kOcCols; j++) h[j] = fma(t, oc_ld(col[j] + ro), h[j]);
    }
    uint32_t dh[kOcCols];
#pragma unroll
    for (int j = 0; j < kOcCols; j++) dh[j] = v.dh + (s0 + j) * v.dhstep;
#pragma unroll 2
    for (int e = 0; e < ndmax; e++) {
#pragma unroll
        for (int j = 0; j < kOcCols; j++)
            if (e < nd[j]) {
                const OcHop q = oc_ldhop(dh[j] + e * 16u);
                h[j] = fma(q.t, oc_ldn<CL>(q.addr + r8), h[j]);
            }
    }
#pragma unroll
    for (int j = 0; j < kOcCols; j++)
        if (s0 + j >= v.nv) h[j] = 0.0;
}

}  // namespace dmfted
