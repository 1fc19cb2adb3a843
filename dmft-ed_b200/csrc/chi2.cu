// Batched chi^2 of the Delta fit and its reverse-mode gradient, for many bath
// parameter sets at once (the reference evaluates one set per call inside
// SciFortran's fmin_cg):
//   Delta_n   = sum_k V_k^2 / (i w_n - e_k)           delta_normal_normal
//   chi2      = sum_n |G_n - Delta_n|^2 / W_n          chi2_delta_normal_normal
//   d chi2/da = -2 sum_n [Re(G-Delta) Re dDelta + Im(G-Delta) Im dDelta] / W_n
//   dDelta/de_k = V_k^2/(i w_n - e_k)^2,  dDelta/dV_k = 2 V_k/(i w_n - e_k)
// (ED_CHI2FIT/fitgf_normal_normal.f90:193-226,256-316).
//
// One CTA per parameter set, threads over Matsubara points.  With NB levels known
// at compile time (up to kChi2Levels) a thread's 1/(e_k^2 + w^2) and its sums of
// chi^2 and of both derivatives stay in registers; V_k^2 and 2 V_k, the same for
// every point, multiply the sums once at the end.  The reciprocal is a Newton
// iteration from the single-precision one, without a branch between the NB chains.
// The sums are folded compensated, one warp per sum, in a fixed order.  What bounds
// it: the FP64 pipe's latency at the few CTAs per SM that the registers allow.
// 4096 sets of 9 levels, 1000 points: 72 us against 133 us with the sums in shared
// memory and divisions (k_chi2); the 20 FP64 operations per level and point are
// 42 us of the pipe.
// Errors against extended precision over 81,920 sets (1 to 16 levels, 200 to 1500
// points), relative to the value or the gradient's norm, this kernel and k_chi2:
// chi^2 4.145e-16 and 4.167e-16 in the mean, gradient 5.110e-16 and 5.124e-16.
// They come from the residual g - Delta, so Im Delta is summed with one rounding
// per level (fma of V^2 and the reciprocal; a rounded product and an addition:
// 4.183e-16 and 5.140e-16), and every term of a final sum is formed first and added
// with one rounding.
#include <algorithm>

#include "internal.cuh"
#include "reduce.cuh"

namespace dmfted {

// Registers hold 3 NB + 1 FP64 values; more CTAs per SM hide latency until the
// spills cost more.  4096 sets, 1000 points, us a call with 2 / 3 / 4 / 5 CTAs:
// 5 levels 49 / 49 / 49 / 47, 8 levels 74 / 74 / 71 / 76, 10 levels 102 / 90 / 88 /
// 115, 11 levels 110 / 99 / 100 / 144, 13 levels 125 / 113 / 127 / 208, 15 levels
// 143 / 141 / 186 / 258, 16 levels 150 / 155 / 222 / 296; up to four levels the
// choice makes no difference.  At 11 levels four are taken for small batches (512
// sets are one wave of four per SM: 12.3 against 14.4 us).
constexpr int kChi2Levels = 16;
constexpr int kChi2Threads = 128;
constexpr int chi2_ctas(int nb) { return nb <= 5 ? 5 : nb <= 11 ? 4 : nb <= 15 ? 3 : 2; }

// 1/d: Newton iteration from the approximate single-precision reciprocal, whose
// argument and result change format by integer shifts of the bit pattern (the
// conversion instructions share the FP64 pipe's slow path).  Each of the two
// steps doubles the 22 bits of the start; the last one leaves its own rounding.
// Against the division: the same bits for all of 1e9 random d, and within one ulp
// (0.8 % of the cases) where d is within 4096 ulp of a power of two.  For d within
// about 1e-29 .. 1e29, where the shifts hold (chi2_in_range).
__device__ __forceinline__ bool chi2_in_range(double d) {
    const int hi = __double2hiint(d);
    return hi > 0x3a000000 && hi < 0x46000000;
}
__device__ __forceinline__ double chi2_recip(double d) {
    const int hi = __double2hiint(d);
    const unsigned f = ((unsigned)(hi - 0x38000000) << 3) | ((unsigned)__double2loint(d) >> 29);
    const unsigned r = __float_as_uint(__fdividef(1.0f, __uint_as_float(f)));
    double y = __hiloint2double((int)(r >> 3) + 0x38000000, (int)(r << 29));
    y = fma(y, fma(-d, y, 1.0), y);
    return fma(y, fma(-d, y, 1.0), y);
}

template <int NB>
__global__ void __launch_bounds__(kChi2Threads, chi2_ctas(NB))
    k_chi2_reg(int L, const double *__restrict__ a, const double *__restrict__ x,
               const double *__restrict__ g, const double *__restrict__ w, double *chi2,
               double *grad) {
    constexpr int NA = 1 + 2 * NB;
    __shared__ double pe[NB], pv[NB], pv2[NB], sums[NA][kChi2Threads];
    const int tid = threadIdx.x;
    const double *ab = a + (int64_t)blockIdx.x * 2 * NB;
    if (tid < NB) {
        pe[tid] = ab[tid];
        pv[tid] = ab[NB + tid];
        pv2[tid] = pv[tid] * pv[tid];
    }
    __syncthreads();
    double s0 = 0.0, se[NB], sv[NB];
#pragma unroll
    for (int k = 0; k < NB; k++) se[k] = sv[k] = 0.0;
    for (int n = tid; n < L; n += kChi2Threads) {
        const double om = x[n], iw = 1.0 / w[n];
        const double2 gn = make_double2(g[2 * n], g[2 * n + 1]);  // g: 8-byte aligned
        const double om2 = om * om;
        double inv[NB], dre = 0.0, dim = 0.0;
        bool ok = true;  // one branch per point: the NB chains run together
#pragma unroll
        for (int k = 0; k < NB; k++) {
            const double d = fma(pe[k], pe[k], om2);
            ok = ok && chi2_in_range(d);
            inv[k] = chi2_recip(d);
        }
        if (!ok) {
#pragma unroll
            for (int k = 0; k < NB; k++) inv[k] = 1.0 / fma(pe[k], pe[k], om2);
        }
        // 1/(i om - e) = (-e - i om) inv; the signs and -om go outside the sums
#pragma unroll
        for (int k = 0; k < NB; k++) {
            dre = fma(pv2[k], pe[k] * inv[k], dre);
            dim = fma(pv2[k], inv[k], dim);
        }
        const double Rr = gn.x + dre, Ri = fma(om, dim, gn.y);
        const double Wr = Rr * iw, Wi = Ri * iw;
        s0 += fma(Rr, Wr, Ri * Wi);
#pragma unroll
        for (int k = 0; k < NB; k++) {
            // dDelta/de = v^2 r^2 ; dDelta/dV = 2 v r, with r = 1/(i om - e)
            const double re = -pe[k] * inv[k], im = -om * inv[k];
            const double t = fma(Wr, re, Wi * im);  // Re(conj(R) r) / W
            const double u = fma(Wi, re, -Wr * im);
            sv[k] += t;
            se[k] += fma(t, re, u * im);  // Re(conj(R) r^2) / W
        }
    }
    sums[0][tid] = s0;
#pragma unroll
    for (int k = 0; k < NB; k++) {
        sums[1 + k][tid] = se[k];
        sums[1 + NB + k][tid] = sv[k];
    }
    __syncthreads();
    const int lane = tid & 31;
    for (int q = tid >> 5; q < NA; q += kChi2Threads / 32) {
        CSum s;
        s.zero();
#pragma unroll
        for (int t = 0; t < kChi2Threads; t += 32) s.add(sums[q][t + lane]);
        warp_reduce(s);
        if (lane == 0) {
            if (q == 0) {
                chi2[blockIdx.x] = s.value();
            } else if (grad) {
                // -2 V^2 or -4 V times the sum, rounded once (V^2 = f + fl exactly)
                const double v = pv[(q - 1) % NB];
                const double f = q <= NB ? v * v : 2.0 * v, fl = q <= NB ? fma(v, v, -f) : 0.0;
                const double p = s.hi * f;
                const double pl = fma(s.hi, f, -p) + fma(s.hi, fl, s.lo * f);
                grad[(int64_t)blockIdx.x * 2 * NB + (q - 1)] = -2.0 * (p + pl);
            }
        }
    }
}

// Any number of levels: r_k and the sums in shared memory, one slot per thread.
__global__ void k_chi2(int nbath, int L, const double *a, const double *x, const double *g,
                       const double *w, double *chi2, double *grad) {
    extern __shared__ double sm[];
    const int nt = blockDim.x, tid = threadIdx.x;
    const int b = blockIdx.x;
    const int na = 1 + 2 * nbath;
    double *pe = sm, *pv = sm + nbath;        // parameters
    double *acc = sm + 2 * nbath;              // [na][nt]
    double *rr = acc + (size_t)na * nt;        // [nbath][nt] real part of r_k
    double *ri = rr + (size_t)nbath * nt;      // imaginary part
    for (int k = tid; k < 2 * nbath; k += nt) sm[k] = a[(int64_t)b * 2 * nbath + k];
    for (int q = 0; q < na; q++) acc[q * nt + tid] = 0.0;
    __syncthreads();
    for (int n = tid; n < L; n += nt) {
        const double om = x[n];
        const double2 gn = make_double2(g[2 * n], g[2 * n + 1]);
        const double iw = 1.0 / w[n];
        double dre = 0.0, dim = 0.0;
        for (int k = 0; k < nbath; k++) {
            const double e = pe[k], v = pv[k];
            const double inv = 1.0 / (e * e + om * om);
            const double re = -e * inv, im = -om * inv;  // 1/(i om - e)
            rr[k * nt + tid] = re;
            ri[k * nt + tid] = im;
            dre += v * v * re;
            dim += v * v * im;
        }
        const double Rr = gn.x - dre, Ri = gn.y - dim;
        acc[tid] += (Rr * Rr + Ri * Ri) * iw;
        for (int k = 0; k < nbath; k++) {
            const double v = pv[k], re = rr[k * nt + tid], im = ri[k * nt + tid];
            // dDelta/de = v^2 r^2 ; dDelta/dV = 2 v r
            const double r2r = re * re - im * im, r2i = 2.0 * re * im;
            acc[(1 + k) * nt + tid] += (Rr * v * v * r2r + Ri * v * v * r2i) * iw;
            acc[(1 + nbath + k) * nt + tid] += (Rr * 2.0 * v * re + Ri * 2.0 * v * im) * iw;
        }
    }
    __syncthreads();
    for (int q = tid; q < na; q += nt) {
        CSum s;
        s.zero();
        for (int t = 0; t < nt; t++) s.add(acc[q * nt + t]);
        const double val = s.value();
        if (q == 0) chi2[b] = val;
        else if (grad) grad[(int64_t)b * 2 * nbath + (q - 1)] = -2.0 * val;
    }
}

template <int NB = 1>
static bool launch_chi2_reg(dmfted_ctx *c, int nbatch, int nbath, int L, const double *a,
                            const double *x, const double *g, const double *w, double *chi2,
                            double *grad) {
    if constexpr (NB > kChi2Levels) {
        return false;
    } else {
        if (nbath != NB) return launch_chi2_reg<NB + 1>(c, nbatch, nbath, L, a, x, g, w, chi2, grad);
        k_chi2_reg<NB><<<nbatch, kChi2Threads, 0, c->stream>>>(L, a, x, g, w, chi2, grad);
        return true;
    }
}

void chi2_batch_device(dmfted_ctx *c, int nbatch, int nbath, int L, const double *a,
                       const double *x, const double *g, const double *w, double *chi2,
                       double *grad) {
    DM_REQUIRE(nbatch > 0 && nbath > 0 && L > 0, DMFTED_ERR_ARG, "chi2: empty batch or grid");
    if (!launch_chi2_reg(c, nbatch, nbath, L, a, x, g, w, chi2, grad)) {
        int nt = 128;
        auto bytes = [&](int t) {
            return (size_t)(2 * nbath + (1 + 2 * nbath) * t + 2 * nbath * t) * 8;
        };
        while (nt > 32 && bytes(nt) > 160 * 1024) nt /= 2;
        DM_REQUIRE(bytes(nt) <= 200 * 1024, DMFTED_ERR_UNSUPPORTED, "chi2: too many bath levels");
        // the attribute belongs to the device current when it is set: once per device
        static bool attr[64] = {false};
        if (!attr[c->device & 63]) {
            DM_CUDA(cudaFuncSetAttribute(k_chi2, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         200 * 1024));
            attr[c->device & 63] = true;
        }
        k_chi2<<<nbatch, nt, bytes(nt), c->stream>>>(nbath, L, a, x, g, w, chi2, grad);
    }
    DM_CHECK_LAUNCH();
    c->launches++;
}

}  // namespace dmfted
