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
// iteration from the single-precision one, to the last bit of the division that
// it replaces, without a branch between the NB chains.  The sums are folded
// compensated, one warp per sum, in a fixed order.  What bounds it: the FP64
// pipe's latency at four or five CTAs per SM.  4096 sets of 9 levels, 1000
// points: 72 us against 133 us with the sums in shared memory and divisions; the
// 20 FP64 operations per level and point are 42 us of the pipe.  Largest errors
// against 64-bit references over 24 inputs, of the norm: chi^2 2.9e-16 (3.5e-16
// before), gradient 3.49e-16 (3.53e-16); means 2.07e-16 (2.04e-16) and 2.30e-16
// (2.22e-16).  Every accumulation is one rounded product sum and one addition: a
// gradient term folded in by two chained fma is 2 us faster, with errors of 3.53e-16
// and 2.33e-16.
#include <algorithm>

#include "internal.cuh"
#include "reduce.cuh"

namespace dmfted {

// Registers hold 3 NB + 1 FP64 values: the CTAs per SM that leave no or few
// spills (9 levels: 69 us with four, 77 us with five).
constexpr int kChi2Levels = 16;
constexpr int kChi2Threads = 128;

// 1/d: Newton iteration from the approximate single-precision reciprocal, whose
// argument and result change format by integer shifts of the bit pattern (the
// conversion instructions share the FP64 pipe's slow path).  Each of the two
// steps doubles the 22 bits of the start; the last one leaves its own rounding.
// For d within about 1e-29 .. 1e29, where the shifts hold (chi2_in_range).
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
__global__ void __launch_bounds__(kChi2Threads, NB <= 4 ? 6 : NB <= 8 ? 5 : NB <= 12 ? 4 : 3)
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
            const double t = pv2[k] * inv[k];
            dre = fma(pe[k], t, dre);
            dim += t;
        }
        const double Rr = gn.x + dre, Ri = fma(om, dim, gn.y);
        const double Wr = Rr * iw, Wi = Ri * iw;
        s0 = fma(Rr, Wr, fma(Ri, Wi, s0));
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
