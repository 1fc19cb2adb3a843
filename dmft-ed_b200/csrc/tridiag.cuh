// Device routines on the Lanczos tridiagonal T_n (diagonal a[0..n),
// off-diagonal b[1..n)) shared by the grid-wide and the batched solvers:
// Sturm-sequence multisection for eigenvalues, inverse iteration for
// eigenvectors, the ARPACK-style Ritz test on the lowest m pairs, and the
// seeded random start vector.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

namespace dmfted {

// (seed, i) -> uniform (0, 1]: splitmix64 of the element index, the real
// counterpart of the seeded random resid the reference hands ARPACK
// (.repo/ARPACK_LANCZOS.f90:394-403).
__device__ __forceinline__ double random_start_value(int64_t i, uint64_t seed) {
    uint64_t z = seed + 0x9E3779B97F4A7C15ull * (uint64_t)(i + 1);
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    z = z ^ (z >> 31);
    return ((double)(z >> 11) + 1.0) * (1.0 / 9007199254740992.0);
}

// Sturm count: number of eigenvalues of the n x n tridiagonal (a, b[1..n-1])
// below x, by the pivots of T - x.
__device__ inline int sturm_count(const double *a, const double *b, int n, double x, double pivmin) {
    int cnt = 0;
    double q = a[0] - x;
    if (fabs(q) < pivmin) q = -pivmin;
    if (q < 0.0) cnt++;
    for (int i = 1; i < n; i++) {
        q = (a[i] - x) - b[i] * b[i] / q;
        if (fabs(q) < pivmin) q = -pivmin;
        if (q < 0.0) cnt++;
    }
    return cnt;
}

// Sturm count: number of eigenvalues of the n x n tridiagonal (a, b[1..n-1])
// below x, as sign changes of the leading principal minors
//   p_i = (a_i - x) p_{i-1} - b_i^2 p_{i-2},
// a zero pivot ratio |p_i / p_{i-1}| < pivmin counting as a negative one.  The
// minors are rescaled by a power of two every eight steps, and T, x and pivmin are
// multiplied by s, a power of two too (tridiag_scale): eight pivots, even all at
// pivmin, then stay within the range of FP64 at every energy unit (unscaled,
// eight steps of |T| = 1e-38 underflow to a wrong count).  SCALED = false: s = 1.
// Two FP64 operations, a compare and a select per step (45 cycles) against the
// 320 of the division in sturm_count; the two agree unless x is within rounding
// of an eigenvalue.
template <bool SCALED>
__device__ inline int sturm_count_minors(const double *a, const double *b, int n, double x,
                                         double pivmin, double s) {
    if (SCALED) pivmin *= s;
    double pp = 1.0, p = SCALED ? (a[0] - x) * s : a[0] - x;
    if (fabs(p) < pivmin) p = -pivmin;
    int cnt = p < 0.0 ? 1 : 0;
    auto step = [&](double ai, double bi) {
        double q = ai * p - (bi * bi) * pp;
        if (fabs(q) < pivmin * fabs(p)) q = -pivmin * p;
        pp = p;
        p = q;
        cnt += (unsigned)(__double2hiint(p) ^ __double2hiint(pp)) >> 31;
    };
    int i = 1;
    for (; i + 8 <= n; i += 8) {
        double a8[8], b8[8];  // the operands ahead of the chain
#pragma unroll
        for (int q = 0; q < 8; q++) {
            a8[q] = SCALED ? (a[i + q] - x) * s : a[i + q] - x;
            b8[q] = SCALED ? b[i + q] * s : b[i + q];
        }
#pragma unroll
        for (int q = 0; q < 8; q++) step(a8[q], b8[q]);
        const int e = max((__double2hiint(p) >> 20) & 0x7ff, (__double2hiint(pp) >> 20) & 0x7ff);
        if (e > 0 && e < 2046) {
            const double f = __hiloint2double((2046 - e) << 20, 0);
            p *= f;
            pp *= f;
        }
    }
    for (; i < n; i++) {
        if (SCALED) step((a[i] - x) * s, b[i] * s);
        else step(a[i] - x, b[i]);
    }
    return cnt;
}
__device__ inline int sturm_count_fast(const double *a, const double *b, int n, double x,
                                       double pivmin, double s) {
    return s == 1.0 ? sturm_count_minors<false>(a, b, n, x, pivmin, s)
                    : sturm_count_minors<true>(a, b, n, x, pivmin, s);
}

// The power of two s with 1 <= amax * s < 2; 1 where nine pivots at pivmin =
// 4.8e-32 amax^2 (3e-33 each at 0.25) or of 4 amax stay within the range unscaled.
__device__ inline double tridiag_scale(double amax) {
    if (amax >= 0.25 && amax <= 1e18) return 1.0;
    const int e = min(max((__double2hiint(amax) >> 20) & 0x7ff, 1), 2045);
    return __hiloint2double((2046 - e) << 20, 0);
}

// Bracket width, relative to |T|, above which the counts of a multisection use
// sturm_count_fast: its points are then far from the eigenvalue, both forms
// count alike, and the last rounds with sturm_count give the same digits.
constexpr double kFastBracket = 1e-9;

// j-th lowest eigenvalue (0-based) of T_n by multisection with all threads of
// the block; a, b in shared memory.  Returns the value in every thread.  EXACT:
// to the last digit of sturm_count; else to its rounding.
template <bool EXACT>
__device__ inline double tridiag_eig(const double *a, const double *b, int n, int j) {
    __shared__ int first[2];
    double lo = a[0], hi = a[0], amax = 0.0;  // Gershgorin bounds, every thread
    for (int i = 0; i < n; i++) {
        const double r = (i > 0 ? fabs(b[i]) : 0.0) + (i + 1 < n ? fabs(b[i + 1]) : 0.0);
        lo = fmin(lo, a[i] - r);
        hi = fmax(hi, a[i] + r);
        amax = fmax(amax, fabs(a[i]) + r);
    }
    const double pad = 2.2e-16 * fmax(amax, 1e-300) * 4.0 + 1e-300;
    lo -= pad;
    hi += pad;
    amax = fmax(fabs(lo), fabs(hi));
    const double pivmin = 1e-300 + 2.2e-16 * 2.2e-16 * fmax(amax * amax, 1e-300);
    const double s = tridiag_scale(amax);
    const int nt = blockDim.x;
    if (threadIdx.x < 2) first[threadIdx.x] = nt;
    __syncthreads();
    for (int round = 0; round < 40; round++) {
        if (hi - lo <= 2.0 * 2.2e-16 * fmax(fabs(lo), fabs(hi)) + 1e-300) break;
        const double x = lo + (hi - lo) * (double)(threadIdx.x + 1) / (double)(nt + 1);
        const int c = !EXACT || hi - lo > kFastBracket * amax
                          ? sturm_count_fast(a, b, n, x, pivmin, s)
                          : sturm_count(a, b, n, x, pivmin);
        // first point whose count exceeds j
        int *f = &first[round & 1];
        if (c > j) atomicMin(f, (int)threadIdx.x);
        __syncthreads();
        const int t = *f;
        if (threadIdx.x == 0) first[(round + 1) & 1] = nt;
        __syncthreads();
        const double nlo = t == 0 ? lo : lo + (hi - lo) * (double)t / (double)(nt + 1);
        const double nhi = t == nt ? hi : lo + (hi - lo) * (double)(t + 1) / (double)(nt + 1);
        lo = nlo;
        hi = nhi;
    }
    return 0.5 * (lo + hi);
}

// Eigenvector y of T_n (diag a[0..n), off-diagonal b[1..n)) for eigenvalue
// lam: three steps of inverse iteration, Gaussian elimination with partial
// pivoting on the tridiagonal.  Single thread.  ws: 5n doubles, sw: n bytes.
// nprev > 0: lam belongs to a cluster of eigenvalues (several copies of an
// eigenvalue, as a Lanczos run past rounding-level growth of a degenerate
// partner holds them) and prev[q*n..] (q < nprev) are the eigenvectors of
// the cluster's lower members.  Inverse iteration alone would return the same
// vector for every member; as in LAPACK's dstein, the iteration then starts
// from a pseudo-random vector (seed: the member's index) and is
// re-orthogonalised against the lower members after every solve, which
// converges to an orthonormal basis of the cluster's invariant subspace.
__device__ inline void tridiag_evec(const double *a, const double *b, int n, double lam, double *yv,
                             double *ws, unsigned char *sw, const double *prev = nullptr,
                             int nprev = 0) {
    double *D = ws, *U1 = ws + n, *U2 = ws + 2 * n, *M = ws + 3 * n;
    double nrm = 0.0;
    for (int i = 0; i < n; i++) nrm = fmax(nrm, fabs(a[i] - lam) + (i > 0 ? fabs(b[i]) : 0.0));
    // the replacement of a zero pivot; T - lam = 0 (a 1 x 1 sector, or lam I)
    // has no scale of its own, and 1e-15 keeps 1/tiny and the squares of the
    // solve finite
    const double tiny = (nrm > 1e-290 ? nrm : 1.0) * 1e-15;
    double d = a[0] - lam, u1 = n > 1 ? b[1] : 0.0, u2 = 0.0;
    for (int i = 0; i < n - 1; i++) {
        const double l = b[i + 1], dn = a[i + 1] - lam, un = (i + 2 < n) ? b[i + 2] : 0.0;
        if (fabs(d) >= fabs(l)) {
            if (d == 0.0) d = tiny;
            const double m = l / d;
            D[i] = d; U1[i] = u1; U2[i] = u2; M[i] = m; sw[i] = 0;
            d = dn - m * u1;
            u1 = un - m * u2;
            u2 = 0.0;
        } else {
            const double m = d / l;
            D[i] = l; U1[i] = dn; U2[i] = un; M[i] = m; sw[i] = 1;
            d = u1 - m * dn;
            u1 = u2 - m * un;
            u2 = 0.0;
        }
    }
    if (d == 0.0) d = tiny;
    D[n - 1] = d;
    // reciprocal pivots: independent divisions here, multiplications on the
    // serial back substitutions below
    for (int i = 0; i < n; i++) D[i] = 1.0 / D[i];
    if (nprev > 0)
        for (int i = 0; i < n; i++) yv[i] = random_start_value(i, 977ull + 131ull * (uint64_t)nprev) - 0.5;
    else
        for (int i = 0; i < n; i++) yv[i] = 1.0 / sqrt((double)n);
    const int iters = nprev > 0 ? 5 : 3;
    for (int it = 0; it < iters; it++) {
        for (int i = 0; i < n - 1; i++) {
            if (sw[i]) {
                const double t = yv[i];
                yv[i] = yv[i + 1];
                yv[i + 1] = t;
            }
            yv[i + 1] -= M[i] * yv[i];
        }
        yv[n - 1] *= D[n - 1];
        if (n > 1) yv[n - 2] = (yv[n - 2] - U1[n - 2] * yv[n - 1]) * D[n - 2];
        for (int i = n - 3; i >= 0; i--) yv[i] = (yv[i] - U1[i] * yv[i + 1] - U2[i] * yv[i + 2]) * D[i];
        for (int rep = 0; rep < 2 && nprev > 0; rep++)
            for (int q = 0; q < nprev; q++) {
                const double *pq = prev + (int64_t)q * n;
                double d = 0.0;
                for (int i = 0; i < n; i++) d += pq[i] * yv[i];
                for (int i = 0; i < n; i++) yv[i] -= d * pq[i];
            }
        double ss = 0.0;
        for (int i = 0; i < n; i++) ss += yv[i] * yv[i];
        ss = 1.0 / sqrt(ss);
        for (int i = 0; i < n; i++) yv[i] *= ss;
    }
    const double sg = yv[0] < 0.0 ? -1.0 : 1.0;  // deterministic sign
    for (int i = 0; i < n; i++) yv[i] *= sg;
}

// Sum over the warp, in every lane (a fixed tree).
__device__ __forceinline__ double warp_sum(double d) {
    for (int o = 16; o > 0; o >>= 1) d += __shfl_xor_sync(0xffffffffu, d, o);
    return d;
}

// 1/d to the last bit or two: Newton-Raphson from the single-precision
// reciprocal (each of the two steps doubles its 23 bits).  The pivots of an
// inverse iteration need no more, and the chain of one full FP64 division per
// step was most of its time (320 cycles each).
__device__ __forceinline__ double newton_recip(double d) {
    const double m = fabs(d);
    if (!(m > 1e-30 && m < 1e30)) return 1.0 / d;
    double y = (double)(1.0f / (float)d);
    y = fma(y, fma(-d, y, 1.0), y);
    return fma(y, fma(-d, y, 1.0), y);
}

// The same for the residual tests, which need the last component to a few
// digits: called by a whole warp, lane 0 runs the serial chains with one Newton
// reciprocal per pivot, all lanes the sums.  yv, ws (4n doubles), sw (n bytes):
// memory all lanes see.
__device__ inline void tridiag_evec_fast(const double *a, const double *b, int n, double lam, double *yv,
                             double *ws, unsigned char *sw, const double *prev = nullptr,
                             int nprev = 0) {
    double *D = ws, *U1 = ws + n, *U2 = ws + 2 * n, *M = ws + 3 * n;
    const double y00 = 1.0 / sqrt((double)n);
    const int lane = threadIdx.x & 31;
    double nrm = 0.0;
    for (int i = lane; i < n; i += 32) nrm = fmax(nrm, fabs(a[i] - lam) + (i > 0 ? fabs(b[i]) : 0.0));
    for (int o = 16; o > 0; o >>= 1) nrm = fmax(nrm, __shfl_xor_sync(0xffffffffu, nrm, o));
    // the replacement of a zero pivot; T - lam = 0 (a 1 x 1 sector, or lam I)
    // has no scale of its own, and 1e-15 keeps 1/tiny and the squares of the
    // solve finite
    const double tiny = (nrm > 1e-290 ? nrm : 1.0) * 1e-15;
    // Each pivot's reciprocal is the one division of its step (the multiplier
    // is a product with it), and the back substitutions below multiply by it.
    double d = a[0] - lam, u1 = n > 1 ? b[1] : 0.0, u2 = 0.0;
    double an = n > 1 ? a[1] : 0.0, bn = n > 2 ? b[2] : 0.0;  // a_{i+1}, b_{i+2}, loaded ahead
    double l = u1;
    for (int i = 0; i < n - 1 && lane == 0; i++) {
        const double dn = an - lam, un = bn;
        an = i + 2 < n ? a[i + 2] : 0.0;
        bn = i + 3 < n ? b[i + 3] : 0.0;
        if (fabs(d) >= fabs(l)) {
            if (d == 0.0) d = tiny;
            const double r = newton_recip(d), m = l * r;
            D[i] = r; U1[i] = u1; U2[i] = u2; M[i] = m; sw[i] = 0;
            d = dn - m * u1;
            u1 = un - m * u2;
            u2 = 0.0;
        } else {
            const double r = newton_recip(l), m = d * r;
            D[i] = r; U1[i] = dn; U2[i] = un; M[i] = m; sw[i] = 1;
            d = u1 - m * dn;
            u1 = u2 - m * un;
            u2 = 0.0;
        }
        l = un;
    }
    if (lane == 0) {
        if (d == 0.0) d = tiny;
        D[n - 1] = 1.0 / d;
    }
    if (nprev > 0)
        for (int i = lane; i < n; i += 32) yv[i] = random_start_value(i, 977ull + 131ull * (uint64_t)nprev) - 0.5;
    else
        for (int i = lane; i < n; i += 32) yv[i] = y00;
    __syncwarp();
    const int iters = nprev > 0 ? 5 : 3;
    for (int it = 0; it < iters; it++) {
        // forward and back substitution with the running elements in
        // registers and four steps' operands loaded ahead of the chain (the
        // stores to yv would otherwise keep every load behind them)
        double cur = yv[0];
        for (int i0 = 0; i0 < n - 1 && lane == 0; i0 += 4) {
            double y4[4], m4[4];
            unsigned char s4[4];
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const int i = min(i0 + q, n - 2);
                y4[q] = yv[i + 1];
                m4[q] = M[i];
                s4[q] = sw[i];
            }
#pragma unroll
            for (int q = 0; q < 4; q++)
                if (i0 + q < n - 1) {
                    const double keep = s4[q] ? y4[q] : cur, next = s4[q] ? cur : y4[q];
                    yv[i0 + q] = keep;
                    cur = next - m4[q] * keep;
                }
        }
        double y1 = 0.0, y2 = 0.0;
        if (lane == 0) {
            y1 = cur * D[n - 1];
            yv[n - 1] = y1;
        }
        for (int i0 = n - 2; i0 >= 0 && lane == 0; i0 -= 4) {
            double y4[4], u4[4], w4[4], d4[4];
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const int i = max(i0 - q, 0);
                y4[q] = yv[i];
                u4[q] = U1[i];
                w4[q] = U2[i];
                d4[q] = D[i];
            }
#pragma unroll
            for (int q = 0; q < 4; q++)
                if (i0 - q >= 0) {
                    const double t = (y4[q] - w4[q] * y2) - u4[q] * y1;
                    y2 = y1;
                    y1 = t * d4[q];
                    yv[i0 - q] = y1;
                }
        }
        __syncwarp();
        for (int rep = 0; rep < 2 && nprev > 0; rep++)
            for (int q = 0; q < nprev; q++) {
                const double *pq = prev + (int64_t)q * n;
                double d = 0.0;
                for (int i = lane; i < n; i += 32) d += pq[i] * yv[i];
                d = warp_sum(d);
                for (int i = lane; i < n; i += 32) yv[i] -= d * pq[i];
            }
        double ss = 0.0;
        for (int i = lane; i < n; i += 32) ss += yv[i] * yv[i];
        ss = 1.0 / sqrt(warp_sum(ss));
        for (int i = lane; i < n; i += 32) yv[i] *= ss;
        __syncwarp();
    }
    const double sg = yv[0] < 0.0 ? -1.0 : 1.0;  // deterministic sign
    __syncwarp();
    for (int i = lane; i < n; i += 32) yv[i] *= sg;
    __syncwarp();
}

// Lowest m eigenvalues of T_n, one warp per eigenvalue (warp w takes j = w,
// w + nwarps, ...), all warps at once: multisection on 32 points per round,
// the new bracket between the last lane whose Sturm count is at most j and the
// next (a ballot, no block barrier).  Sturm counts are latency-bound chains,
// so 32 points per eigenvalue in parallel cost far less than the whole block
// on one eigenvalue after another.  a, b in shared memory; lane 0 writes
// evals[j]; the caller synchronises the block before reading them.
template <bool EXACT>
__device__ inline void tridiag_eigs_warp(const double *a, const double *b, int n, int m,
                                         double *evals) {
    const int lane = threadIdx.x & 31, nw = (int)(blockDim.x >> 5);
    double lo = INFINITY, hi = -INFINITY, amax = 0.0;
    for (int i = lane; i < n; i += 32) {
        const double r = (i > 0 ? fabs(b[i]) : 0.0) + (i + 1 < n ? fabs(b[i + 1]) : 0.0);
        lo = fmin(lo, a[i] - r);
        hi = fmax(hi, a[i] + r);
        amax = fmax(amax, fabs(a[i]) + r);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        lo = fmin(lo, __shfl_xor_sync(0xffffffffu, lo, o));
        hi = fmax(hi, __shfl_xor_sync(0xffffffffu, hi, o));
        amax = fmax(amax, __shfl_xor_sync(0xffffffffu, amax, o));
    }
    const double pad = 2.2e-16 * fmax(amax, 1e-300) * 4.0 + 1e-300;
    lo -= pad;
    hi += pad;
    const double am = fmax(fabs(lo), fabs(hi));
    const double pivmin = 1e-300 + 2.2e-16 * 2.2e-16 * fmax(am * am, 1e-300);
    const double scale = tridiag_scale(am);
    for (int j = (int)(threadIdx.x >> 5); j < m; j += nw) {
        double l = lo, h = hi;
        for (int round = 0; round < 96; round++) {
            if (h - l <= 2.0 * 2.2e-16 * fmax(fabs(l), fabs(h)) + 1e-300) break;
            const double x = l + (h - l) * (double)(lane + 1) / 33.0;
            const int c = !EXACT || h - l > kFastBracket * am
                              ? sturm_count_fast(a, b, n, x, pivmin, scale)
                              : sturm_count(a, b, n, x, pivmin);
            const unsigned below = __ballot_sync(0xffffffffu, c <= j);
            const int t = below == 0xffffffffu ? 32 : __ffs(~below) - 1;
            const double nl = t == 0 ? l : l + (h - l) * (double)t / 33.0;
            const double nh = t == 32 ? h : l + (h - l) * (double)(t + 1) / 33.0;
            l = nl;
            h = nh;
        }
        if (lane == 0) evals[j] = 0.5 * (l + h);
    }
}

// Dynamic shared memory of the two Ritz kernels for n steps.
__host__ __device__ inline size_t ritz_smem(int n) { return (size_t)8 * n * sizeof(double) + n + 16; }

// Doubles of one eigenvector work space of ritz_multi_dev (vector, the four
// factor arrays of tridiag_evec, its pivot flags).
__host__ __device__ inline int ritz_evec_doubles(int n) { return 5 * n + (n + 7) / 8 + 1; }

// Lowest min(mwant, n) Ritz pairs of T_n with all threads of the block: a, b
// in shared memory, work = work_cap doubles of shared memory after them (at
// least ritz_evec_doubles(n)).  evals[j], Y[j*n + i] (eigenvector j, first
// component positive, re-orthogonalised against the lower ones in the small
// space) and the Ritz estimate est[j] = b_n |Y[j*n + n-1]|.  Returns, in every
// thread, whether every estimate passes ARPACK's test est <= tol *
// max(eps^(2/3), |theta|).  EXACT: the pairs a result is made of; else the test
// alone, with the division-free counts and Newton reciprocals (n = 100, six
// pairs: 290 against 640 thousand cycles).  The eigenvalues are found one warp each; the
// inverse iterations run on lane 0 of as many warps as work spaces fit in
// work; the re-orthogonalisation, in order of j, on thread 0.
template <bool EXACT>
__device__ inline bool ritz_multi_dev(const double *sa, const double *sb, int n, int mwant,
                                      double tol, double bn, double *evals, double *Y, double *est,
                                      double *work, int work_cap) {
    __shared__ int okflag;
    if (threadIdx.x == 0) okflag = 1;
    const int m = min(mwant, n);
    tridiag_eigs_warp<EXACT>(sa, sb, n, m, evals);
    __syncthreads();
    const int per = ritz_evec_doubles(n);
    const int lanes = max(1, min(min(m, work_cap / per), (int)(blockDim.x >> 5)));
    const int w = (int)(threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if ((lane == 0 || !EXACT) && w < lanes) {
        double *yv = work + (size_t)w * per, *ws = yv + n;
        unsigned char *sw = reinterpret_cast<unsigned char *>(ws + 4 * n);
        // clusters: consecutive eigenvalues closer than 1e-3 |T| (dstein's
        // ORTOL); lane w takes clusters w, w + lanes, ..., each member in turn
        double tn = 0.0;
        for (int i = 0; i < n; i++)
            tn = fmax(tn, fabs(sa[i]) + (i > 0 ? fabs(sb[i]) : 0.0) + (i + 1 < n ? fabs(sb[i + 1]) : 0.0));
        const double ortol = 1e-3 * tn;
        int g = -1;
        for (int j = 0, head = 0; j < m; j++) {
            if (j == 0 || evals[j] - evals[j - 1] > ortol) {
                head = j;
                g++;
            }
            if (g % lanes != w) continue;
            if constexpr (EXACT) {
                tridiag_evec(sa, sb, n, evals[j], yv, ws, sw, Y + (int64_t)head * n, j - head);
                for (int i = 0; i < n; i++) Y[(int64_t)j * n + i] = yv[i];
            } else {
                tridiag_evec_fast(sa, sb, n, evals[j], yv, ws, sw, Y + (int64_t)head * n, j - head);
                for (int i = lane; i < n; i += 32) Y[(int64_t)j * n + i] = yv[i];
                __syncwarp();
            }
        }
    }
    __syncthreads();
    const double eps23 = 3.666852862501036e-11;
    if (!EXACT && threadIdx.x < 32) {
        for (int j = 0; j < m; j++) {
            double *yj = Y + (int64_t)j * n;
            for (int q = 0; q < j; q++) {
                const double *yq = Y + (int64_t)q * n;
                double d = 0.0;
                for (int i = lane; i < n; i += 32) d += yq[i] * yj[i];
                d = warp_sum(d);
                for (int i = lane; i < n; i += 32) yj[i] -= d * yq[i];
            }
            double nr = 0.0;
            for (int i = lane; i < n; i += 32) nr += yj[i] * yj[i];
            nr = sqrt(warp_sum(nr));
            for (int i = lane; i < n; i += 32) yj[i] /= nr;
            __syncwarp();
            if (lane == 0) {
                est[j] = fabs(bn) * fabs(yj[n - 1]);
                if (!(est[j] <= tol * fmax(eps23, fabs(evals[j])))) okflag = 0;
            }
        }
    }
    if (EXACT && threadIdx.x == 0) {
        for (int j = 0; j < m; j++) {
            double *yj = Y + (int64_t)j * n;
            // orthogonalise against the lower eigenvectors (close eigenvalues)
            for (int q = 0; q < j; q++) {
                double d = 0.0;
                for (int i = 0; i < n; i++) d += Y[(int64_t)q * n + i] * yj[i];
                for (int i = 0; i < n; i++) yj[i] -= d * Y[(int64_t)q * n + i];
            }
            double nr = 0.0;
            for (int i = 0; i < n; i++) nr += yj[i] * yj[i];
            nr = 1.0 / sqrt(nr);
            const double sg = yj[0] < 0.0 ? -nr : nr;
            for (int i = 0; i < n; i++) yj[i] *= sg;
            est[j] = fabs(bn) * fabs(yj[n - 1]);
            if (!(est[j] <= tol * fmax(eps23, fabs(evals[j])))) okflag = 0;
        }
    }
    __syncthreads();
    const bool ok = okflag != 0;
    __syncthreads();
    return ok;
}

}  // namespace dmfted
