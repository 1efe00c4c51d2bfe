// Augmented analytic kludge (AAK) waveform: the harmonic sum of the AAK model
// over a sparse trajectory.
//
// Reference: AAKSummation.sum (src/few/summation/aakwave.py:35-196) and its
// kernel make_waveform / get_waveform (src/few/cutils/gpuAAK.cu:181-578,
// geometry d_RotCoeff :141-177).  Per output sample t = i dt, on the
// trajectory segment holding it: e, Y = cos(iota), Phi_phi, Phi_theta, Phi_r
// and the three frequencies from the 8-term dense-output basis; the orbit
// orientation (L), the spin (S) and the line of sight give the polarisation
// rotation and the precession angle gamma; the optional long-wavelength LISA
// response (mich); then the sum over harmonics n = 1..nmodes of the Peters &
// Mathews amplitudes with J_{n-2..n+2}(n e), rotated and projected.  The
// sample is (hI, -hII).
//
// B200 layout: one launch over all samples (the reference launches one kernel
// per trajectory segment); a thread finds its samples' segments by bisection over
// the segments' first samples.
//   * Amplitudes.  The three Bessel combinations of a harmonic depend on e alone,
//     and e hardly moves over the few hundred samples of a CTA: they are computed
//     at 6, 8 or 12 Chebyshev nodes of the CTA's own range of e (the fewest whose
//     truncation error stays below 1e-17) and evaluated as polynomials there.
//     At a node the five Bessel values of a harmonic come from one backward
//     (Miller) recurrence normalised by J_0 + 2 sum J_2k = 1, moved to the node's
//     exact argument.  Where e moves too far for 12 nodes, every sample runs the
//     recurrence.  Rounding: against long double on a CPU, over e = 0.2-0.65 and
//     up to 40 harmonics, the strong harmonics (above 1e-3) are off by 2.8, 3.7
//     and 3.7e-16 of their largest value (rms; at most 1.7, 2.6 and 2.6e-15) with
//     6, 8 and 12 nodes; by the recurrence alone 4.6, 4.5 and 5.0e-16 (3.2, 3.3
//     and 4.8e-15) over the same ranges.
//   * Phases.  e^{i n Phi} by a running product of e^{i Phi}; the reference rounds
//     n Phi (+ Doppler), at phases of ~1e7 rad, and that rounding is part of the
//     result: its exact error eps (|eps| < 4e-9) comes from error-free
//     transformations and enters as the factor 1 - i eps.
//   * The three sums over harmonics leave the orientation, the polarisation
//     rotation and the response to be applied once per sample.
// FP64 throughout.
#include <cuda_runtime.h>

#include <cmath>
#include <vector>

#include "few_common.cuh"
#include "few_internal.h"

namespace few {
namespace aak {

constexpr double kPi = 3.141592653589793238462643383279502884;
constexpr double kMTSUN = 4.9254909491978065e-06;      // solar mass in s (global.h:24)
constexpr double kGPCINSEC = 1.02927125054339e+17;     // Gpc in s (global.h:26)
constexpr double kAUsec = 499.00478383615643;          // AU in s (global.h:27)
constexpr double kYRSID = 31558149.763545595;          // sidereal year in s (global.h:23)

// J_{n-2}(x) .. J_{n+2}(x) into J[0..4] for n >= 1, x >= 0 (J_{-1} = -J_1), by
// Miller's backward recurrence b_{k-1} = (2k/x) b_k - b_{k+1} from a start
// index M = top + 16 + sqrt(30 top) above top = max(n + 2, x), normalised by
// b_0 + 2 (b_2 + b_4 + ...).  The start's relative error is of order
// (x/2)^{2M} / (M! (M-1)!): below 1e-38 for every x <= top <= 64.
__device__ void bessel_band(int n, double x, double J[5]) {
    if (x == 0.0) {
#pragma unroll
        for (int q = 0; q < 5; ++q) J[q] = (n - 2 + q == 0) ? 1.0 : 0.0;
        return;
    }
    const int top = n + 2 > (int)x ? n + 2 : (int)x;
    int M = top + 16 + (int)sqrt(30.0 * top);
    M += M & 1;  // even start
    const double tox = 2.0 / x;
    double bp = 0.0, b = 1.0, sum = 0.0;
    double Jm1 = 0.0;  // b_1, for J_{-1} = -J_1
    double got[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
    for (int k = M; k >= 1; --k) {
        // b holds b_k, bp holds b_{k+1}; constant indices keep got[] in registers
#pragma unroll
        for (int q = 0; q < 5; ++q)
            if (k == n - 2 + q) got[q] = b;
        if ((k & 1) == 0) sum += b;
        double bm = k * tox * b - bp;  // b_{k-1}
        bp = b;
        b = bm;
        if (fabs(b) > 1e250) {  // rescale everything carried
            b *= 1e-250;
            bp *= 1e-250;
            sum *= 1e-250;
#pragma unroll
            for (int q = 0; q < 5; ++q) got[q] *= 1e-250;
        }
    }
    // b = b_0, bp = b_1
    Jm1 = bp;
#pragma unroll
    for (int q = 0; q < 5; ++q)
        if (n - 2 + q == 0) got[q] = b;  // k = 0 lies in the band when n <= 2
    const double norm = b + 2.0 * sum;
#pragma unroll
    for (int q = 0; q < 5; ++q) J[q] = got[q] / norm;
    if (n == 1) J[0] = -Jm1 / norm;  // J_{-1} = -J_1
}

// bessel_band for two harmonics at once (n and n + 1 at x1 = n e and x2 =
// (n + 1) e): one recurrence loop from a common start index (the larger one,
// which only adds accuracy to the other), two independent chains for the
// scheduler to interleave.  The loop runs in three phases so that only the six
// steps inside the bands capture values (with constant indices, so the bands
// stay in registers).
// One recurrence step of both chains at index k.  EVEN: k is even (b_k joins
// the normalisation sum); CHECK: test for overflow after the step (every
// other step suffices: two steps grow the values by less than 1e58 for any
// argument the kernel sees).
template <bool EVEN, bool CHECK>
__device__ __forceinline__ void miller_step(double kf, double t1, double t2, double &b1, double &bp1, double &s1,
                                            double &b2, double &bp2, double &s2, double g1[5], double g2[5]) {
    if (EVEN) {
        s1 += b1;
        s2 += b2;
    }
    const double m1 = kf * t1 * b1 - bp1, m2 = kf * t2 * b2 - bp2;
    bp1 = b1; b1 = m1;
    bp2 = b2; b2 = m2;
    if (CHECK) {
        if (fabs(b1) > 1e250) {
            b1 *= 1e-250; bp1 *= 1e-250; s1 *= 1e-250;
#pragma unroll
            for (int q = 0; q < 5; ++q) g1[q] *= 1e-250;
        }
        if (fabs(b2) > 1e250) {
            b2 *= 1e-250; bp2 *= 1e-250; s2 *= 1e-250;
#pragma unroll
            for (int q = 0; q < 5; ++q) g2[q] *= 1e-250;
        }
    }
}

__device__ void bessel_band2(int n, double x1, double x2, double J1[5], double J2[5]) {
    if (x1 == 0.0 || x2 == 0.0) {
        bessel_band(n, x1, J1);
        bessel_band(n + 1, x2, J2);
        return;
    }
    const int top = n + 3 > (int)x2 ? n + 3 : (int)x2;
    int M = top + 16 + (int)sqrt(30.0 * top);
    M += M & 1;
    const double t1 = 2.0 / x1, t2 = 2.0 / x2;
    double bp1 = 0.0, b1 = 1.0, s1 = 0.0, bp2 = 0.0, b2 = 1.0, s2 = 0.0;
    double g1[5] = {0.0, 0.0, 0.0, 0.0, 0.0}, g2[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
    // n is odd and M even: the steps pair up as (even k, odd k) in every phase
    for (int k = M; k > n + 3; k -= 2) {
        miller_step<true, false>((double)k, t1, t2, b1, bp1, s1, b2, bp2, s2, g1, g2);
        miller_step<false, true>((double)(k - 1), t1, t2, b1, bp1, s1, b2, bp2, s2, g1, g2);
    }
    // k = n+3 .. n-2: band 1 holds k = n-2+q (q = 0..4), band 2 holds k = n-1+q;
    // k = n-2+q is even exactly when q is odd
#pragma unroll
    for (int q = 5; q >= 0; --q) {
        const int k = n - 2 + q;
        if (k >= 1) {
            if (q <= 4) g1[q] = b1;
            if (q >= 1) g2[q - 1] = b2;
            if (q & 1) miller_step<true, false>((double)k, t1, t2, b1, bp1, s1, b2, bp2, s2, g1, g2);
            else miller_step<false, true>((double)k, t1, t2, b1, bp1, s1, b2, bp2, s2, g1, g2);
        }
    }
    for (int k = n - 3; k >= 1; k -= 2) {
        miller_step<true, false>((double)k, t1, t2, b1, bp1, s1, b2, bp2, s2, g1, g2);
        miller_step<false, true>((double)(k - 1), t1, t2, b1, bp1, s1, b2, bp2, s2, g1, g2);
    }
    // k = 0 (b = b_0, bp = b_1) lies in band 1 when n <= 2 and in band 2 when n == 1
    if (n == 1) { g1[1] = b1; g2[0] = b2; }
    if (n == 2) g1[0] = b1;
    const double nm1 = b1 + 2.0 * s1, nm2 = b2 + 2.0 * s2;
#pragma unroll
    for (int q = 0; q < 5; ++q) {
        J1[q] = g1[q] / nm1;
        J2[q] = g2[q] / nm2;
    }
    if (n == 1) J1[0] = -bp1 / nm1;  // J_{-1} = -J_1
}

struct AakArgs {
    double2 *wf;
    const double *coef;  // (8, cstride, 6): coefficient c of parameter q on segment j at (c*cstride + j)*6 + q
    const double *t;     // knots
    const int *first;    // (nseg + 1,): segment j writes samples [first[j], first[j+1])
    int nseg, cstride, nmodes, mich;
    double M, S, mu, qS, phiS, qK, phiK, dist, dt;
};

__device__ __forceinline__ double nested(const double *c, double s, double s1) {
    return c[0] + s * (c[1] + s1 * (c[2] + s * (c[3] + s1 * (c[4] + s * (c[5] + s1 * (c[6] + s * c[7]))))));
}

__device__ __forceinline__ double nested_ds(const double *c, double s, double h) {
    const double s2 = s * s, s3 = s * s2, s4 = s * s3, s5 = s * s4, s6 = s * s5;
    return (c[1] + c[2] * (1. - 2. * s) + c[3] * (2. * s - 3. * s2) + c[4] * (2. * s - 6. * s2 + 4. * s3) +
            c[5] * (3. * s2 - 8. * s3 + 5. * s4) + c[6] * (3. * s2 - 12. * s3 + 15 * s4 - 6. * s5) +
            c[7] * (4. * s3 - 15. * s4 + 18. * s5 - 7. * s6)) /
           h;
}

__device__ __forceinline__ void cross3(const double *u, const double *v, double *w) {
    w[0] = u[1] * v[2] - u[2] * v[1];
    w[1] = u[2] * v[0] - u[0] * v[2];
    w[2] = u[0] * v[1] - u[1] * v[0];
}

// ---- Chebyshev interpolation on Q nodes ------------------------------------------
// node[j] = cos((j + 1/2) pi / Q); sum_j d[m][j] f(node_j): the coefficient of T_m of
// the interpolant; t[m][k]: T_m's coefficient of u^k (whole numbers).
//
// The interpolant is evaluated by powers of u, whose true coefficients fall off as
// (n delta)^k / k!, so that Horner's rule loses nothing; the way there must not lose
// anything either: the T_m's coefficients reach 2^(Q-1) and cancel.  So the
// coefficients of T_m are formed from differences to one node's value, and the sums
// over m that turn them into powers of u carry their rounding errors (two-sum and
// two-product): what a node's value is off by then stays a polynomial of that size
// (Chebyshev nodes pass it on by a factor of 2 at most, less than 1 on average).  With
// plain sums 12 nodes are off by up to 3e-13 and 8 by 1e-14.
constexpr double const_cos(double x) {  // Taylor, 0 <= x <= pi
    const bool flip = x > 1.5707963267948966;
    const double r = flip ? kPi - x : x;
    double term = 1.0, sum = 1.0;
    for (int k = 1; k < 16; ++k) {
        term *= -r * r / ((2.0 * k - 1.0) * (2.0 * k));
        sum += term;
    }
    return flip ? -sum : sum;
}

constexpr int kMaxNodes = 12;

struct Cheb {
    double node[kMaxNodes];
    double d[kMaxNodes][kMaxNodes];
    double t[kMaxNodes][kMaxNodes];
};

constexpr Cheb make_cheb(int Q) {
    Cheb t{};
    t.t[0][0] = 1.0;
    t.t[1][1] = 1.0;
    for (int m = 2; m < Q; ++m)
        for (int k = 0; k < Q; ++k) t.t[m][k] = (k > 0 ? 2.0 * t.t[m - 1][k - 1] : 0.0) - t.t[m - 2][k];
    for (int j = 0; j < Q; ++j) {
        t.node[j] = const_cos((j + 0.5) * kPi / Q);
        double c[kMaxNodes] = {};  // T_m(node_j)
        c[0] = 1.0;
        c[1] = t.node[j];
        for (int m = 2; m < Q; ++m) c[m] = 2.0 * t.node[j] * c[m - 1] - c[m - 2];
        for (int m = 0; m < Q; ++m) t.d[m][j] = (m == 0 ? 1.0 : 2.0) / Q * c[m];
    }
    return t;
}

// in global memory: the lanes of a warp read different entries
__device__ const Cheb c_cheb[3] = {make_cheb(6), make_cheb(8), make_cheb(12)};

constexpr int kThreads = 128;
constexpr int kHarm = 24;  // harmonics whose polynomials a CTA holds at a time (even: they come in pairs)

// Values at the nodes, co[row * kMaxNodes + j] -> coefficients of the powers of u, in
// place; by way of cheb[row * (kMaxNodes + 1) + m], the coefficients of T_m, and behind
// them the value that these are relative to.  One barrier inside.
template <int Q>
__device__ __forceinline__ void to_powers(const Cheb &T, int rows, double *co, double *cheb) {
    for (int w = threadIdx.x; w < rows * Q; w += kThreads) {
        const int r = w / Q, m = w - r * Q;
        const double *f = co + r * kMaxNodes;
        const double ref = f[Q / 2];
        double sum = 0.0;
#pragma unroll
        for (int j = 0; j < Q; ++j) sum = fma(T.d[m][j], f[j] - ref, sum);
        cheb[r * (kMaxNodes + 1) + m] = sum;
        if (m == 0) cheb[r * (kMaxNodes + 1) + kMaxNodes] = ref;
    }
    __syncthreads();
    for (int w = threadIdx.x; w < rows * Q; w += kThreads) {
        const int r = w / Q, k = w - r * Q;
        const double *a = cheb + r * (kMaxNodes + 1);
        double hi = 0.0, lo = 0.0;
#pragma unroll
        for (int i = 0; i < Q / 2; ++i) {  // m of k's parity; below k T_m has no u^k
            const int m = 2 * i + (k & 1);
            const double t = T.t[m][k], p = rmul(t, a[m]), sum = radd(hi, p);
            lo += two_sum_err(hi, p, sum) + fma(t, a[m], -p);
            hi = sum;
        }
        co[r * kMaxNodes + k] = radd(hi, lo) + (k == 0 ? a[kMaxNodes] : 0.0);
    }
}

// Largest n * (half width of the e range) for Q nodes: the interpolant of a
// function whose Q-th derivative is at most n^Q errs by at most
// (n delta)^Q / (2^(Q-1) Q!), kept below 1e-17 (of the sum's scale; a harmonic too
// weak to matter is truncated at a larger share of itself).
__device__ __forceinline__ int node_set(double nd) { return nd <= 7.8e-3 ? 0 : (nd <= 0.052 ? 1 : (nd <= 0.38 ? 2 : 3)); }

// The three combinations of harmonic n's Bessel values J_{n-2..n+2}(n e).
__device__ __forceinline__ void combine(int n, double e, const double J[5], double f[3]) {
    f[0] = -n * (J[0] - 2. * e * J[1] + 2. / n * J[2] + 2. * e * J[3] - J[4]);
    f[1] = -n * (J[0] - 2. * J[2] + J[4]);
    f[2] = 2. * J[2];
}

// Bessel values J_{n-2..n+2} that the recurrence gave for x = fl(n e), moved to n e: it
// worked at 2 / fl(2 / x), an n-th power of whose rounding a value of order n carries
// (the largest part of its error).  J_k' = J_{k-1} - k/x J_k = k/x J_k - J_{k+1}.
__device__ __forceinline__ void to_exact_argument(int n, double e, double x, double J[5]) {
    if (x == 0.0) return;
    const double tox = 2.0 / x;
    const double dx = fma(0.5 * fma(tox, x, -2.0), x, fma((double)n, e, -x));
    const double ix = 0.5 * tox;
    double d[5];
    d[0] = (n - 2) * ix * J[0] - J[1];
#pragma unroll
    for (int q = 1; q < 5; ++q) d[q] = J[q - 1] - (n - 2 + q) * ix * J[q];
#pragma unroll
    for (int q = 0; q < 5; ++q) J[q] = fma(dx, d[q], J[q]);
}

// Per-launch angles, once per CTA (one sine and cosine a lane).
struct Sky {
    double sinqS, cosqS, sinqK, cosqK, sinPS, cosPS, sinPK, cosPK, sindP, cosdP;  // dP = phiK - phiS
};

// Sums of one group of harmonics [n0, n0 + count) for the thread's P samples, with
// Q coefficients per function in co[(harmonic * 3 + function) * kMaxNodes + k].
template <int P, bool MICH>
struct Harmonics {
    double u[P], Phi[P];                // position in the CTA's e range, Phi_r
    double2 E[P], Z[P];                 // e^{i Phi} (and the Doppler's share), its running power
    double Sa[P], Sb[P], Sc[P];
    double nu[P], gd[P], W[P];          // Doppler of harmonic n: W (n nu + gd)  (MICH)
    bool large;                         // phases past the first-order rounding factor: sincos for each

    // e^{i nPhi} of harmonic n for sample q, nPhi rounded as the reference rounds it
    __device__ __forceinline__ void phasor(int n, int q, const AakArgs &A, const Sky &K, const double *cosorb,
                                           double &cn, double &sn) const {
        const double dn = (double)n;
        double nPhi, eps;
        if (MICH) {
            const double fn = fma(dn, nu[q], gd[q]);
            const double D = 2. * kPi * fn * kAUsec * K.sinqS * cosorb[q];
            nPhi = fma(dn, Phi[q], D);
            const double p = rmul(dn, Phi[q]), pe = fma(dn, Phi[q], -p);
            const double t = radd(p, D);
            eps = (rsub(t, nPhi) + two_sum_err(p, D, t)) + pe;
        } else {
            nPhi = rmul(dn, Phi[q]);
            eps = fma(dn, Phi[q], -nPhi);
        }
        if (large) {
            sincos_phase(nPhi, &sn, &cn);
        } else {
            cn = fma(Z[q].y, eps, Z[q].x);
            sn = fma(-Z[q].x, eps, Z[q].y);
        }
    }

    template <int Q>
    __device__ __forceinline__ void table(int n0, int count, const double *co, const AakArgs &A, const Sky &K,
                                          const double *cosorb) {
        for (int h = 0; h < count; ++h) {
            const double *c = co + h * 3 * kMaxNodes;
            double f[3][P];
#pragma unroll
            for (int w = 0; w < 3; ++w) {
#pragma unroll
                for (int q = 0; q < P; ++q) f[w][q] = c[w * kMaxNodes + Q - 1];
#pragma unroll
                for (int k = Q - 2; k >= 0; --k) {
                    const double ck = c[w * kMaxNodes + k];
#pragma unroll
                    for (int q = 0; q < P; ++q) f[w][q] = fma(f[w][q], u[q], ck);
                }
            }
#pragma unroll
            for (int q = 0; q < P; ++q) {
                double cn, sn;
                phasor(n0 + h, q, A, K, cosorb, cn, sn);
                Sa[q] = fma(f[0][q], cn, Sa[q]);
                Sb[q] = fma(f[1][q], sn, Sb[q]);
                Sc[q] = fma(f[2][q], cn, Sc[q]);
                Z[q] = cmul(Z[q], E[q]);
            }
        }
    }
};

// Bound by FP64 latency and issue at 16 warps per SM.  One year at dt = 10 s, 18
// harmonics: 0.405 ms (2.02 ms with the nine recurrences, a sincos per harmonic and
// the geometry's angles per sample), with the response 0.605 ms (2.17 ms); 0.39 and
// 0.59 ms with plain sums on the way to powers of u, which lose digits.  A few
// thousand samples of 24 harmonics: 16 us (41 us).
template <int P, bool MICH>
__global__ void __launch_bounds__(kThreads, 4) k_aak(AakArgs A) {
    __shared__ Sky K;
    __shared__ double s_co[kHarm * 3 * kMaxNodes];
    __shared__ double s_cheb[kHarm * 3 * (kMaxNodes + 1)];  // coefficients of T_m; the value they are relative to
    __shared__ double s_min[kThreads / 32], s_max[kThreads / 32];
    const int tid = threadIdx.x, lane = tid & 31;
    const int i0 = A.first[0], i1 = A.first[A.nseg];
    const int chunk = i0 + (int)blockIdx.x * (kThreads * P);
    if (chunk >= i1) return;

    double qS = A.qS, qK = A.qK;
    const double fill = 1e-6;
    if (qS < fill) qS = fill;
    if (qK < fill) qK = fill;
    if (qS > kPi - fill) qS = kPi - fill;
    if (qK > kPi - fill) qK = kPi - fill;
    if (tid < 5) {
        const double ang = tid == 0 ? qS : tid == 1 ? qK : tid == 2 ? A.phiS : tid == 3 ? A.phiK : A.phiK - A.phiS;
        double sn, cs;
        sincos(ang, &sn, &cs);
        double *d = &K.sinqS + 2 * tid;
        d[0] = sn;
        d[1] = cs;
    }

    // segment of each sample: the last j with first[j] <= i
    int seg[P];
    double sa[P], e[P];
    double emin = INFINITY, emax = -INFINITY;
#pragma unroll
    for (int q = 0; q < P; ++q) {
        const int i = min(chunk + tid + q * kThreads, i1 - 1);
        int lo = 0, hi = A.nseg - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (A.first[mid] <= i) lo = mid; else hi = mid - 1;
        }
        seg[q] = lo;
        const double h = A.t[lo + 1] - A.t[lo];
        sa[q] = (A.dt * i - A.t[lo]) / h;
        double c[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) c[k] = A.coef[((long long)k * A.cstride + lo) * 6 + 1];
        e[q] = nested(c, sa[q], 1.0 - sa[q]);
        emin = fmin(emin, e[q]);
        emax = fmax(emax, e[q]);
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        emin = fmin(emin, __shfl_xor_sync(0xffffffffu, emin, off));
        emax = fmax(emax, __shfl_xor_sync(0xffffffffu, emax, off));
    }
    if (lane == 0) {
        s_min[tid >> 5] = emin;
        s_max[tid >> 5] = emax;
    }
    __syncthreads();
#pragma unroll
    for (int w = 0; w < kThreads / 32; ++w) {
        emin = fmin(emin, s_min[w]);
        emax = fmax(emax, s_max[w]);
    }
    const double ec = 0.5 * (emin + emax), delta = fmax(0.5 * (emax - emin), 1e-15);

    Harmonics<P, MICH> H;
    double cosorb[P];
    H.large = false;
#pragma unroll
    for (int q = 0; q < P; ++q) {
        const int j = seg[q];
        const double s = sa[q], s1 = 1.0 - s;
        double c[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) c[k] = A.coef[((long long)k * A.cstride + j) * 6 + 5];
        H.Phi[q] = nested(c, s, s1);
        H.large = H.large || !(fabs(H.Phi[q]) * A.nmodes < 3e7);
        H.u[q] = (e[q] - ec) / delta;
        double sn, cs;
        sincos_phase(H.Phi[q], &sn, &cs);
        H.E[q] = make_double2(cs, sn);
        H.Z[q] = H.E[q];
        H.Sa[q] = H.Sb[q] = H.Sc[q] = 0.0;
        cosorb[q] = 0.0;
        if (MICH) {
            const double h = A.t[j + 1] - A.t[j];
            const double Om_r = nested_ds(c, s, h);
#pragma unroll
            for (int k = 0; k < 8; ++k) c[k] = A.coef[((long long)k * A.cstride + j) * 6 + 4];
            const double Om_theta = nested_ds(c, s, h);
            H.nu[q] = Om_r / (2. * kPi);
            H.gd[q] = (Om_theta - Om_r) / kPi;
            const int i = min(chunk + tid + q * kThreads, i1 - 1);
            cosorb[q] = cos(2. * kPi * (A.dt * i) / kYRSID - A.phiS);
            H.W[q] = 2. * kPi * kAUsec * K.sinqS * cosorb[q];
            sincos(H.W[q] * H.nu[q], &sn, &cs);
            H.E[q] = cmul(H.E[q], make_double2(cs, sn));
            sincos(H.W[q] * H.gd[q], &sn, &cs);
            H.Z[q] = cmul(H.E[q], make_double2(cs, sn));
            H.large = H.large || !(fabs(H.W[q] * H.nu[q]) * A.nmodes < 1e6);
        }
    }

    for (int n0 = 1; n0 <= A.nmodes; n0 += kHarm) {
        const int count = min(kHarm, A.nmodes + 1 - n0);
        const int set = node_set((n0 + count - 1) * delta);
        if (set < 3) {
            const int Q = set == 0 ? 6 : (set == 1 ? 8 : 12);
            const Cheb &T = c_cheb[set];
            __syncthreads();  // the previous group's coefficients have been read
            const int pairs = (count + 1) / 2;
            for (int w = tid; w < pairs * Q; w += kThreads) {
                const int pr = w / Q, j = w - pr * Q, n = n0 + 2 * pr;
                const double en = fma(delta, T.node[j], ec);
                double Ja[5], Jb[5], f[3];
                const double xa = n * en, xb = (n + 1) * en;
                bessel_band2(n, xa, xb, Ja, Jb);
                to_exact_argument(n, en, xa, Ja);
                to_exact_argument(n + 1, en, xb, Jb);
                combine(n, en, Ja, f);
#pragma unroll
                for (int q = 0; q < 3; ++q) s_co[(2 * pr * 3 + q) * kMaxNodes + j] = f[q];
                combine(n + 1, en, Jb, f);
#pragma unroll
                for (int q = 0; q < 3; ++q) s_co[((2 * pr + 1) * 3 + q) * kMaxNodes + j] = f[q];
            }
            __syncthreads();
            if (set == 0) to_powers<6>(T, count * 3, s_co, s_cheb);
            else if (set == 1) to_powers<8>(T, count * 3, s_co, s_cheb);
            else to_powers<12>(T, count * 3, s_co, s_cheb);
            __syncthreads();
            if (set == 0) H.template table<6>(n0, count, s_co, A, K, cosorb);
            else if (set == 1) H.template table<8>(n0, count, s_co, A, K, cosorb);
            else H.template table<12>(n0, count, s_co, A, K, cosorb);
        } else {
#pragma unroll
            for (int q = 0; q < P; ++q) {
                double Ja[5], Jb[5], f[3];
                for (int h = 0; h < count; ++h) {
                    const int n = n0 + h;
                    const bool odd = (n & 1) != 0;
                    if (odd) bessel_band2(n, n * e[q], (n + 1) * e[q], Ja, Jb);  // the last n + 1 may go unused
                    double J[5];
#pragma unroll
                    for (int k = 0; k < 5; ++k) J[k] = odd ? Ja[k] : Jb[k];
                    combine(n, e[q], J, f);
                    double cn, sn;
                    H.phasor(n, q, A, K, cosorb, cn, sn);
                    H.Sa[q] = fma(f[0], cn, H.Sa[q]);
                    H.Sb[q] = fma(f[1], sn, H.Sb[q]);
                    H.Sc[q] = fma(f[2], cn, H.Sc[q]);
                    H.Z[q] = cmul(H.Z[q], H.E[q]);
                }
            }
        }
    }

    const double halfsqrt3 = sqrt(3.) / 2.;
    const double zeta = A.mu * kMTSUN / A.dist / kGPCINSEC;
    const double nv[3] = {K.sinqS * K.cosPS, K.sinqS * K.sinPS, K.cosqS};
    const double Sv[3] = {K.sinqK * K.cosPK, K.sinqK * K.sinPK, K.cosqK};
    double nxS[3];
    cross3(nv, Sv, nxS);
    const double nS = sqrt(nxS[0] * nxS[0] + nxS[1] * nxS[1] + nxS[2] * nxS[2]);
    const double Sdotn = K.cosqK * K.cosqS + K.sinqK * K.sinqS * K.cosdP;
#pragma unroll
    for (int q = 0; q < P; ++q) {
        const int i = chunk + tid + q * kThreads;
        if (i >= i1) continue;
        const int j = seg[q];
        const double s = sa[q], s1 = 1.0 - s;
        double c[3][8];  // Y, Phi_phi, Phi_theta
#pragma unroll
        for (int w = 0; w < 3; ++w)
#pragma unroll
            for (int k = 0; k < 8; ++k) c[w][k] = A.coef[((long long)k * A.cstride + j) * 6 + w + 2];
        const double h = A.t[j + 1] - A.t[j];
        const double Y = nested(c[0], s, s1), Phi_phi = nested(c[1], s, s1), Phi_theta = nested(c[2], s, s1);
        const double Om_phi = nested_ds(c[1], s, h);
        const double gim = Phi_theta - H.Phi[q], alp = Phi_phi - Phi_theta;
        // lam = acos(Y): its cosine is Y, its sine the root below
        const double coslam = Y, sinlam = sqrt((1.0 - Y) * (1.0 + Y));
        double sinalp, cosalp;
        sincos_phase(alp, &sinalp, &cosalp);
        const double Lv[3] = {coslam * K.sinqK * K.cosPK + sinlam * (sinalp * K.sinPK - cosalp * K.cosqK * K.cosPK),
                              coslam * K.sinqK * K.sinPK - sinlam * (sinalp * K.cosPK + cosalp * K.cosqK * K.sinPK),
                              coslam * K.cosqK + sinlam * cosalp * K.sinqK};
        // cos q_L cos q_S + sin q_L sin q_S cos(phi_L - phi_S), sin q_L from cos q_L as the
        // reference forms it (it loses digits near the poles, and they show in the result)
        const double horiz = Lv[0] * Lv[0] + Lv[1] * Lv[1];
        const double cosL = horiz > 0.0 ? (Lv[0] * K.cosPS + Lv[1] * K.sinPS) / sqrt(horiz) : K.cosPS;
        const double Ldotn = Lv[2] * K.cosqS + sqrt(1. - Lv[2] * Lv[2]) * K.sinqS * cosL;
        const double Ldotn2 = Ldotn * Ldotn;
        double beta = 0.0;
        if (!(A.S == 0.0 || fabs(Y) == 1.0)) {  // lam within 1e-10 of 0 or pi only when |Y| = 1
            const double up = -Sdotn + coslam * Ldotn;
            const double down =
                K.sinqS * K.sindP * sinlam * cosalp + (K.cosqK * Sdotn - K.cosqS) / K.sinqK * sinlam * sinalp;
            beta = atan2(up, down);
        }
        double sin2gam, cos2gam;
        sincos_phase(2. * (gim + beta), &sin2gam, &cos2gam);

        double FpI = 1.0, FcI = 0.0, FpII = 0.0, FcII = 1.0;
        if (MICH) {
            const double orb = 2. * kPi * (A.dt * i) / kYRSID;
            double sorb, corb;
            sincos(orb, &sorb, &corb);
            const double sinorb = sorb * K.cosPS - corb * K.sinPS;  // of orb - phiS
            const double cosq = .5 * K.cosqS - halfsqrt3 * K.sinqS * cosorb[q];
            // phiw = orb + atan2(wy, wx); twice the angles enter, as (x + iy)^2 / |x + iy|^2
            const double wy = halfsqrt3 * K.cosqS + .5 * K.sinqS * cosorb[q], wx = K.sinqS * sinorb;
            const double psiup = .5 * K.cosqK - halfsqrt3 * K.sinqK * (corb * K.cosPK + sorb * K.sinPK) -
                                 cosq * (K.cosqK * K.cosqS + K.sinqK * K.sinqS * K.cosdP);
            const double psidown = .5 * K.sinqK * K.sinqS * K.sindP -
                                   halfsqrt3 * corb * (K.cosqK * K.sinqS * K.sinPS - K.cosqS * K.sinqK * K.sinPK) -
                                   halfsqrt3 * sorb * (K.cosqS * K.sinqK * K.cosPK - K.cosqK * K.sinqS * K.cosPS);
            const double cosq1 = .5 * (1. + cosq * cosq);
            const double zx = wx * corb - wy * sorb, zy = wx * sorb + wy * corb;
            const double zr = zx * zx + zy * zy, pr = psiup * psiup + psidown * psidown;
            const double s2phi = zr > 0.0 ? 2. * zx * zy / zr : 0.0, c2phi = zr > 0.0 ? (zx - zy) * (zx + zy) / zr : 1.0;
            const double s2psi = pr > 0.0 ? 2. * psiup * psidown / pr : 0.0;
            const double c2psi = pr > 0.0 ? (psidown - psiup) * (psidown + psiup) / pr : 1.0;
            FpI = halfsqrt3 * (cosq1 * c2phi * c2psi - cosq * s2phi * s2psi);
            FcI = halfsqrt3 * (cosq1 * c2phi * s2psi + cosq * s2phi * c2psi);
            FpII = halfsqrt3 * (cosq1 * s2phi * c2psi + cosq * c2phi * s2psi);
            FcII = halfsqrt3 * (cosq1 * s2phi * s2psi - cosq * c2phi * c2psi);
        }
        const double root = cbrt(fabs(Om_phi) * A.M * kMTSUN);
        const double Amp = root * root * zeta;

        // polarisation rotation (gpuAAK.cu:141-177)
        double nxL[3];
        cross3(nv, Lv, nxL);
        double norm = sqrt(nxL[0] * nxL[0] + nxL[1] * nxL[1] + nxL[2] * nxL[2]) * nS;
        if (norm < 1e-6) norm = 1e-6;
        const double cosrot = (nxL[0] * nxS[0] + nxL[1] * nxS[1] + nxL[2] * nxS[2]) / norm;
        const double sinrot = (Lv[0] * nxS[0] + Lv[1] * nxS[1] + Lv[2] * nxS[2] -
                               (Sv[0] * nxL[0] + Sv[1] * nxL[1] + Sv[2] * nxL[2])) /
                              norm;
        const double rot0 = 2. * cosrot * cosrot - 1., rot1 = cosrot * sinrot;

        const double a = Amp * H.Sa[q], b = Amp * sqrt(1 - e[q] * e[q]) * H.Sb[q], cc = Amp * H.Sc[q];
        const double Ap0 = -(1. + Ldotn2) * (a * cos2gam - b * sin2gam) + cc * (1 - Ldotn2);
        const double Ac0 = 2. * Ldotn * (b * cos2gam + a * sin2gam);
        const double Ap = Ap0 * rot0 + Ac0 * rot1;
        const double Ac = Ac0 * rot0 - Ap0 * rot1;
        A.wf[i] = make_double2(FpI * Ap + FcI * Ac, -(FpII * Ap + FcII * Ac));
    }
}

// Four samples a thread share each coefficient read, two with the response (whose
// state for four spills: 0.60 against 0.59 ms at one year, 80 against 60 us at
// 310,000 samples); one when more would leave SMs without a CTA.  Four CTAs per
// SM: with plain sums 0.39 ms at one year, 0.42 and 0.51 at three and two.
int launch_aak(const AakArgs &A, int total, cudaStream_t st) {
    const int per = total < 148 * 2 * 4 * kThreads ? 1 : (A.mich ? 2 : 4);
    const int ctas = (total + per * kThreads - 1) / (per * kThreads);
    if (per == 4) k_aak<4, false><<<ctas, kThreads, 0, st>>>(A);
    else if (per == 2) k_aak<2, true><<<ctas, kThreads, 0, st>>>(A);
    else if (A.mich) k_aak<1, true><<<ctas, kThreads, 0, st>>>(A);
    else k_aak<1, false><<<ctas, kThreads, 0, st>>>(A);
    FEW_LAUNCH_CHECK("k_aak");
    return FEW_OK;
}

}  // namespace aak
}  // namespace few

// Segment ownership of the reference (gpuAAK.cu:495-519): first[0] = 0, then
// ceil(t_j / dt) for knots before T = (out_len - 1) dt; the first knot at or
// after T closes the list with out_len.  Returns the number of segments.
static int aak_segments(const double *h_t, int init_len, int out_len, double dt, std::vector<int> &first) {
    const double T = (out_len - 1) * dt;
    first.assign(init_len, 0);
    int i = 1;
    for (; i < init_len; ++i) {
        const double tt = h_t[i];
        if (tt < T) {
            first[i] = (int)std::ceil(tt / dt);
        } else {
            first[i] = out_len;
            break;
        }
    }
    const int npts = (i + 1 < init_len ? i + 1 : init_len);
    first.resize(npts);
    return npts - 1;
}

// The kernel on device tables, without allocation or synchronisation (what
// AAKSummation calls): t_knots [device] (>= nseg + 1), first [device]
// (nseg + 1) from the segment rule below, coef [device] (8, cstride, 6).
extern "C" FEW_API int few_aak_sum(void *waveform, const double *coef, int cstride, const double *t_knots,
                                   const int *first, int nseg, int total, double M_phys, double S_phys, double mu,
                                   double qS, double phiS, double qK, double phiK, double dist, int nmodes, int mich,
                                   double delta_t, void *stream) {
    few::clear_error();
    if (nseg < 0 || cstride < nseg || total < 0 || nmodes < 0 || nmodes > 4096)
        return few::fail(FEW_ERR_SIZE, "few_aak_sum: nseg=%d cstride=%d total=%d nmodes=%d", nseg, cstride, total,
                         nmodes);
    if (nseg == 0 || total == 0) return FEW_OK;
    if (!waveform || !coef || !t_knots || !first) return few::fail(FEW_ERR_ARG, "few_aak_sum: null pointer");
    few::aak::AakArgs A;
    A.wf = static_cast<double2 *>(waveform);
    A.coef = coef;
    A.t = t_knots;
    A.first = first;
    A.nseg = nseg;
    A.cstride = cstride;
    A.nmodes = nmodes;
    A.mich = mich;
    A.M = M_phys; A.S = S_phys; A.mu = mu; A.qS = qS; A.phiS = phiS; A.qK = qK; A.phiK = phiK; A.dist = dist;
    A.dt = delta_t;
    return few::aak::launch_aak(A, total, static_cast<cudaStream_t>(stream));
}

// Drop-in for get_waveform of gpuAAK.hh:6-10 (AAKSummation's kernel call,
// aakwave.py:175-192): interp_array [device] (8, init_len-1, 6) =
// the trajectory's dense-output coefficients of (p, e, Y, Phi_phi, Phi_theta,
// Phi_r); h_t [host] (init_len,) knots; waveform [device] (out_len,) complex,
// samples of covered segments overwritten.  Plus the stream.
extern "C" FEW_API int few_aak_waveform(void *waveform, const double *interp_array, double M_phys, double S_phys,
                                        double mu, double qS, double phiS, double qK, double phiK, double dist,
                                        int nmodes, int mich, int init_len, int out_len, double delta_t,
                                        const double *h_t, void *stream) {
    few::clear_error();
    if (init_len < 2 || out_len < 1 || nmodes < 0 || nmodes > 4096)
        return few::fail(FEW_ERR_SIZE, "few_aak_waveform: init_len=%d out_len=%d nmodes=%d", init_len, out_len,
                         nmodes);
    if (!waveform || !interp_array || !h_t) return few::fail(FEW_ERR_ARG, "few_aak_waveform: null pointer");
    if (!(delta_t > 0.0)) return few::fail(FEW_ERR_ARG, "few_aak_waveform: delta_t must be positive");
    std::vector<int> first;
    const int nseg = aak_segments(h_t, init_len, out_len, delta_t, first);
    if (nseg < 1) return FEW_OK;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    void *buf = nullptr;
    const size_t tbytes = (size_t)init_len * sizeof(double), fbytes = first.size() * sizeof(int);
    FEW_CUDA_TRY(cudaMallocAsync(&buf, tbytes + fbytes, st));
    double *t_d = static_cast<double *>(buf);
    int *first_d = reinterpret_cast<int *>(t_d + init_len);
    cudaError_t e1 = cudaMemcpyAsync(t_d, h_t, tbytes, cudaMemcpyHostToDevice, st);
    if (e1 == cudaSuccess) e1 = cudaMemcpyAsync(first_d, first.data(), fbytes, cudaMemcpyHostToDevice, st);
    int status = FEW_OK;
    if (e1 != cudaSuccess) {
        status = few::fail(FEW_ERR_CUDA, "few_aak_waveform: upload failed: %s", cudaGetErrorString(e1));
    } else {
        few::aak::AakArgs A;
        A.wf = static_cast<double2 *>(waveform);
        A.coef = interp_array;
        A.t = t_d;
        A.first = first_d;
        A.nseg = nseg;
        A.cstride = init_len - 1;
        A.nmodes = nmodes;
        A.mich = mich;
        A.M = M_phys; A.S = S_phys; A.mu = mu; A.qS = qS; A.phiS = phiS; A.qK = qK; A.phiK = phiK; A.dist = dist;
        A.dt = delta_t;
        status = few::aak::launch_aak(A, first.back(), st);
    }
    // the host vector must outlive the copy
    cudaError_t e3 = cudaStreamSynchronize(st);
    cudaError_t e4 = cudaFreeAsync(buf, st);
    if (status != FEW_OK) return status;
    if (e3 != cudaSuccess) return few::fail(FEW_ERR_CUDA, "few_aak_waveform: %s", cudaGetErrorString(e3));
    if (e4 != cudaSuccess) return few::fail(FEW_ERR_CUDA, "few_aak_waveform: free failed: %s", cudaGetErrorString(e4));
    return FEW_OK;
}
