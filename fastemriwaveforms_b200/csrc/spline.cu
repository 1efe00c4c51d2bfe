// Batched not-a-knot cubic splines: build (tridiagonal solve) and evaluation.
//
// Build.  The reference fills the not-a-knot rows (src/few/cutils/interpolate.cu:48-145),
// solves every system with a pivoting tridiagonal solver (cuSPARSE gtsv2StridedBatch
// on the GPU, LAPACK dgtsv on the CPU, interpolate.cu:201-239) and then derives
// the cubic coefficients (interpolate.cu:29-43, 149-198, 241-280) in three more
// launches with host synchronisations between them.
//
// Here one thread owns one interpolant and does all of it in one launch:
//   * The first and last not-a-knot rows are not diagonally dominant, so they
//     are eliminated up front.  Row 0 reads h1*s0 + (x2-x0)*s1 = b0 and row 1
//     has h1 as its s0 coefficient, so row1 - row0 removes s0 with an exact
//     factor of 1 (the same elimination a pivoting solver makes at that step);
//     the last row is removed from row N-2 the same way.  Rows 1..N-2 are then
//     strictly diagonally dominant and a Thomas sweep without pivoting is
//     stable.
//   * The forward sweep writes its two running values (c'_i, r'_i) into the
//     c2/c3 output rows of knot i; the backward sweep reads them back, forms the
//     slope s_i and immediately overwrites knot i with the final coefficients,
//     so no scratch memory is used.
//   * The coefficient formulas are those of fill_coefficients and
//     fill_final_derivs (the last knot carries the derivative-extrapolated
//     c1, c2, c3 of the last segment).
// y is read through a strided view, so the (N, K) complex Teukolsky amplitudes
// are splined in place (real parts as interpolants 0..K-1, imaginary parts as
// K..2K-1) with no (2K, N) copy.  Output layout (4, N, ninterps) makes every
// store of a warp one contiguous run.
//
// Evaluation restates CubicSplineInterpolant.__call__
// (src/few/summation/interpolatedmodesum.py:118-257): interval by
// searchsorted(side="right") - 1 with the last knot mapped to the last interval,
// y + c1 x + c2 x^2 + c3 x^3 (or a derivative), edge values outside the range.
#include <algorithm>

#include "few_common.cuh"
#include "few_internal.h"

namespace few {

namespace {

struct SplineArgs {
    const double *t;
    long long t_rs;
    const double *y;
    long long sk, sp, off2;
    int split;
    int ni, N;
    double *out;
    long long os_i, os_p;  // output stride per knot / per interpolant inside one plane
};

__device__ __forceinline__ void write_segment(double *o1, double *o2, double *o3, long long off, double s_i,
                                              double s_ip1, double y_i, double y_ip1, double dx)
{
    // fill_coefficients (interpolate.cu:29-43)
    double slope = (y_ip1 - y_i) / dx;
    double tt = (s_i + s_ip1 - 2 * slope) / dx;
    o1[off] = s_i;
    o2[off] = (slope - s_i) / dx - tt;
    o3[off] = tt / dx;
}

// What k_spline_build_rows leaves in place of the first slope of a series that it gives up
// (a NaN's bits: a series that happens to have them is built twice, alike).
constexpr long long kGivenUp = 0x7ff8b2005eed0001LL;

// MARKED: only the series that k_spline_build_rows has given up.
template <bool MARKED>
__global__ void __launch_bounds__(128) k_spline_build(SplineArgs a)
{
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= a.ni) return;
    const int N = a.N;
    if (MARKED && __double_as_longlong(a.out[(long long)p * a.os_p + (long long)N * a.ni]) != kGivenUp) return;
    const double *x = a.t + (long long)p * a.t_rs;
    const double *yb = (p < a.split) ? a.y + (long long)p * a.sp : a.y + a.off2 + (long long)(p - a.split) * a.sp;
    const long long sk = a.sk;
    const long long plane = (long long)N * a.ni, oi = a.os_i;
    double *o0 = a.out + (long long)p * a.os_p;
    double *o1 = o0 + plane;
    double *o2 = o1 + plane;
    double *o3 = o2 + plane;

    // First not-a-knot row (interpolate.cu:71-86).
    const double x0 = x[0], x1 = x[1], x2 = x[2];
    const double y0 = yb[0], y1 = yb[sk], y2 = yb[2 * sk];
    const double h0 = x1 - x0, h1 = x2 - x1, d0 = x2 - x0;
    const double b0 = ((h0 + 2 * d0) * h1 * ((y1 - y0) / h0) + h0 * h0 * ((y2 - y1) / h1)) / d0;
    // Last not-a-knot row (interpolate.cu:56-69).
    const double xa = x[N - 3], xb = x[N - 2], xc = x[N - 1];
    const double ya = yb[(long long)(N - 3) * sk], yv = yb[(long long)(N - 2) * sk], yc = yb[(long long)(N - 1) * sk];
    const double hA = xb - xa, hB = xc - xb, dE = xc - xa;
    const double bE = (hB * hB * ((yv - ya) / hA) + (2 * dE + hB) * hA * ((yc - yv) / hB)) / dE;

    // Forward sweep over rows 1..N-2 (interior rows of interpolate.cu:88-101).
    double cprev = 0.0, rprev = 0.0;
    double xm = x0, xi = x1, ym = y0, yi = y1;
    for (int i = 1; i <= N - 2; ++i) {
        const double xn = x[i + 1];
        const double yn = yb[(long long)(i + 1) * sk];
        const double hl = xi - xm, hr = xn - xi;
        double lo = hr, dg = 2 * (hl + hr), up = hl;
        double rhs = 3.0 * (hr * ((yi - ym) / hl) + hl * ((yn - yi) / hr));
        if (i == 1) {  // row 1 - row 0
            dg -= d0;
            rhs -= b0;
            lo = 0.0;
        }
        if (i == N - 2) {  // row N-2 - row N-1
            dg -= dE;
            rhs -= bE;
            up = 0.0;
        }
        const double den = dg - lo * cprev;
        const double cp = up / den;
        const double rp = (rhs - lo * rprev) / den;
        o2[i * oi] = cp;
        o3[i * oi] = rp;
        cprev = cp;
        rprev = rp;
        xm = xi;
        xi = xn;
        ym = yi;
        yi = yn;
    }

    // Backward sweep.  s_{N-2} = r'_{N-2}; s_{N-1} from the last row.
    double s_ip1 = rprev;
    const double s_last = (bE - dE * s_ip1) / hA;
    {
        const long long off = (long long)(N - 2) * oi;
        write_segment(o1, o2, o3, off, s_ip1, s_last, yv, yc, hB);
        o0[off] = yv;
        // fill_final_derivs (interpolate.cu:241-280)
        const double c1 = o1[off], c2 = o2[off], c3 = o3[off];
        const double xx = hB, x2v = xx * xx;
        const long long offe = (long long)(N - 1) * oi;
        o0[offe] = yc;
        o1[offe] = c1 + 2 * c2 * xx + 3 * c3 * x2v;
        o2[offe] = (2. * c2 + 6. * c3 * xx) / 2.;
        o3[offe] = c3;
    }
    double xr = xb, yr = yv;  // knot i+1
    for (int i = N - 3; i >= 1; --i) {
        const long long off = (long long)i * oi;
        const double cp = o2[off], rp = o3[off];
        const double s_i = rp - cp * s_ip1;
        const double xl = x[i];
        const double yl = yb[(long long)i * sk];
        write_segment(o1, o2, o3, off, s_i, s_ip1, yl, yr, xr - xl);
        o0[off] = yl;
        s_ip1 = s_i;
        xr = xl;
        yr = yl;
    }
    // s_0 from the first row.
    const double s0 = (b0 - d0 * s_ip1) / h1;
    write_segment(o1, o2, o3, 0, s0, s_ip1, y0, y1, h0);
    o0[0] = y0;
}

// The same build with a CTA per series, for every bit of the thread form's
// result.  The two sweeps are serial chains of a multiply-add and a division per
// knot (0.6 us a knot with their loads, whatever the number of series), but they
// forget their start: a step shrinks a difference by 0.6 at most, 0.3 as a rule.
// So each thread takes one run of rows and starts kWarmup rows before it from an
// arbitrary state; the threads then compare the state they came to at their first
// row with the one the thread before ended with, and only if all agree to the
// last bit is the result that of the serial sweep.  Sweeps that differ by 1e-25 of
// themselves agree in every bit, but the state behind a pulse, a step or a NaN does not:
// then one thread sweeps the series, or (give_up: more series than a few at a time on an
// SM, where that would take longer) it is left to the thread form.  Knots, right-hand sides and sweep values stay in shared memory;
// everything else is formed with consecutive knots on consecutive threads.  Bound
// by the chain of 64 + N/128 steps: 34 us for 3 series of 1000 knots and 46 us for
// 256 (592 and 800 us with a thread per series); with a warp per series and the
// sweep values in global memory 73 and 105 us.
constexpr int kWarmup = 64;
constexpr int kRowThreads = 128;
constexpr int kRowSmem = 200 * 1024;

struct RowSweep {
    const double *x, *rhs;  // shared: knots, right-hand sides of the interior rows
    double *cp, *rp;        // shared: c'_i, r'_i
    int N;
    double d0, dE;
};

// Rows [a, e) of the forward sweep from state (c, r) = (c'_{a-1}, r'_{a-1}); rows
// from `keep` on are stored.  (ck, rk): the state before row `keep`.
__device__ __forceinline__ void forward_rows(const RowSweep &w, int a, int keep, int e, double &c, double &r,
                                             double &ck, double &rk)
{
    for (int i = a; i < e; ++i) {
        if (i == keep) {
            ck = c;
            rk = r;
        }
        const double hl = w.x[i] - w.x[i - 1], hr = w.x[i + 1] - w.x[i];
        double lo = hr, dg = 2 * (hl + hr), up = hl;
        if (i == 1) {  // row 1 - row 0
            dg -= w.d0;
            lo = 0.0;
        }
        if (i == w.N - 2) {  // row N-2 - row N-1
            dg -= w.dE;
            up = 0.0;
        }
        const double den = dg - lo * c;
        const double cp = up / den;
        const double rp = (w.rhs[i] - lo * r) / den;
        if (i >= keep) {
            w.cp[i] = cp;
            w.rp[i] = rp;
        }
        c = cp;
        r = rp;
    }
}

__device__ __forceinline__ bool same_bits(double a, double b)
{
    return __double_as_longlong(a) == __double_as_longlong(b);
}

__global__ void __launch_bounds__(kRowThreads) k_spline_build_rows(SplineArgs a, bool give_up)
{
    extern __shared__ __align__(16) double row_smem[];
    __shared__ double s_c[kRowThreads + 1], s_r[kRowThreads + 1];
    const int p = blockIdx.x, tid = threadIdx.x;
    const int N = a.N;
    const double *xg = a.t + (long long)p * a.t_rs;
    const double *yb = (p < a.split) ? a.y + (long long)p * a.sp : a.y + a.off2 + (long long)(p - a.split) * a.sp;
    const long long sk = a.sk;
    const long long plane = (long long)N * a.ni, oi = a.os_i;
    double *o0 = a.out + (long long)p * a.os_p;
    double *o1 = o0 + plane;
    double *o2 = o1 + plane;
    double *o3 = o2 + plane;
    double *x = row_smem, *rhs = x + N;  // rhs: later the slopes s_i
    RowSweep w;
    w.x = x;
    w.rhs = rhs;
    w.cp = rhs + N;
    w.rp = w.cp + N;
    w.N = N;
    for (int i = tid; i < N; i += kRowThreads) x[i] = xg[i];
    __syncthreads();

    // First and last not-a-knot rows (interpolate.cu:56-86).
    const double x0 = x[0], x1 = x[1], x2 = x[2];
    const double y0 = yb[0], y1 = yb[sk], y2 = yb[2 * sk];
    const double h0 = x1 - x0, h1 = x2 - x1, d0 = x2 - x0;
    const double b0 = ((h0 + 2 * d0) * h1 * ((y1 - y0) / h0) + h0 * h0 * ((y2 - y1) / h1)) / d0;
    const double xa = x[N - 3], xb = x[N - 2], xc = x[N - 1];
    const double ya = yb[(long long)(N - 3) * sk], yv = yb[(long long)(N - 2) * sk], yc = yb[(long long)(N - 1) * sk];
    const double hA = xb - xa, hB = xc - xb, dE = xc - xa;
    const double bE = (hB * hB * ((yv - ya) / hA) + (2 * dE + hB) * hA * ((yc - yv) / hB)) / dE;
    w.d0 = d0;
    w.dE = dE;
    for (int i = 1 + tid; i <= N - 2; i += kRowThreads) {
        const double xm = x[i - 1], xi = x[i], xn = x[i + 1];
        const double ym = yb[(long long)(i - 1) * sk], yi = yb[(long long)i * sk], yn = yb[(long long)(i + 1) * sk];
        const double hl = xi - xm, hr = xn - xi;
        double v = 3.0 * (hr * ((yi - ym) / hl) + hl * ((yn - yi) / hr));
        if (i == 1) v -= b0;
        if (i == N - 2) v -= bE;
        rhs[i] = v;
    }
    __syncthreads();

    // forward sweep, rows 1..N-2
    const int L = (N - 2 + kRowThreads - 1) / kRowThreads;
    const int first = 1 + tid * L, last = min(first + L, N - 1);  // this thread's rows [first, last)
    const bool has = first < last;
    double c = 0.0, r = 0.0, ck = 0.0, rk = 0.0;
    if (has) forward_rows(w, max(1, first - kWarmup), first, last, c, r, ck, rk);
    s_c[tid + 1] = c;
    s_r[tid + 1] = r;
    __syncthreads();
    if (__syncthreads_or(has && tid > 0 && !(same_bits(ck, s_c[tid]) && same_bits(rk, s_r[tid])))) {
        if (give_up) {
            if (tid == 0) o1[0] = __longlong_as_double(kGivenUp);
            return;
        }
        c = r = 0.0;
        if (tid == 0) forward_rows(w, 1, 1, N - 1, c, r, ck, rk);
        __syncthreads();
    }

    // backward sweep: s_{N-2} = r'_{N-2}, s_i = r'_i - c'_i s_{i+1}
    double *slope = rhs;
    double s = 0.0, s_in = 0.0;
    if (has) {
        int i = min(last - 1 + kWarmup, N - 2);
        s = w.rp[i];
        if (i == last - 1) slope[i] = s;
        for (--i; i >= first; --i) {
            if (i == last - 1) s_in = s;
            s = w.rp[i] - w.cp[i] * s;
            if (i < last) slope[i] = s;
        }
    }
    s_c[tid] = s;
    __syncthreads();
    if (__syncthreads_or(has && last < N - 1 && !same_bits(s_in, s_c[tid + 1]))) {
        if (give_up) {
            if (tid == 0) o1[0] = __longlong_as_double(kGivenUp);
            return;
        }
        if (tid == 0) {
            s = w.rp[N - 2];
            slope[N - 2] = s;
            for (int i = N - 3; i >= 1; --i) {
                s = w.rp[i] - w.cp[i] * s;
                slope[i] = s;
            }
        }
        __syncthreads();
    }

    // coefficients of the segments 1..N-3, then the two end segments and the last knot
    for (int i = 1 + tid; i <= N - 3; i += kRowThreads) {
        const long long of = (long long)i * oi;
        const double yl = yb[(long long)i * sk], yr = yb[(long long)(i + 1) * sk];
        write_segment(o1, o2, o3, of, slope[i], slope[i + 1], yl, yr, x[i + 1] - x[i]);
        o0[of] = yl;
    }
    if (tid == 0) {
        const long long of = (long long)(N - 2) * oi, offe = (long long)(N - 1) * oi;
        const double s_ip1 = slope[N - 2];
        const double s_last = (bE - dE * s_ip1) / hA;
        write_segment(o1, o2, o3, of, s_ip1, s_last, yv, yc, hB);
        o0[of] = yv;
        const double c1 = o1[of], c2 = o2[of], c3 = o3[of];
        const double xx = hB, x2v = xx * xx;
        o0[offe] = yc;
        o1[offe] = c1 + 2 * c2 * xx + 3 * c3 * x2v;
        o2[offe] = (2. * c2 + 6. * c3 * xx) / 2.;
        o3[offe] = c3;
    }
    if (tid == 32) {
        const double s1 = slope[1];
        const double s0 = (b0 - d0 * s1) / h1;
        write_segment(o1, o2, o3, 0, s0, s1, y0, y1, h0);
        o0[0] = y0;
    }
}

// Shared-knot build from a host factorization (few_spline_factor), in scan form.
// The sweeps are linear recurrences whose factors depend on the knots only:
//     r'_i = A_i r'_{i-1} + (alpha_i delta_{i-1} + beta_i delta_i) / den_i,  A_i = -lo_i / den_i
//     s_i  = C_i s_{i+1} + r'_i,                                            C_i = -c'_i
// so the interior rows are cut into kScanChunks chunks (one warp each; lane =
// series, 32 series per CTA, every access coalesced across the series): each
// warp runs its chunk's forward sweep from a zero carry, the chunk carries are
// chained through shared memory (r'_end = rho_end + (prod A) r'_in), the
// warp corrects its rows (r' = rho + prod_{chunk start..i} A x carry) and runs
// the backward sweep from a zero carry the same way, and finally writes the
// coefficients of its segments from the corrected slopes.  The products come
// from the factor table; the sweep temporaries are parked in the c3 output
// row, which the last pass overwrites.  Loads are issued kSweepBatch steps
// ahead of the arithmetic that uses them.
//
// COEF = false stores the slopes alone, s[i * ni + series] (the same bits as the c1
// plane): a consumer that forms the coefficients from (y, s) spares three of the four
// planes' writes and reads, and the sweep temporaries then stay in L2.  7686 series of
// 1000 knots: 66 us, 122 us with the coefficients.
//
// CHECK: `out` holds what k_spline_chunks built with `overlap`; a CTA whose 32 series'
// records chk say that nothing was left out that shows returns at once (3 us for 256
// series of 1000 knots).
constexpr int kSweepBatch = 8;
constexpr int kChunkRows = 32;

template <bool COEF, bool CHECK>
__global__ void __launch_bounds__(32 * kScanChunks) k_spline_build_factored(
    const double *__restrict__ fac, const double *__restrict__ y, long long sk, long long sp, int split,
    long long off2, int ni, int N, double *__restrict__ out, long long os_i, long long os_p,
    const double *__restrict__ chk, int overlap)
{
    constexpr int W = kFacWidth;
    constexpr int P = kScanChunks;
    __shared__ double s_end[P][32];
    __shared__ double s_carry[P + 1][32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int p0 = blockIdx.x * 32 + lane;
    const bool live = p0 < ni;
    const int p = live ? p0 : ni - 1;  // idle lanes compute on a valid series and store nothing
    const double *yb = (p < split) ? y + (long long)p * sp : y + off2 + (long long)(p - split) * sp;
    const long long plane = (long long)N * ni;
    double *o0 = out + (long long)p * os_p;
    double *o1 = o0 + plane;
    double *o2 = o1 + plane;
    double *o3 = COEF ? o2 + plane : o0;  // the sweep temporaries, then c3 (or the slopes)
    if (CHECK) {
        const int chunks = (N - 2 + kChunkRows - 1) / kChunkRows;
        bool anew = false;
        for (int c = w; c < chunks; c += P) {
            const int ca = 1 + c * kChunkRows, ce = min(ca + kChunkRows, N - 1);
            const int before = ca - overlap - 1;    // the row whose state the forward sweep left out; none below 1
            const long long after = ce + overlap;   // and the backward one; none from N - 1 on
            const double *lim = chk + (long long)c * 3 * ni + p;
            if (before >= 1)
                anew |= !(fabs(chk[(long long)((before - 1) / kChunkRows) * 3 * ni + p]) <= lim[ni]);
            if (after < N - 1) anew |= !(fabs(o1[after * os_i]) <= lim[2LL * ni]);
        }
        if (!__syncthreads_or(anew)) return;
    }
    const int L = (N - 2 + P - 1) / P;
    const int a = 1 + w * L, e = min(a + L, N - 1);  // this warp's rows [a, e); empty if a >= e

    // pass 1: forward sweep from a zero carry
    double rho = 0.0;
    if (a < e) {
        double ym = yb[(long long)a * sk];
        double dprev = (ym - yb[(long long)(a - 1) * sk]) * __ldg(fac + W * (a - 1) + 6);
        for (int i0 = a; i0 < e; i0 += kSweepBatch) {
            double yv[kSweepBatch], fl[kSweepBatch], fi[kSweepBatch], fa[kSweepBatch], fb[kSweepBatch], fh[kSweepBatch];
#pragma unroll
            for (int q = 0; q < kSweepBatch; ++q) {
                const int i = min(i0 + q, e - 1);
                yv[q] = yb[(long long)(i + 1) * sk];
                const double *f = fac + (long long)W * i;
                fl[q] = __ldg(f + 0);
                fi[q] = __ldg(f + 1);
                fa[q] = __ldg(f + 3);
                fb[q] = __ldg(f + 4);
                fh[q] = __ldg(f + 6);
            }
#pragma unroll
            for (int q = 0; q < kSweepBatch; ++q) {
                const int i = i0 + q;
                if (i < e) {
                    const double del = (yv[q] - ym) * fh[q];
                    rho = (fa[q] * dprev + fb[q] * del - fl[q] * rho) * fi[q];
                    if (live) o3[(long long)i * os_i] = rho;
                    dprev = del;
                    ym = yv[q];
                }
            }
        }
    }
    s_end[w][lane] = rho;
    __syncthreads();
    if (w == 0) {  // chain the forward carries: r' entering chunk q
        double c = 0.0;
        for (int q = 0; q < P; ++q) {
            s_carry[q][lane] = c;
            const int aq = 1 + q * L, eq = min(aq + L, N - 1);
            if (aq < eq) c = s_end[q][lane] + __ldg(fac + (long long)W * (eq - 1) + 10) * c;
        }
    }
    __syncthreads();
    const double cf = s_carry[w][lane];

    // pass 2: r' = rho + prod(A) cf, then the backward sweep from a zero carry
    double sig = 0.0;
    if (a < e) {
        for (int i0 = e - 1; i0 >= a; i0 -= kSweepBatch) {
            double rv[kSweepBatch], fp[kSweepBatch], fc[kSweepBatch];
#pragma unroll
            for (int q = 0; q < kSweepBatch; ++q) {
                const int i = max(i0 - q, a);
                rv[q] = o3[(long long)i * os_i];
                fp[q] = __ldg(fac + (long long)W * i + 10);
                fc[q] = __ldg(fac + (long long)W * i + 2);
            }
#pragma unroll
            for (int q = 0; q < kSweepBatch; ++q) {
                const int i = i0 - q;
                if (i >= a) {
                    const double r = fma(fp[q], cf, rv[q]);
                    sig = r - fc[q] * sig;
                    if (live) o3[(long long)i * os_i] = sig;
                }
            }
        }
    }
    __syncthreads();
    s_end[w][lane] = sig;
    __syncthreads();
    if (w == 0) {  // chain the backward carries: s at the row after chunk q; s_1 last
        double c = 0.0;
        for (int q = P - 1; q >= 0; --q) {
            s_carry[q][lane] = c;
            const int aq = 1 + q * L, eq = min(aq + L, N - 1);
            if (aq < eq) c = s_end[q][lane] + __ldg(fac + (long long)W * aq + 11) * c;
        }
        s_carry[P][lane] = c;
    }
    __syncthreads();
    if (a >= e || !live) return;
    const double cb = s_carry[w][lane];

    // pass 3: slopes s_i = sig_i + prod(C) cb and the coefficients of segments
    // [a, e) (fill_coefficients, interpolate.cu:29-43); the last chunk also the
    // extrapolated last knot (fill_final_derivs, interpolate.cu:241-280), the
    // first chunk segment 0 from the first not-a-knot row
    double s_ip1, yr;
    int top = e - 1;
    if (e == N - 1) {
        const double *bnd = fac + (long long)W * N;
        const double e0 = __ldg(bnd + 4), e1 = __ldg(bnd + 5), dE = __ldg(bnd + 6), hA = __ldg(bnd + 7);
        const long long i = N - 2;
        const double ya = yb[(i - 1) * sk], yl = yb[i * sk], yc = yb[(i + 1) * sk];
        const double sN2 = fma(__ldg(fac + W * i + 11), cb, o3[i * os_i]);
        const double dA = (yl - ya) * __ldg(fac + W * (i - 1) + 6);
        const double ih = __ldg(fac + W * i + 6), xx = __ldg(fac + W * i + 5);
        const double dl = (yc - yl) * ih;
        const double bE = e0 * dA + e1 * dl;
        const double s_last = (bE - dE * sN2) / hA;
        const double tt = (sN2 + s_last - 2 * dl) * ih;
        const double c1 = sN2, c2 = (dl - sN2) * ih - tt, c3 = tt * ih;
        const long long off = i * os_i, offe = (long long)(N - 1) * os_i;
        if (COEF) {
            __stcs(o0 + off, yl);
            __stcs(o1 + off, c1);
            __stcs(o2 + off, c2);
            __stcs(o3 + off, c3);
            __stcs(o0 + offe, yc);
            __stcs(o1 + offe, c1 + 2 * c2 * xx + 3 * c3 * xx * xx);
            __stcs(o2 + offe, (2. * c2 + 6. * c3 * xx) / 2.);
            __stcs(o3 + offe, c3);
        } else {
            o3[off] = sN2;
            o3[offe] = s_last;
        }
        s_ip1 = sN2;
        yr = yl;
        top = N - 3;
    } else {
        s_ip1 = cb;
        yr = yb[(long long)e * sk];
    }
    for (int i0 = top; i0 >= a; i0 -= kSweepBatch) {
        double yv[kSweepBatch], rv[kSweepBatch], fq[kSweepBatch], fh[kSweepBatch];
#pragma unroll
        for (int q = 0; q < kSweepBatch; ++q) {
            const int i = max(i0 - q, a);
            rv[q] = o3[(long long)i * os_i];
            fq[q] = __ldg(fac + (long long)W * i + 11);
            if (COEF) {
                yv[q] = yb[(long long)i * sk];
                fh[q] = __ldg(fac + (long long)W * i + 6);
            }
        }
#pragma unroll
        for (int q = 0; q < kSweepBatch; ++q) {
            const int i = i0 - q;
            if (i >= a) {
                const long long off = (long long)i * os_i;
                const double s_i = fma(fq[q], cb, rv[q]);
                if (!COEF) {
                    o3[off] = s_i;
                    s_ip1 = s_i;
                    continue;
                }
                const double dl = (yr - yv[q]) * fh[q];
                const double tt = (s_i + s_ip1 - 2 * dl) * fh[q];
                // final coefficients: streaming stores (evict first), so that they do
                // not push the sweep temporaries and y out of L2
                __stcs(o0 + off, yv[q]);
                __stcs(o1 + off, s_i);
                __stcs(o2 + off, (dl - s_i) * fh[q] - tt);
                __stcs(o3 + off, tt * fh[q]);
                s_ip1 = s_i;
                yr = yv[q];
            }
        }
    }
    if (w == 0) {
        // s_0 from the first row: b0 = gamma0 delta_0 + gamma1 delta_1
        const double *bnd = fac + (long long)W * N;
        const double g0 = __ldg(bnd + 0), g1 = __ldg(bnd + 1), d0 = __ldg(bnd + 2), h1 = __ldg(bnd + 3);
        const double y0 = yb[0], y1 = COEF ? yr : yb[sk], y2 = yb[2 * sk];
        const double ih0 = __ldg(fac + 6);
        const double del0 = (y1 - y0) * ih0, del1 = (y2 - y1) * __ldg(fac + W + 6);
        const double s0 = (g0 * del0 + g1 * del1 - d0 * s_ip1) / h1;
        if (!COEF) {
            o3[0] = s0;
            return;
        }
        const double tt = (s0 + s_ip1 - 2 * del0) * ih0;
        o0[0] = y0;
        o1[0] = s0;
        o2[0] = (del0 - s0) * ih0 - tt;
        o3[0] = tt * ih0;
    }
}

// Shared-knot build in one pass, for knots whose sweeps forget their start within
// `overlap` rows (few_spline_overlap: every product of that many factors is below
// 2^-70).  A warp takes 32 series (lane = series) and a chunk of kChunkRows rows: it
// sweeps forward from `overlap` rows before the chunk to `overlap` rows past it and
// backward over the chunk, so no carries are exchanged and nothing but y is read from
// memory; the forward values of the chunk stay in shared memory, a column per
// thread.  The neighbouring chunks' rows read again are in L2.
//
// What a chunk leaves out is the share of the sweeps' states at its far ends, a product
// of `overlap` factors times the state.  For most data that is below any rounding here,
// but not for every value: a NaN or an infinity reaches every knot of its series, and
// beside values 2^17 times smaller the share of a large one shows.  So each chunk
// records how large these states may be for their shares to stay within a rounding of
// what is added up here (chk: the state that another chunk left out, and the limits for
// its own two), and k_spline_build_factored<true, true> then compares them with the
// states that the other chunks came to, and builds the 32 series anew in scan form where
// one is larger or not a number.  Bound by the writes (2048 series of 2000 knots: 116 us
// with the comparison, 148 us in scan form) or, for few series, by the chain of a chunk
// and its overlaps (256 series of 1000 knots: 23 us, 67 us).
constexpr int kChunkWarps = 4;
constexpr int kMaxOverlap = 96;
constexpr int kAhead = 8;  // rows whose loads are in flight ahead of the sweep
constexpr int kTabRows = kChunkWarps * kChunkRows + 2 * kMaxOverlap + 1;

struct ChunkArgs {
    const double *fac, *y;
    long long sk, sp, off2;
    int split, ni, N, overlap;
    double *out;
    long long os_i, os_p;
    double *chk;  // (chunks, 3, ni)
    int groups;   // of 32 series
};

__host__ __device__ inline int spline_chunks(int N) { return (N - 2 + kChunkRows - 1) / kChunkRows; }

// Limit of a left-out state whose share is `share` of it, beside a sum of size `sum`.
__device__ __forceinline__ double state_limit(double sum, double share)
{
    const double v = 0x1p-53 * sum / share;
    return v > 1.7976931348623157e308 ? 1.7976931348623157e308 : v;  // NaN stays; an infinite state is over any limit
}

// Row i of the factorization as the sweeps use it:
// r'_i = A r'_{i-1} + alpha delta_{i-1} + beta delta_i, s_i = r'_i + C s_{i+1}.
struct ChunkRow {
    double A, alpha, beta, C, ih, pad;
};

__global__ void __launch_bounds__(32 * kChunkWarps) k_spline_chunks(ChunkArgs A)
{
    extern __shared__ __align__(16) double chunk_smem[];
    __shared__ __align__(16) ChunkRow tab[kTabRows];
    constexpr int W = kFacWidth, T = 32 * kChunkWarps;
    const int tid = threadIdx.x, lane = tid & 31;
    const int N = A.N, ni = A.ni, ov = A.overlap;
    const double *__restrict__ fac = A.fac;
    const int tile = blockIdx.x / A.groups, group = blockIdx.x - tile * A.groups;
    const int a0 = 1 + tile * kChunkWarps * kChunkRows;
    const int t0 = max(0, a0 - ov - 1), t1 = min(a0 + kChunkWarps * kChunkRows + ov, N - 1);  // rows [t0, t1) of the table
    for (int i = t0 + tid; i < t1; i += T) {
        const double *g = fac + (long long)W * i;
        const double inv = g[1];
        tab[i - t0] = ChunkRow{-g[0] * inv, g[3] * inv, g[4] * inv, -g[2], g[6], 0.0};
    }
    __syncthreads();
    const ChunkRow *row = tab - t0;
    const int a = a0 + (tid >> 5) * kChunkRows, e = min(a + kChunkRows, N - 1);
    if (a >= e) return;
    const int p0 = group * 32 + lane;
    const bool live = p0 < ni;
    const int p = live ? p0 : ni - 1;  // idle lanes compute on a valid series and store nothing
    double *chk = A.chk + (long long)(a - 1) / kChunkRows * 3 * ni + p;
    const double *__restrict__ yb =
        (p < A.split) ? A.y + (long long)p * A.sp : A.y + A.off2 + (long long)(p - A.split) * A.sp;
    const long long sk = A.sk;
    double *col = chunk_smem + tid;  // r'_i of row i at col[(i - a) * T]

    // forward sweep over rows [b, f); the next rows' y are on their way meanwhile.
    // Past the chunk it adds up s_e = r'_e + C_e r'_{e+1} + C_e C_{e+1} r'_{e+2} ...
    const int b = max(1, a - ov), f = min(e + ov, N - 1);
    double s_next = 0.0;  // s_e, then s_{i+1} of the backward sweep
    {
        double prod = 1.0, before = 1.0;         // shares of s_f and r'_{b-1}
        double sum_s = 0.0, sum_r = 0.0;         // what s_e and r'_{a-1} are added up from, by size
        double r = 0.0, ym = yb[(long long)b * sk];
        double dprev = (ym - yb[(long long)(b - 1) * sk]) * row[b - 1].ih;
        double ahead[kAhead];
#pragma unroll
        for (int q = 0; q < kAhead; ++q) ahead[q] = yb[(long long)(min(b + q, f - 1) + 1) * sk];
        for (int i0 = b; i0 < f; i0 += kAhead) {
            double del[kAhead], u[kAhead];
#pragma unroll
            for (int q = 0; q < kAhead; ++q) {
                const ChunkRow &g = row[min(i0 + q, f - 1)];
                del[q] = (ahead[q] - ym) * g.ih;
                ym = ahead[q];
                u[q] = fma(g.alpha, q ? del[q - 1] : dprev, g.beta * del[q]);
            }
            dprev = del[kAhead - 1];
#pragma unroll
            for (int q = 0; q < kAhead; ++q)
                ahead[q] = yb[(long long)(min(i0 + kAhead + q, f - 1) + 1) * sk];
#pragma unroll
            for (int q = 0; q < kAhead; ++q) {
                const int i = i0 + q;
                if (i < f) {
                    r = fma(row[i].A, r, u[q]);
                    if (i >= e) {
                        s_next = fma(prod, r, s_next);
                        sum_s = fma(fabs(prod), fabs(r), sum_s);
                        prod *= row[i].C;
                    } else if (i >= a) {
                        col[(i - a) * T] = r;
                        // the state before the first row of a later chunk's forward sweep
                        if ((i + ov) % kChunkRows == 0 && live) chk[0] = r;
                    } else {
                        sum_r = fma(fabs(row[i].A), sum_r, fabs(u[q]));
                        before *= row[i].A;
                    }
                }
            }
        }
        if (live) {
            chk[ni] = state_limit(sum_r, fabs(before));
            chk[2LL * ni] = state_limit(sum_s, fabs(prod));
        }
    }
    // backward sweep over rows [a, e): the slopes
    double *o0 = A.out + (long long)p * A.os_p;
    const long long plane = (long long)N * ni, os = A.os_i;
    double yr = 0.0;
    const double *bnd = fac + (long long)W * N;
    if (e == N - 1) {
        // row N-2 and the end knot from the last not-a-knot row (interpolate.cu:56-69)
        const long long i = N - 2;
        const double e0 = __ldg(bnd + 4), e1 = __ldg(bnd + 5), dE = __ldg(bnd + 6), hA = __ldg(bnd + 7);
        const double ya = yb[(i - 1) * sk], yl = yb[i * sk], yc = yb[(i + 1) * sk];
        const double sN2 = col[(i - a) * T];
        const double dA = (yl - ya) * __ldg(fac + W * (i - 1) + 6);
        const double ih = __ldg(fac + W * i + 6), xx = __ldg(fac + W * i + 5);
        const double dl = (yc - yl) * ih;
        const double s_last = (e0 * dA + e1 * dl - dE * sN2) / hA;
        if (live) {
            const double tt = (sN2 + s_last - 2 * dl) * ih;
            const double c1 = sN2, c2 = (dl - sN2) * ih - tt, c3 = tt * ih;
            const long long off = i * os, offe = (i + 1) * os;
            __stcs(o0 + off, yl);
            __stcs(o0 + plane + off, c1);
            __stcs(o0 + 2 * plane + off, c2);
            __stcs(o0 + 3 * plane + off, c3);
            // fill_final_derivs (interpolate.cu:241-280)
            __stcs(o0 + offe, yc);
            __stcs(o0 + plane + offe, c1 + 2 * c2 * xx + 3 * c3 * xx * xx);
            __stcs(o0 + 2 * plane + offe, (2. * c2 + 6. * c3 * xx) / 2.);
            __stcs(o0 + 3 * plane + offe, c3);
        }
        s_next = sN2;
        yr = yl;
    } else {
        yr = yb[(long long)e * sk];
    }
    for (int i0 = (e == N - 1 ? N - 3 : e - 1); i0 >= a; i0 -= kAhead) {
        double yv[kAhead];
#pragma unroll
        for (int q = 0; q < kAhead; ++q) yv[q] = yb[(long long)max(i0 - q, a) * sk];
#pragma unroll
        for (int q = 0; q < kAhead; ++q) {
            const int i = i0 - q;
            if (i >= a) {
                const double s = fma(row[i].C, s_next, col[(i - a) * T]);
                // fill_coefficients (interpolate.cu:29-43)
                const double ih = row[i].ih, dl = (yr - yv[q]) * ih;
                const double tt = (s + s_next - 2 * dl) * ih;
                if (live) {
                    const long long off = i * os;
                    __stcs(o0 + off, yv[q]);
                    __stcs(o0 + plane + off, s);
                    __stcs(o0 + 2 * plane + off, (dl - s) * ih - tt);
                    __stcs(o0 + 3 * plane + off, tt * ih);
                }
                yr = yv[q];
                s_next = s;
            }
        }
    }
    if (a == 1 && live) {
        // s_0 from the first row: b0 = gamma0 delta_0 + gamma1 delta_1
        const double g0 = __ldg(bnd + 0), g1 = __ldg(bnd + 1), d0 = __ldg(bnd + 2), h1 = __ldg(bnd + 3);
        const double y0 = yb[0], y1 = yb[sk], y2 = yb[2 * sk];
        const double ih0 = __ldg(fac + 6);
        const double del0 = (y1 - y0) * ih0, del1 = (y2 - y1) * __ldg(fac + W + 6);
        const double s0 = (g0 * del0 + g1 * del1 - d0 * s_next) / h1;
        const double tt = (s0 + s_next - 2 * del0) * ih0;
        o0[0] = y0;
        o0[plane] = s0;
        o0[2 * plane] = (del0 - s0) * ih0 - tt;
        o0[3 * plane] = tt * ih0;
    }
}

int launch_spline_chunks(ChunkArgs a, cudaStream_t st)
{
    constexpr int T = 32 * kChunkWarps;
    const int smem = std::min(a.N - 2, kChunkRows) * T * 8;
    a.groups = (a.ni + 31) / 32;
    const long long blocks = (long long)((spline_chunks(a.N) + kChunkWarps - 1) / kChunkWarps) * a.groups;
    if (blocks > 0x7fffffffLL) return fail(FEW_ERR_SIZE, "spline build: %d series of %d knots are too many", a.ni, a.N);
    k_spline_chunks<<<(unsigned)blocks, T, smem, st>>>(a);
    FEW_LAUNCH_CHECK("k_spline_chunks");
    k_spline_build_factored<true, true><<<a.groups, 32 * kScanChunks, 0, st>>>(
        a.fac, a.y, a.sk, a.sp, a.split, a.off2, a.ni, a.N, a.out, a.os_i, a.os_p, a.chk, a.overlap);
    FEW_LAUNCH_CHECK("k_spline_build_factored");
    return FEW_OK;
}

// One point of one series (CubicSplineInterpolant.__call__'s rules): tv in segment
// ind at xx, o the coefficients' index there.
__device__ __forceinline__ double eval_point(const double *__restrict__ coeffs, long long plane, int ni, int N, int p,
                                             int ind, double xx, bool left, bool right, int deriv)
{
    const long long o = (long long)ind * ni + p;
    const double y = coeffs[o], c1 = coeffs[plane + o], c2 = coeffs[2 * plane + o], c3 = coeffs[3 * plane + o];
    if (deriv == 0) {
        const double x2 = xx * xx, x3 = x2 * xx;
        double v = y + c1 * xx + c2 * x2 + c3 * x3;
        if (left) v = coeffs[p];
        if (right) v = coeffs[(long long)(N - 1) * ni + p];
        return v;
    }
    if (deriv == 1) return c1 + 2 * c2 * xx + 3 * c3 * (xx * xx);
    if (deriv == 2) return 2 * c2 + 6 * c3 * xx;
    return 6 * c3;
}

// searchsorted(x, tv, side="right") - 1 with the last knot mapped to the last
// interval (points before the first knot: interval 0), and whether tv lies outside.
__device__ __forceinline__ int eval_interval(const double *x, int N, double tv, bool &left, bool &right)
{
    int lo = 0, hi = N;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (x[mid] <= tv) lo = mid + 1;
        else hi = mid;
    }
    const double last = x[N - 1];
    left = tv < x[0];
    right = tv > last;
    return tv == last ? N - 2 : max(lo - 1, 0);
}

// Knots or points per series, or few series: a thread per point of one series, the
// interval search (a dozen dependent reads) on knots staged in shared memory (SMEM;
// up to kEvalKnots of them).
constexpr int kEvalThreads = 256;
constexpr int kEvalKnots = 4096;

template <bool SMEM>
__global__ void __launch_bounds__(kEvalThreads) k_spline_eval(const double *__restrict__ t, long long t_rs,
                                                              const double *__restrict__ coeffs, int ni, int N,
                                                              const double *__restrict__ tnew, long long tn_rs, int M,
                                                              int deriv, double *__restrict__ out,
                                                              int *__restrict__ flags)
{
    extern __shared__ __align__(16) double knots[];
    const long long plane = (long long)N * ni;
    for (int p = blockIdx.y; p < ni; p += gridDim.y) {
        const double *x = t + (long long)p * t_rs;
        if (SMEM) {
            __syncthreads();  // the previous series' searches are done
            for (int i = threadIdx.x; i < N; i += kEvalThreads) knots[i] = x[i];
            __syncthreads();
            x = knots;
        }
        for (long long j = (long long)blockIdx.x * kEvalThreads + threadIdx.x; j < M;
             j += (long long)gridDim.x * kEvalThreads) {
            const double tv = tnew[(long long)p * tn_rs + j];
            bool left, right;
            const int ind = eval_interval(x, N, tv, left, right);
            if (left) atomicOr(&flags[0], 1);
            if (right) atomicOr(&flags[1], 1);
            out[(long long)p * M + j] = eval_point(coeffs, plane, ni, N, p, ind, tv - x[ind], left, right, deriv);
        }
    }
}

// Knots and points shared by the series: a CTA takes 32 series (lane = series, so
// that a coefficient row is read in whole lines) and kEvalPoints points, whose
// intervals are searched once; results are turned in shared memory so that each
// series' points are written together.  256 series of 1000 knots at 10,000 points:
// 13 us (25 us with a thread per (series, point), its search in global memory); 2048
// series of 2000 knots at 1900 points: 26 us (60 us).
constexpr int kEvalPoints = 64;
constexpr int kEvalShared = 16;  // fewer series than this leave most lanes idle

__global__ void __launch_bounds__(kEvalThreads) k_spline_eval_shared(const double *__restrict__ t,
                                                                     const double *__restrict__ coeffs, int ni, int N,
                                                                     const double *__restrict__ tnew, int M, int deriv,
                                                                     double *__restrict__ out, int *__restrict__ flags)
{
    __shared__ double s_x[kEvalPoints], s_out[32][kEvalPoints + 1];
    __shared__ int s_ind[kEvalPoints];  // interval, plus kLeft / kRight for a point outside
    constexpr int kLeft = 1 << 30, kRight = 1 << 29, kMask = kRight - 1;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const long long j0 = (long long)blockIdx.x * kEvalPoints;
    const int count = (int)min((long long)kEvalPoints, M - j0);
    if (threadIdx.x < count) {
        const double tv = tnew[j0 + threadIdx.x];
        bool left, right;
        const int ind = eval_interval(t, N, tv, left, right);
        if (left) atomicOr(&flags[0], 1);
        if (right) atomicOr(&flags[1], 1);
        s_ind[threadIdx.x] = ind | (left ? kLeft : 0) | (right ? kRight : 0);
        s_x[threadIdx.x] = tv - t[ind];
    }
    __syncthreads();
    const long long plane = (long long)N * ni;
    for (int p0 = blockIdx.y * 32; p0 < ni; p0 += gridDim.y * 32) {
        const int p = min(p0 + lane, ni - 1);
#pragma unroll 4
        for (int q = w; q < count; q += kEvalThreads / 32) {
            const int ind = s_ind[q];
            s_out[lane][q] = eval_point(coeffs, plane, ni, N, p, ind & kMask, s_x[q], ind & kLeft, ind & kRight, deriv);
        }
        __syncthreads();
        for (int i = threadIdx.x; i < 32 * kEvalPoints; i += kEvalThreads) {
            const int r = i / kEvalPoints, q = i - r * kEvalPoints;
            if (p0 + r < ni && q < count) out[(long long)(p0 + r) * M + j0 + q] = s_out[r][q];
        }
        __syncthreads();
    }
}

}  // namespace

int launch_spline_build(const double *t, long long t_rs, const double *y, long long sk, long long sp, int split,
                        long long off2, int ni, int N, double *out, int layout, cudaStream_t st)
{
    SplineArgs a;
    a.t = t;
    a.t_rs = t_rs;
    a.y = y;
    a.sk = sk;
    a.sp = sp;
    a.off2 = off2;
    a.split = split;
    a.ni = ni;
    a.N = N;
    a.out = out;
    if (layout == FEW_LAYOUT_KNOT_MAJOR) {
        a.os_i = ni;
        a.os_p = 1;
    } else {
        a.os_i = 1;
        a.os_p = N;
    }
    const int threads = 128;
    const size_t smem = (size_t)4 * N * sizeof(double);
    // A CTA per series until the thread form has enough series to fill the chip: it takes
    // 0.8-1.3 us a knot whatever their number, the CTAs 8, 22, 36, 130, 280, 610 and 600 ns
    // a series at 12, 50, 200, 1000, 2000, 4000 and 6000 knots.  Series that the CTAs give
    // up are better swept there, one thread each, while few go to an SM: 256 pulses of
    // 1000 knots 422 us (thread form 2060), 400 of 6000 6.9 ms (12.5); 5000 of 4000 knots
    // 12.5 ms given up and 52 ms swept there (9.8).
    if (ni <= std::min(1024 + 3LL * N, 8000LL) && smem <= kRowSmem) {
        const int per_sm = std::min(16, 228 * 1024 / ((int)smem + 3328));
        const bool give_up = ni > 3 * 148 * per_sm;
        FEW_CUDA_TRY(ensure_smem_attr((const void *)k_spline_build_rows, kRowSmem));
        k_spline_build_rows<<<ni, kRowThreads, smem, st>>>(a, give_up);
        FEW_LAUNCH_CHECK("k_spline_build_rows");
        if (give_up) {
            k_spline_build<true><<<(ni + threads - 1) / threads, threads, 0, st>>>(a);
            FEW_LAUNCH_CHECK("k_spline_build");
        }
        return FEW_OK;
    }
    const int blocks = (ni + threads - 1) / threads;
    k_spline_build<false><<<blocks, threads, 0, st>>>(a);
    FEW_LAUNCH_CHECK("k_spline_build");
    return FEW_OK;
}

}  // namespace few

extern "C" int few_spline_build_factored(const double *fac, const double *y, long long y_knot_stride,
                                         long long y_interp_stride, int y_split, long long y_split_offset, int ninterps,
                                         int length, double *coeffs, int layout, void *stream)
{
    few::clear_error();
    if (!fac || !y || !coeffs) return few::fail(FEW_ERR_ARG, "few_spline_build_factored: null pointer");
    if (ninterps < 1) return few::fail(FEW_ERR_SIZE, "few_spline_build_factored: ninterps=%d < 1", ninterps);
    if (length < 4) return few::fail(FEW_ERR_SIZE, "few_spline_build_factored: length=%d < 4", length);
    if (layout != FEW_LAYOUT_KNOT_MAJOR && layout != FEW_LAYOUT_INTERP_MAJOR)
        return few::fail(FEW_ERR_ARG, "few_spline_build_factored: unknown layout %d", layout);
    if (y_split < 0 || y_split > ninterps) return few::fail(FEW_ERR_ARG, "few_spline_build_factored: bad y_split");
    const long long os_i = layout == FEW_LAYOUT_KNOT_MAJOR ? ninterps : 1;
    const long long os_p = layout == FEW_LAYOUT_KNOT_MAJOR ? 1 : length;
    few::k_spline_build_factored<true, false><<<(ninterps + 31) / 32, 32 * few::kScanChunks, 0, (cudaStream_t)stream>>>(
        fac, y, y_knot_stride, y_interp_stride, y_split, y_split_offset, ninterps, length, coeffs, os_i, os_p, nullptr, 0);
    FEW_LAUNCH_CHECK("k_spline_build_factored");
    return FEW_OK;
}

extern "C" int few_spline_max_overlap(void) { return few::kMaxOverlap; }

extern "C" long long few_spline_joined_scratch(int ninterps, int length)
{
    return ninterps < 1 || length < 4 ? 0 : 3LL * few::spline_chunks(length) * ninterps;
}

namespace few {
namespace {
int check_joined(const char *who, const double *fac, int overlap, const double *y, int y_split, int ninterps, int length,
                 const double *coeffs, int layout)
{
    clear_error();
    if (!fac || !y || !coeffs) return fail(FEW_ERR_ARG, "%s: null pointer", who);
    if (ninterps < 1) return fail(FEW_ERR_SIZE, "%s: ninterps=%d < 1", who, ninterps);
    if (length < 4) return fail(FEW_ERR_SIZE, "%s: length=%d < 4", who, length);
    if (overlap < 1 || overlap > kMaxOverlap)
        return fail(FEW_ERR_SIZE, "%s: overlap=%d out of 1..%d", who, overlap, kMaxOverlap);
    if (layout != FEW_LAYOUT_KNOT_MAJOR && layout != FEW_LAYOUT_INTERP_MAJOR)
        return fail(FEW_ERR_ARG, "%s: unknown layout %d", who, layout);
    if (y_split < 0 || y_split > ninterps) return fail(FEW_ERR_ARG, "%s: bad y_split", who);
    return FEW_OK;
}
}  // namespace
}  // namespace few

extern "C" int few_spline_build_joined(const double *fac, int overlap, const double *y, long long y_knot_stride,
                                       long long y_interp_stride, int y_split, long long y_split_offset, int ninterps,
                                       int length, double *coeffs, int layout, double *scratch, void *stream)
{
    const int rc = few::check_joined("few_spline_build_joined", fac, overlap, y, y_split, ninterps, length, coeffs, layout);
    if (rc) return rc;
    if (!scratch) return few::fail(FEW_ERR_ARG, "few_spline_build_joined: null pointer");
    few::ChunkArgs a{fac, y, y_knot_stride, y_interp_stride, y_split_offset, y_split, ninterps, length, overlap, coeffs,
                     layout == FEW_LAYOUT_KNOT_MAJOR ? ninterps : 1, layout == FEW_LAYOUT_KNOT_MAJOR ? 1 : length,
                     scratch, 0};
    return few::launch_spline_chunks(a, (cudaStream_t)stream);
}

extern "C" int few_spline_build_chunked(const double *fac, int overlap, const double *y, long long y_knot_stride,
                                        long long y_interp_stride, int y_split, long long y_split_offset, int ninterps,
                                        int length, double *coeffs, int layout, void *stream)
{
    int rc = few::check_joined("few_spline_build_chunked", fac, overlap, y, y_split, ninterps, length, coeffs, layout);
    if (rc) return rc;
    cudaStream_t st = (cudaStream_t)stream;
    void *scratch = nullptr;
    FEW_CUDA_TRY(cudaMallocAsync(&scratch, (size_t)few_spline_joined_scratch(ninterps, length) * 8, st));
    rc = few_spline_build_joined(fac, overlap, y, y_knot_stride, y_interp_stride, y_split, y_split_offset, ninterps, length,
                                 coeffs, layout, static_cast<double *>(scratch), stream);
    FEW_CUDA_TRY(cudaFreeAsync(scratch, st));
    return rc;
}

extern "C" int few_spline_slopes(const double *fac, const double *y, int ninterps, int length, double *slopes,
                                 void *stream)
{
    few::clear_error();
    if (!fac || !y || !slopes) return few::fail(FEW_ERR_ARG, "few_spline_slopes: null pointer");
    if (ninterps < 1) return few::fail(FEW_ERR_SIZE, "few_spline_slopes: ninterps=%d < 1", ninterps);
    if (length < 4) return few::fail(FEW_ERR_SIZE, "few_spline_slopes: length=%d < 4", length);
    few::k_spline_build_factored<false, false><<<(ninterps + 31) / 32, 32 * few::kScanChunks, 0, (cudaStream_t)stream>>>(
        fac, y, ninterps, 1, ninterps, 0, ninterps, length, slopes, ninterps, 1, nullptr, 0);
    FEW_LAUNCH_CHECK("k_spline_build_factored");
    return FEW_OK;
}

extern "C" int few_spline_build(const double *t, long long t_row_stride, const double *y, long long y_knot_stride,
                                long long y_interp_stride, int y_split, long long y_split_offset, int ninterps,
                                int length, double *coeffs, int layout, void *stream)
{
    few::clear_error();
    if (!t || !y || !coeffs) return few::fail(FEW_ERR_ARG, "few_spline_build: null pointer");
    if (ninterps < 1) return few::fail(FEW_ERR_SIZE, "few_spline_build: ninterps=%d < 1", ninterps);
    if (length < 4)
        return few::fail(FEW_ERR_SIZE, "few_spline_build: length=%d; not-a-knot splines need at least 4 knots",
                         length);
    if (layout != FEW_LAYOUT_KNOT_MAJOR && layout != FEW_LAYOUT_INTERP_MAJOR)
        return few::fail(FEW_ERR_ARG, "few_spline_build: unknown layout %d", layout);
    if (y_split < 0 || y_split > ninterps) return few::fail(FEW_ERR_ARG, "few_spline_build: bad y_split");
    if ((long long)ninterps * length * 4 > (1LL << 40)) return few::fail(FEW_ERR_SIZE, "few_spline_build: too large");
    return few::launch_spline_build(t, t_row_stride, y, y_knot_stride, y_interp_stride, y_split, y_split_offset,
                                    ninterps, length, coeffs, layout, (cudaStream_t)stream);
}

extern "C" int few_spline_eval(const double *t, long long t_row_stride, const double *coeffs, int ninterps,
                               int length, const double *tnew, long long tnew_row_stride, int M, int deriv_order,
                               double *out, int *flags, void *stream)
{
    few::clear_error();
    if (!t || !coeffs || !tnew || !out || !flags) return few::fail(FEW_ERR_ARG, "few_spline_eval: null pointer");
    if (ninterps < 1 || length < 2 || M < 0) return few::fail(FEW_ERR_SIZE, "few_spline_eval: bad sizes");
    if (deriv_order < 0 || deriv_order > 3)
        return few::fail(FEW_ERR_ARG, "deriv_order must be within 0 <= deriv_order <= 3.");
    if (M == 0) return FEW_OK;
    const long long total = (long long)ninterps * M;
    if ((total + 255) / 256 > 0x7fffffffLL) return few::fail(FEW_ERR_SIZE, "few_spline_eval: too many points");
    cudaStream_t st = (cudaStream_t)stream;
    if (t_row_stride == 0 && tnew_row_stride == 0 && ninterps >= few::kEvalShared && length < (1 << 29)) {
        const dim3 grid((unsigned)(((long long)M + few::kEvalPoints - 1) / few::kEvalPoints),
                        (unsigned)std::min((ninterps + 31) / 32, 65535));
        few::k_spline_eval_shared<<<grid, few::kEvalThreads, 0, st>>>(t, coeffs, ninterps, length, tnew, M, deriv_order,
                                                                      out, flags);
        FEW_LAUNCH_CHECK("k_spline_eval_shared");
        return FEW_OK;
    }
    const long long tiles = ((long long)M + few::kEvalThreads - 1) / few::kEvalThreads;
    const int gy = std::min(ninterps, 65535);
    // the staging of the knots is shared by up to four tiles of points
    const long long gx = std::max((tiles + 3) / 4, std::min(tiles, std::max(1LL, 148LL * 8 / gy)));
    const dim3 grid((unsigned)gx, (unsigned)gy);
    if (length <= few::kEvalKnots && M >= length)
        few::k_spline_eval<true><<<grid, few::kEvalThreads, (size_t)length * 8, st>>>(
            t, t_row_stride, coeffs, ninterps, length, tnew, tnew_row_stride, M, deriv_order, out, flags);
    else
        few::k_spline_eval<false><<<grid, few::kEvalThreads, 0, st>>>(
            t, t_row_stride, coeffs, ninterps, length, tnew, tnew_row_stride, M, deriv_order, out, flags);
    FEW_LAUNCH_CHECK("k_spline_eval");
    return FEW_OK;
}
