// Shared device helpers for the B200 interpolated mode sum.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "few_b200.h"

namespace few {

// Nanoseconds of the GPU's global timer.
__device__ __forceinline__ unsigned long long global_ns()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// ---------------------------------------------------------------------------
// Complex FP64 helpers (double2: x = real, y = imaginary).  These are ordinary
// FP64 expressions; nvcc may contract them into FMAs, which is intended.
// ---------------------------------------------------------------------------
__device__ __forceinline__ double2 cmul(double2 a, double2 b)
{
    return make_double2(fma(a.x, b.x, -a.y * b.y), fma(a.x, b.y, a.y * b.x));
}
__device__ __forceinline__ double2 cconj(double2 a) { return make_double2(a.x, -a.y); }
__device__ __forceinline__ double2 cadd(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }

// a * (1 + i e) for a tiny angle e (first order of exp(i e); |e| < 1e-8 keeps
// the dropped e^2/2 term below 1e-16).
__device__ __forceinline__ double2 crot_small(double2 a, double e)
{
    return make_double2(fma(-a.y, e, a.x), fma(a.x, e, a.y));
}

// z^p for an integer p by binary powering (conjugate base for p < 0).
__device__ __forceinline__ double2 cpow_int(double2 z, int p)
{
    if (p < 0) {
        z = cconj(z);
        p = -p;
    }
    double2 r = make_double2(1.0, 0.0);
    while (p) {
        if (p & 1) r = cmul(r, z);
        p >>= 1;
        if (p) z = cmul(z, z);
    }
    return r;
}

// ---------------------------------------------------------------------------
// Exactly rounded operations used where the reference's rounding is replayed.
// The intrinsics stop nvcc from contracting a*b+c into one FMA.
// ---------------------------------------------------------------------------
__device__ __forceinline__ double rmul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double radd(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double rsub(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ double rdiv(double a, double b) { return __ddiv_rn(a, b); }

// Error of the rounded sum s = fl(a + b): a + b = s + err exactly (Knuth's TwoSum).
__device__ __forceinline__ double two_sum_err(double a, double b, double s)
{
    double bb = __dsub_rn(s, a);
    return __dadd_rn(__dsub_rn(a, __dsub_rn(s, bb)), __dsub_rn(b, bb));
}

// sin and cos of a large angle: Cody & Waite reduction mod 2 pi (2 pi split in
// three parts, k*C1 and k*C2 exact for |k| < 2^21), then sincos on |r| <= pi,
// which stays on the function's short path (large arguments take its slow,
// table-driven reduction).
__device__ __forceinline__ void sincos_reduced(double ph, double *s, double *c)
{
    const double kInv2Pi = 0.15915494309189535;
    const double kC1 = 0x1.921fb54400000p+2, kC2 = 0x1.0b4611a600000p-32, kC3 = 0x1.3198a2e037073p-67;
    double r = ph;
    const double kq = rint(ph * kInv2Pi);
    if (fabs(kq) < 2097152.0) {
        r = __fma_rn(-kq, kC1, ph);
        r = __fma_rn(-kq, kC2, r);
        r = __fma_rn(-kq, kC3, r);
    }
    sincos(r, s, c);
}

// sin and cos of an angle of any size met in a phase (|ph| < kPhaseMax), both to
// about an ulp: the angle is reduced mod pi/2 by Cody & Waite's method (pi/2 in
// three parts of 32, 32 and 53 bits; with fused multiply-adds the first
// difference is exact for every such angle, being a multiple of 2^-31 below 1
// or of ph's own last place), then Taylor's series on |r| <= pi/4, whose first
// dropped terms (r^19/19!, r^18/18!) are below 1e-19 and 3e-18.  A third fewer
// FP64 operations than a reduction mod 2 pi followed by sincos, which reduces
// again.
constexpr double kPhaseMax = 1073741824.0;  // 2^30

__device__ __forceinline__ void sincos_phase_core(double ph, double *s, double *c)
{
    const double kMagic = 6755399441055744.0;  // 1.5 * 2^52: the sum's low word is the rounded integer
    const double kC1 = 0x1.921fb54400000p+0, kC2 = 0x1.0b4611a600000p-34, kC3 = 0x1.3198a2e037073p-69;
    const double km = __fma_rn(ph, 0.63661977236758134, kMagic);
    const int q = __double2loint(km);
    const double k = __dsub_rn(km, kMagic);
    double r = __fma_rn(-k, kC1, ph);
    r = __fma_rn(-k, kC2, r);
    r = __fma_rn(-k, kC3, r);
    const double z = r * r;
    double p = 1.0 / 355687428096000.0;
    p = __fma_rn(p, z, -1.0 / 1307674368000.0);
    p = __fma_rn(p, z, 1.0 / 6227020800.0);
    p = __fma_rn(p, z, -1.0 / 39916800.0);
    p = __fma_rn(p, z, 1.0 / 362880.0);
    p = __fma_rn(p, z, -1.0 / 5040.0);
    p = __fma_rn(p, z, 1.0 / 120.0);
    p = __fma_rn(p, z, -1.0 / 6.0);
    const double sn = __fma_rn(r * z, p, r);
    double u = 1.0 / 20922789888000.0;
    u = __fma_rn(u, z, -1.0 / 87178291200.0);
    u = __fma_rn(u, z, 1.0 / 479001600.0);
    u = __fma_rn(u, z, -1.0 / 3628800.0);
    u = __fma_rn(u, z, 1.0 / 40320.0);
    u = __fma_rn(u, z, -1.0 / 720.0);
    u = __fma_rn(u, z, 1.0 / 24.0);
    const double hz = 0.5 * z, w = 1.0 - hz;
    const double cn = w + __fma_rn(z * z, u, (1.0 - w) - hz);
    const double a = (q & 1) ? cn : sn, b = (q & 1) ? sn : cn;
    // the quadrant's signs, into the sign bits
    *s = __hiloint2double(__double2hiint(a) ^ ((q & 2) << 30), __double2loint(a));
    *c = __hiloint2double(__double2hiint(b) ^ (((q + 1) & 2) << 30), __double2loint(b));
}

// The same for any angle: larger and non-finite ones go to sincos.
__device__ __forceinline__ void sincos_phase(double ph, double *s, double *c)
{
    if (fabs(ph) < kPhaseMax) sincos_phase_core(ph, s, c);
    else sincos(ph, s, c);
}

// The 8-term dense-output phase polynomial in s, s1 = 1 - s, in the
// operation order of src/few/cutils/interpolate.cu:642-644, every product and
// sum rounded separately.
__device__ __forceinline__ double phase_poly(const double *c, double s, double s1)
{
    double a = rmul(s, c[7]);
    a = rmul(s1, radd(c[6], a));
    a = rmul(s, radd(c[5], a));
    a = rmul(s1, radd(c[4], a));
    a = rmul(s, radd(c[3], a));
    a = rmul(s1, radd(c[2], a));
    a = rmul(s, radd(c[1], a));
    return radd(c[0], a);
}

}  // namespace few
