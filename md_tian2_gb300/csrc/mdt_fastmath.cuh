// mdt_fastmath.cuh -- FP32 building blocks of the fast force kernels (mdt_nnf.cu,
// mdt_nnr.cu): the cosine cutoff as a polynomial in s = r^2/rc^2, hardware 2^x / log2 /
// reciprocal approximations, the softplus activation with its derivative from one
// exponential, and shared-memory float reductions.
#pragma once
#include <cstdint>

#include "mdt_common.cuh"
#include "mdt_convert.h"
#include "mdt_exp2tab.cuh"

namespace mdt {

// Cosine cutoff fc = (cos(pi r/rc) + 1)/2 = c^2 with c = cos(pi sqrt(s)/2), s = r^2/rc^2.
// c is the Taylor series sum_n (-pi^2 s/4)^n / (2n)! truncated after n = 7 (remainder
// below 1e-10 on [0, 1], alternating terms no larger than 1.24, so FP32 Horner loses
// little), and fc = c^2 keeps the absolute error vanishing at the cutoff.
constexpr double half_cos_sqrt_coef(int n) {
    double c = 1.0;
    for (int k = 1; k <= n; ++k) c *= -(kPi * kPi / 4.0) / ((2.0 * k - 1.0) * (2.0 * k));
    return c;
}
constexpr float kCs0 = (float)half_cos_sqrt_coef(0), kCs1 = (float)half_cos_sqrt_coef(1),
                kCs2 = (float)half_cos_sqrt_coef(2), kCs3 = (float)half_cos_sqrt_coef(3),
                kCs4 = (float)half_cos_sqrt_coef(4), kCs5 = (float)half_cos_sqrt_coef(5),
                kCs6 = (float)half_cos_sqrt_coef(6), kCs7 = (float)half_cos_sqrt_coef(7);

// fc(s)
__device__ __forceinline__ float fc_of_s(float s) {
    float c = kCs7;
    c = fmaf(c, s, kCs6);
    c = fmaf(c, s, kCs5);
    c = fmaf(c, s, kCs4);
    c = fmaf(c, s, kCs3);
    c = fmaf(c, s, kCs2);
    c = fmaf(c, s, kCs1);
    c = fmaf(c, s, kCs0);
    return c * c;
}

// fc(s) and dfc/ds = 2 c c'(s) (Horner with derivative)
__device__ __forceinline__ void fc_of_s_d(float s, float &fc, float &dfds) {
    float c = kCs7, d = 0.f;
#define MDT_STEP(k)        \
    d = fmaf(d, s, c);     \
    c = fmaf(c, s, k);
    MDT_STEP(kCs6) MDT_STEP(kCs5) MDT_STEP(kCs4) MDT_STEP(kCs3) MDT_STEP(kCs2) MDT_STEP(kCs1) MDT_STEP(kCs0)
#undef MDT_STEP
    fc = c * c;
    dfds = 2.f * c * d;
}

// 2^x (hardware approximation, relative error about 2^-22; results below the FP32
// normal range flush to zero, far below any radial function that matters)
__device__ __forceinline__ float ex2a(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// log2(x) for x in [1, 2] (hardware approximation, absolute error about 2^-22)
__device__ __forceinline__ float lg2a(float x) {
    float y;
    asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// 1/x (hardware approximation, about 1 ulp)
__device__ __forceinline__ float rcpa(float x) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

constexpr float kLog2eF = 1.4426950408889634f;
constexpr float kLn2F = 0.6931471805599453f;

// softplus v = log(1 + e^z) and its derivative dv/dz = 1/(1 + e^-z) in the form that
// cannot overflow: v = max(z, 0) + log(1 + e^-|z|), one exponential for both.
__device__ __forceinline__ void softplus_d(float z, float &v, float &dv) {
    const float e = ex2a(-fabsf(z) * kLog2eF);
    const float d = 1.f + e;
    v = fmaf(lg2a(d), kLn2F, fmaxf(z, 0.f));
    const float r = rcpa(d);
    dv = z >= 0.f ? r : e * r;
}

__device__ __forceinline__ void red_shared(float *p, float v) {
    const unsigned a = (unsigned)__cvta_generic_to_shared(p);
    asm volatile("red.shared.add.f32 [%0], %1;" ::"r"(a), "f"(v) : "memory");
}

// x in FP32 for range decisions (a screen whose undecided values go to FP64): to the nearest, halves
// away from zero, |x| < 2^-126 as 0, |x| >= 2^127, infinities and NaN as infinity.  f32_of
// (mdt_convert.h) without its rare branch, which the pair loops would carry three times.
static __device__ __forceinline__ float f32_screen(double x) {
    const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
    const unsigned e = hi & 0x7ff00000u;
    const unsigned m = ((__funnelshift_l(lo, hi, 3) ^ 0x40000000u) & 0x7fffffffu) + (lo >> 28 & 1u);
    const unsigned v = e < 0x38100000u ? 0u : e >= 0x47e00000u ? 0x7f800000u : m;
    return __uint_as_float(v | (hi & 0x80000000u));
}

// exponent of the largest magnitudes: infinity or NaN (a FP64 comparison runs on the FP64 pipe)
static __device__ __forceinline__ bool not_finite(double x) {
    return (__double2hiint(x) & 0x7ff00000) == 0x7ff00000;
}

// ---- FP64 building blocks ------------------------------------------------------------
static __device__ __forceinline__ double rcp_nr(double x) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = fma(-x, y, 1.0);  // 1/x = y (1 + e + e^2 + ...)
    return fma(y, fma(e, e, e), y);
}

static __device__ __forceinline__ double rsqrt_nr(double x) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = fma(-x, y * y, 1.0);  // 1/sqrt(x) = y (1 + e/2 + 3 e^2/8 + ...)
    return fma(y * e, fma(e, 0.375, 0.5), y);
}

// Distance r of r2 = r^2, and 1/r.  Two atoms on one site (r2 = 0, or too small for the approximation) have r = 0 and
// 1/r infinite as by sqrt and division, so that the forces between them are not finite numbers.
static __device__ __noinline__ double2 dist_rare(double r2) {
    const double r = sqrt(r2);
    return make_double2(r, 1.0 / r);
}
static __device__ __forceinline__ double dist_of(double r2, double &inv) {
    if ((unsigned)__double2hiint(r2) < 0x00100000u) {
        const double2 d = dist_rare(r2);
        inv = d.y;
        return d.x;
    }
    inv = rsqrt_nr(r2);
    return r2 * inv;
}

// n/d from the reciprocal id of d (within an ulp or two): the residual's correction makes the
// quotient round as a division does, in 3 FP64 instructions instead of about 10
static __device__ __forceinline__ double div_by(double n, double d, double id) {
    const double q = n * id;
    return fma(fma(-q, d, n), id, q);
}

// Rare paths of the pair loops are calls: inlined, the compiler predicates their FP64 instructions
// and every pair issues them.
static __device__ __noinline__ double exp_far(double x) { return exp(x); }

// FP64 exp by the table-driven method of Tang (ACM TOMS 15(2), 1989): x = (512 n_hi + j)
// ln2/512 + r with |r| <= ln2/1024, exp(x) = 2^n_hi 2^(j/512) (1 + p(r)), p the Taylor series
// of exp(r) - 1 to r^4 (truncation below 2^-59).  ln2/512 enters in two parts (its double,
// then the remainder) so that r is exact to ~2^-100, and n = round(512 x / ln2) comes from
// adding 1.5 * 2^52.  10 FP64 instructions (13 with 64 entries and r^5, ~19 for exp()); the
// range test reads the high word, because a FP64 comparison costs as much as an addition.
// Outside [-700, 700], and for NaN, exp() itself.
static __device__ __forceinline__ double exp_t64(double x) {
    if ((__double2hiint(x) & 0x7fffffff) >= 0x4085e000) return exp_far(x);  // |x| >= 700
    const double shifter = 6755399441055744.0;
    const double t = fma(x, 738.65986093514926, shifter);
    const int n = __double2loint(t);
    const double nd = t - shifter;
    double r = fma(-nd, 0x1.62e42fefa39efp-10, x);
    r = fma(-nd, 0x1.abc9e3b39803fp-65, r);
    double q = fma(r, 1.0 / 24.0, 1.0 / 6.0);
    q = fma(r, q, 0.5);
    const double pr = fma(r * r, q, r);
    const double tj = __ldg(kExp2Tab + (n & 511));
    const double y = fma(tj, pr, tj);
    return __hiloint2double(__double2hiint(y) + (n >> 9) * (1 << 20), __double2loint(y));
}

}  // namespace mdt
