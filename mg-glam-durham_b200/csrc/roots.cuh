// Roots of the cells' equations: the cubic of f(R) n = 1 and the symmetron, the quartic
// of f(R) n = 2.  The functions compile for the host too (the special-function unit's
// approximations become their plain counterparts), so that tests reach them alone.
#pragma once
#include <cuda_runtime.h>
#include <cmath>

namespace mgg {

namespace {

__host__ __device__ __forceinline__ float nan32() {
#ifdef __CUDA_ARCH__
    return __int_as_float(0x7fffffff);
#else
    return NAN;
#endif
}

// cube root with the sign of x (the reference's DSIGN(DABS(x)**(1/3), x))
__host__ __device__ __forceinline__ double scbrt(double x) { return cbrt(x); }

// Roots of the depressed cubic u^3 + P u + Q = 0 as the reference selects them
// (PMP2MGsolver_fR.f90:165-179, PMP2MGsolver_sym.f90:110-129), with
// D0 = -3P, D1 = 27Q, CC = D1^2 - 4 D0^3:
//   CC >= 0 : Cardano, u = -(cbrt(t1) - cbrt(t2))/3, t1 = (sqrt(CC) + D1)/2, t2 = t1 - D1
//   CC <  0 : u = -(2/3) sqrt(D0) cos(acos(c)/3 + 2 pi/3), c = D1 / (2 D0^(3/2))
// Each root is evaluated as an FP32 seed of the same closed form and refined by
// two chord-Newton steps on the cubic in FP64.  Cardano's seed uses
// cbrt(t1) cbrt(t2) = -D0: with T = (D1 + sign(D1) sqrt(CC))/2 (no cancellation)
// and C = cbrt(T), u = -(C + D0/C)/3, so one cube root, taken as
// exp2(log2|T|/3) on the special-function unit, gives a seed with relative
// error ~1e-6.  The chord slope 3u0^2 + P is of order |P| or larger away from
// a double root, so each step multiplies the relative error by ~1e-6 and the
// result equals the closed form to FP64 rounding.  Whenever the seed is not
// finite, leaves [1e-15, 1e15], or sits near a double root, the FP64 closed
// form itself is evaluated.
__host__ __device__ __forceinline__ bool f32_ok(float v) {
    const float a = fabsf(v);
    return a < 1.0e30f && (a > 1.0e-30f || a == 0.0f);
}

// Special-function-unit approximations (PTX *.approx.ftz.f32, relative error
// ~2^-22; subnormal inputs and results flush to zero), used only for seeds
// that are refined in FP64 or checked and replaced
__host__ __device__ __forceinline__ float ex2_approx(float x) {
#ifdef __CUDA_ARCH__
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
#else
    return exp2f(x);
#endif
}
__host__ __device__ __forceinline__ float lg2_approx(float x) {
#ifdef __CUDA_ARCH__
    float y;
    asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
#else
    return log2f(x);
#endif
}
__host__ __device__ __forceinline__ float rcp_approx(float x) {
#ifdef __CUDA_ARCH__
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
#else
    return 1.0f / x;
#endif
}
__host__ __device__ __forceinline__ float rsqrt_approx(float x) {
#ifdef __CUDA_ARCH__
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
#else
    return 1.0f / sqrtf(x);
#endif
}

__host__ __device__ __forceinline__ double chord_refine(double u, double P, double Q) {
    const float uf = (float)u;
    const float fp = 3.0f * uf * uf + (float)P;
    const double r = (double)rcp_approx(fp);   // chord slope: any close value converges
#pragma unroll
    for (int it = 0; it < 2; ++it) {
        const double f = fma(u * u + P, u, Q);
        u = fma(-f, r, u);
    }
    return u;
}

__host__ __device__ __attribute__((noinline)) double cardano_fp64(double CC, double D1) {
    const double tmp1 = 0.5 * (sqrt(CC) + D1);
    const double tmp2 = tmp1 - D1;
    return -(scbrt(tmp1) - scbrt(tmp2)) * (1.0 / 3.0);
}

__host__ __device__ __attribute__((noinline)) double trig_fp64(double D0, double D1) {
    const double sq = sqrt(D0);
    const double S = acos(0.5 * D1 / (sq * sq * sq));
    return -(2.0 / 3.0) * sq * cos(S * (1.0 / 3.0) + 2.0 / 3.0 * 3.141592653589793);
}

__host__ __device__ __forceinline__ double cardano_root(double P, double Q, double CC, double D0, double D1) {
    const float D0f = (float)D0, D1f = (float)D1, CCf = (float)CC;
    const float sf = CCf * rsqrt_approx(CCf);               // sqrt(CC) (CC > 0; CC = 0 gives NaN -> FP64)
    const float T = 0.5f * (D1f >= 0.0f ? D1f + sf : D1f - sf);
    const float C = copysignf(ex2_approx(lg2_approx(fabsf(T)) * (1.0f / 3.0f)), T);
    const float u0 = -(C + D0f * rcp_approx(C)) * (1.0f / 3.0f);
    const float au = fabsf(u0);
    const float fp = 3.0f * u0 * u0 + (float)P;
    if (!(au > 1.0e-15f && au < 1.0e15f && fabsf(fp) > 3.0e-3f * u0 * u0)) return cardano_fp64(CC, D1);
    return chord_refine((double)u0, P, Q);
}

__host__ __device__ __forceinline__ double trig_root(double P, double Q, double D0, double D1) {
    const float Pf = (float)P, Qf = (float)Q;
    const float sqf = sqrtf(-3.0f * Pf);
    const float cf = 0.5f * (27.0f * Qf) / (sqf * sqf * sqf);
    if (!(f32_ok(Pf) && f32_ok(Qf) && f32_ok(sqf * sqf * sqf) && cf > -1.0f && cf < 0.9f)) return trig_fp64(D0, D1);
    const float y = cosf(acosf(cf) * (1.0f / 3.0f) + 2.09439510239f);
    return chord_refine((double)(-(2.0f / 3.0f) * sqf * y), P, Q);
}

// The largest root of u^3 + P u + Q = 0 (f(R) n = 1 and symmetron) by Newton's
// method in FP32, from the cell's current value: the precision form's root and
// the plain path's seed.  That is the root the reference's closed form returns: Cardano's
// single real root when CC >= 0, and for CC < 0 the trigonometric form
// -(2/3) sqrt(-3P) cos(acos(c)/3 + 2 pi/3), which lies in
// [sqrt(-P/3), 2 sqrt(-P/3)], right of the local minimum.
// To the right of the local minimum (3u^2 + P > 0) the cubic is convex, so
// Newton converges to that root from any such start, quadratically with
// eps' <= 3.3 eps^2 while 3u^2 + P >= 0.9 u^2: a step below 1e-4 u leaves an
// error below FP32 rounding.  Returns NaN when the start is outside that region
// or five steps do not converge; the caller then takes the FP64 closed form.
__host__ __device__ __forceinline__ float cubic_root_newton32(float u, float P, float Q) {
    if (!(u > 0.0f && u < 1.0e15f && fmaf(2.1f * u, u, P) > 0.0f)) return nan32();
#pragma unroll 1
    for (int it = 0; it < 5; ++it) {
        const float fp = fmaf(3.0f * u, u, P);
        const float f = fmaf(fmaf(u, u, P), u, Q);
        const float du = f * rcp_approx(fp);
        u = u - du;
        if (fabsf(du) <= 1.0e-4f * u) return u;
    }
    return nan32();
}

// f(R) n = 2: the positive root of u^4 + P u + Q = 0 (Q < 0),
// the root the reference's Ferrari closed form returns, by Newton's method in
// FP32 from the cell's current value.  The quartic is convex with one positive
// root; right of its minimum (4u^3 + P > 0) Newton converges from any start,
// with eps' <= 5 eps^2 while 4u^3 + P >= 1.2 u^3.  NaN when the start is
// unusable or five steps do not converge.
__host__ __device__ __forceinline__ float quartic_root_newton32(float u, float P, float Q) {
    if (!(u > 0.0f && u < 1.0e10f && fmaf(2.8f * u * u, u, P) > 0.0f)) return nan32();
#pragma unroll 1
    for (int it = 0; it < 5; ++it) {
        const float u2 = u * u;
        const float fp = fmaf(4.0f * u2, u, P);
        const float f = fmaf(fmaf(u2, u, P), u, Q);
        const float du = f * rcp_approx(fp);
        u = u - du;
        if (fabsf(du) <= 1.0e-4f * u) return u;
    }
    return nan32();
}

// FP64 root of the plain path from an FP32 seed u0 by two chord steps.  The seed's error
// e0 is FP32 rounding of terms up to 9 u^3 over the slope f' (cubic; the quartic with one
// more power of u), so below 1e-6 where f' > u^2; a chord step multiplies an error by
// about 6 e0 u^2 / f', so two leave FP64 rounding.  Returns NaN where the slope is smaller
// (towards a double root, where two steps do not do: that takes Q > 0, which the
// symmetron's coarse levels can have) or negative (not the largest root), and where
// FP32 underflow may have spoilt the seed (u^3 or u^4 below 1e-30).
template <bool QUARTIC>
__host__ __device__ __forceinline__ double refine_seed(float u0, double P, double Q) {
    const float u2 = u0 * u0;
    const float fp = QUARTIC ? fmaf(4.0f * u2, u0, (float)P) : fmaf(3.0f, u2, (float)P);
    if (!(u0 > (QUARTIC ? 3.0e-8f : 1.0e-10f) && fp > (QUARTIC ? u2 * u0 : u2))) return (double)nan32();
    const double r = (double)rcp_approx(fp);
    double u = (double)u0;
#pragma unroll
    for (int it = 0; it < 2; ++it) {
        const double f = QUARTIC ? fma(fma(u * u, u, P), u, Q) : fma(fma(u, u, P), u, Q);
        u = fma(-f, r, u);
    }
    return u;
}

// The closed forms for the rare cells without a usable FP32 root, out of line:
// inlined into every cell of the fused sweep they took its registers and most of
// its code.  third: the root at P = 0.
__host__ __device__ __attribute__((noinline)) double cubic_root_cold(double P, double Q, double D1, double third) {
    const double D0 = -3.0 * P;
    const double CC = D1 * D1 - 4.0 * D0 * D0 * D0;
    if (CC >= 0.0) {
        if (fabs(P) < 1.0e-20) return third;
        return cardano_root(P, Q, CC, D0, D1);
    }
    return trig_root(P, Q, D0, D1);
}
__host__ __device__ __attribute__((noinline)) double sym_root_cold(double P, double Q) { return cubic_root_cold(P, Q, 27.0 * Q, -scbrt(Q)); }
__host__ __device__ __attribute__((noinline)) double quartic_root_cold(double P, double Q, double D20) {
    const double Delta21 = 27.0 * P * P;
    const double tmp1 = 0.5 * (sqrt(Delta21 * Delta21 - 4.0 * D20 * D20 * D20) + Delta21);
    const double cr = scbrt(tmp1);
    const double S = sqrt(cr + D20 / cr) / sqrt(12.0);
    if (P > 1.0e-20) return -S + 0.5 * sqrt(-4.0 * S * S + P / S);
    if (P < -1.0e-20) return S + 0.5 * sqrt(-4.0 * S * S - P / S);
    return sqrt(sqrt(-Q));
}

// The plain path's cubic (quartic) root from the cell's current value: the FP32
// Newton root refined in FP64, else (NaN) the closed form.  The value is the closed
// form's to FP64 rounding at a third of its instructions.
template <bool QUARTIC>
__host__ __device__ __forceinline__ double root_from(float uold, double P, double Q) {
    const float seed = QUARTIC ? quartic_root_newton32(uold, (float)P, (float)Q)
                               : cubic_root_newton32(uold, (float)P, (float)Q);
    return refine_seed<QUARTIC>(seed, P, Q);
}

}  // namespace

}  // namespace mgg
