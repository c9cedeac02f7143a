// Radius and angles of a direction for the equirectangular projector:
// the float nearest to sqrt(x^2 + y^2 + z^2), atan2(y, x) and asin(z / radius)
// (EquirectangularProjector.cpp:60-99; correctly rounded, as the oracle).
//
// The double-precision atan2, asin and sqrt of the CUDA library are right to
// the last bits of a double, of which a float keeps 24.  Here each value is
// computed in double to about 2^-44 and rounded; only where that error could
// reach the rounding boundary (4 in 10^5 directions) or the arguments are
// extreme do the library's functions decide.  The arctangent follows the
// table-driven scheme (P. T. P. Tang, Table-lookup algorithms for elementary
// functions and their error analysis, 1991): with c = k / 64 nearest to Y / X,
// atan(Y / X) = atan(c) + atan((Y - c X) / (X + c Y)), the second by its series,
// and the arcsine is the arctangent of z over sqrt(1 - z^2).
// Mesh stage of 4 x ERP 4096x2048 into ERP 4096x2048 (33.5 M directions): 1093
// -> 1055 us; every float equal.
#pragma once

#include <cuda_runtime.h>

namespace rvsb {
namespace dev {

__device__ const double kAtan64[65] = {
    0.0, 0.015623728620476831, 0.031239833430268277, 0.046840712915969654,
    0.06241880999595735, 0.0779666338315423, 0.09347678115858947, 0.10894195698986579,
    0.12435499454676144, 0.13970887428916365, 0.15499674192394097, 0.1702119252854744,
    0.18534794999569476, 0.2003985538258785, 0.21535769969773805, 0.23021958727684372,
    0.24497866312686414, 0.2596296294082575, 0.2741674511196588, 0.2885873618940774,
    0.3028848683749714, 0.31705575320914703, 0.3310960767041321, 0.34500217720710513,
    0.35877067027057225, 0.3723984466767542, 0.38588266939807375, 0.39922076957525254,
    0.4124104415973873, 0.42544963737004227, 0.43833655985795783, 0.4510696559885235,
    0.4636476090008061, 0.4760693303227612, 0.48833395105640554, 0.5004408131472942,
    0.5123894603107377, 0.5241796287829132, 0.5358112379604637, 0.5472843809874369,
    0.5585993153435624, 0.5697564534829784, 0.5807563535676704, 0.5915997103351114,
    0.6022873461349642, 0.6128202021652414, 0.6231993299340659, 0.6334258829691446,
    0.6435011087932844, 0.6534263411807619, 0.6632029927060933, 0.6728325475937632,
    0.6823165548747481, 0.6916566218531999, 0.7008544078844502, 0.7099116184635249,
    0.7188299996216245, 0.7276113326265107, 0.7362574289814281, 0.7447701257160751,
    0.7531512809621944, 0.7614027698055784, 0.7695264804056583, 0.7775243103733478,
    0.7853981633974483};

// Direct evaluation, the values the fast one must reproduce.
static __device__ __noinline__ void erp_direction_exact(float x, float y, float z, float& radius, float& phi,
                                                        float& theta) {
    double s2 = 0.0;
    s2 = __dadd_rn(s2, __dmul_rn((double)x, (double)x));
    s2 = __dadd_rn(s2, __dmul_rn((double)y, (double)y));
    s2 = __dadd_rn(s2, __dmul_rn((double)z, (double)z));
    radius = (float)__dsqrt_rn(s2);
    phi = (float)atan2((double)y, (double)x);
    theta = (float)asin((double)__fdiv_rn(z, radius));
}

// Whether a double within 2^-41 (relative) of a value rounds to the same
// float as it: the 29 bits a float drops are not within 2^12 of half.
__device__ __forceinline__ bool rounds_safely(double v) {
    return (((unsigned)__double2loint(v) - 0x0ffff000u) & 0x1fffffffu) > 0x2000u;
}

// sqrt(v) for v in [1e-30, 1e30] to about 2^-45: the approximate float
// reciprocal root and one Newton step in double.
__device__ __forceinline__ double sqrt45(double v) {
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"((float)v));
    const double h = v * (double)y;
    return __fma_rn(0.5 * h, __fma_rn(-h, (double)y, 1.0), h);
}

// atan(Y / X) for 0 < Y <= X to about 2^-44.
__device__ __forceinline__ double atan44(double Y, double X) {
    float rx, rd;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(rx) : "f"((float)X));
    // Held to the table whatever X and Y are (subnormals make rx infinite, a
    // vanishing root NaN); the caller discards the result of such arguments.
    const float k = fminf(rintf((float)Y * rx * 64.f), 64.f);
    const double c = (double)(k * 0.015625f);
    const double num = __fma_rn(-c, X, Y), den = __fma_rn(c, Y, X);
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(rd) : "f"((float)den));
    const double r0 = (double)rd;
    const double r = num * __fma_rn(r0, __fma_rn(-den, r0, 1.0), r0);
    const double s = r * r;
    // |r| <= 1/127: the next term of the series is below 2^-44 of the first.
    return __ldg(kAtan64 + (int)k) + __fma_rn(r * s, __fma_rn(s, 0.2, -1.0 / 3.0), r);
}

__device__ __forceinline__ void erp_direction(float x, float y, float z, float& radius, float& phi, float& theta) {
    const double dx = (double)x, dy = (double)y, dz = (double)z;
    const float ax = fabsf(x), ay = fabsf(y), az = fabsf(z);
    bool ok = fmaxf(ax, fmaxf(ay, az)) <= 1e15f && fminf(ax, fminf(ay, az)) >= 1e-15f;
    const double s2 = __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz));
    const double rad = sqrt45(s2);
    radius = (float)rad;
    const bool steep = ay > ax;
    double p = atan44((double)(steep ? ax : ay), (double)(steep ? ay : ax));
    p = steep ? 1.5707963267948966 - p : p;
    p = x < 0.f ? 3.141592653589793 - p : p;
    phi = copysignf((float)p, y);
    const float t = fabsf(__fdiv_rn(z, radius));
    const double dt = (double)t, w = __fma_rn(-dt, dt, 1.0);
    ok = ok && w > 1e-8;
    const double g = sqrt45(w);
    const bool high = dt > g;
    double q = atan44(high ? g : dt, high ? dt : g);
    q = high ? 1.5707963267948966 - q : q;
    theta = copysignf((float)q, z);
    if (!(ok && rounds_safely(rad) && rounds_safely(p) && rounds_safely(q)))
        erp_direction_exact(x, y, z, radius, phi, theta);
}

}  // namespace dev
}  // namespace rvsb
