// Resolve and blend of one output pixel, used by the resolve kernel once a
// view's z-buffer is final: re-evaluate the winning fragment exactly, fold it
// into the running blend in blend order (BlendedViewSimple::blendBasicMode +
// blend_img, BlendedView.cpp:180-212, blending.cpp:310-369).
#pragma once

#include "device_common.cuh"

namespace rvsb {
namespace dev {

struct Fragment {
    float3 col;
    float depth;      // +inf when uncovered
    float validity;   // triangle quality, 0 when uncovered
};

// m * scale for an integer m below 2^23 sitting in the mantissa of 2^23 (bits:
// 0x4B000000 | m): the fused multiply-add takes the 2^23 off exactly, so the
// result is the product rounded once, as __fmul_rn((float)m, scale).
__device__ __forceinline__ float scaled_mantissa(uint32_t bits, float scale, float offset) {
    return __fmaf_rn(__uint_as_float(bits), scale, offset);
}

// Colour word `k` of a view: float3(Y * s, U * s, V * s) as input_color.
// 4U * 0.25 * s is 4U * (s / 4): scaling by a power of two rounds nothing.  V
// is taken where it lies, 4 bits up (16 * 4V, scaled by s / 64).
template <class View>
__device__ __forceinline__ float3 packed_color(const View& V, uint32_t k) {
    const uint2 c = __ldg(reinterpret_cast<const uint2*>(V.color) + k);
    const float cs = V.color_scale, two23 = -8388608.f;
    const uint32_t one = 0x4B000000u;
    float3 r;
    r.x = scaled_mantissa(one | (c.x & 0x3ffffu), cs, two23 * cs);
    r.y = scaled_mantissa(one | (__funnelshift_r(c.x, c.y, 18) & 0x3ffffu), 0.25f * cs, two23 * (0.25f * cs));
    r.z = scaled_mantissa(one | (c.y & 0x3ffff0u), 0.015625f * cs, two23 * (0.015625f * cs));
    return r;
}

// Squared length of (dx, dy) as the unevaluated sum of two floats, exact to
// about 2^-46.
__device__ __forceinline__ float2 sq_len2(float dx, float dy) {
    const float p = __fmul_rn(dx, dx), q = __fmul_rn(dy, dy);
    const float ep = __fmaf_rn(dx, dx, -p), eq = __fmaf_rn(dy, dy, -q);
    const float hi = __fadd_rn(p, q);
    // two-sum (Knuth): hi + e = p + q exactly
    const float t = __fsub_rn(hi, p);
    const float e = __fadd_rn(__fsub_rn(p, __fsub_rn(hi, t)), __fsub_rn(q, t));
    return make_float2(hi, __fadd_rn(e, __fadd_rn(ep, eq)));
}

// tri_quality (device_common.cuh) without double arithmetic, the same float:
// the longest edge is picked by its squared length in float where that decides
// it, its squared length kept to about 46 bits, and an approximate square root
// corrected by one Newton step from the remainder.  Root and correction
// together are within 2^-43 of the root (2^-46 from the square, 2^-45 each
// from the remainder's rounding and from taking 0.5 * y, 2^-22 off, for half
// the reciprocal root); the sum is rounded to float with 2^-40 added and taken
// off, and where the two differ (1 in 2^16 roots), edges tie (to 2^-20) or are
// tiny, the double evaluation runs.  With the colour unpacking and the blend's
// powers below: 94 -> 86.6 M warp instructions, 123 -> 117 us on 4 views of
// 1920x1080.
__device__ __forceinline__ float tri_quality_fast(float4 A, float4 B, float4 C, float precision) {
    const float bx = __fsub_rn(B.x, C.x), by = __fsub_rn(B.y, C.y);
    const float ax = __fsub_rn(A.x, C.x), ay = __fsub_rn(A.y, C.y);
    const float dx = __fsub_rn(A.x, B.x), dy = __fsub_rn(A.y, B.y);
    const float sb = __fmaf_rn(bx, bx, __fmul_rn(by, by)), sa = __fmaf_rn(ax, ax, __fmul_rn(ay, ay)),
                sd = __fmaf_rn(dx, dx, __fmul_rn(dy, dy));
    const float ad = fmaxf(sa, sd), m = fmaxf(sb, ad), second = fmaxf(fminf(sa, sd), fminf(sb, ad));
    const bool is_b = sb == m, is_a = sa == m;
    const float2 l = sq_len2(is_b ? bx : is_a ? ax : dx, is_b ? by : is_a ? ay : dy);
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(l.x));
    const float s = __fmul_rn(l.x, y);
    const float rem = __fadd_rn(__fmaf_rn(-s, s, l.x), l.y);
    const float c = __fmul_rn(rem, __fmul_rn(0.5f, y)), err = __fmul_rn(s, 9.094947e-13f);  // 2^-40
    float stretch = __fadd_rn(s, __fadd_rn(c, err));
    if (!(m > 1e-12f) || second >= __fmul_rn(m, 0.999999f) || stretch != __fadd_rn(s, __fsub_rn(c, err)))
        return tri_quality(A.x, A.y, B.x, B.y, C.x, C.y, precision);
    if (precision != 1.f) stretch = __fdiv_rn(stretch, precision);  // stretch /= g_rescale
    return fminf(10000.f, fmaxf(1.f, __fsub_rn(10000.f, __fmul_rn(1000.f, stretch))));
}

// Re-evaluates the winning triangle at pixel (x, y) exactly as the CPU's
// colorize_triangle does for the fragment it keeps (transform.cpp:109-135).
// kWrap: seam triangles may occur; kScaled: Precision may differ from 1.
template <bool kWrap, bool kScaled, class View>
__device__ __forceinline__ Fragment resolve_fragment(const View& V, unsigned long long key, int x, int y,
                                                     float precision = 1.f) {
    Fragment f;
    f.col = make_float3(0.f, 0.f, 0.f);
    f.depth = INFINITY;
    f.validity = 0.f;
    if (key == kEmptyKey) return f;
    const uint32_t tri = (uint32_t)key;
    const uint32_t t = tri & 3u, w = (uint32_t)V.w;
    const uint32_t i = tri >> V.tri_shift, j = (tri >> 2) & ((1u << (V.tri_shift - 2)) - 1u);
    // Vertex indices (below 2^30); the two triangles of quad (i, j):
    // t = 0: (j, i), (j+1, i), (j, i+1); t = 1: (j+1, i+1), (j, i+1), (j+1, i).
    const uint32_t q = i * w + j;
    uint32_t a = q, b = q + 1u, c = q + w;
    if (t == 1u) {
        a = q + w + 1u; b = q + w; c = q + 1u;
    } else if (kWrap && t > 1u) {
        int ax, ay, bx, by, cx, cy;
        tri_vertices(V.w, (int)i, (int)j, (int)t, ax, ay, bx, by, cx, cy);
        a = (uint32_t)ay * w + (uint32_t)ax;
        b = (uint32_t)by * w + (uint32_t)bx;
        c = (uint32_t)cy * w + (uint32_t)cx;
    }
    const float4 A = __ldg(V.vert + a), B = __ldg(V.vert + b), C = __ldg(V.vert + c);
    const float3 ca = packed_color(V, a), cb = packed_color(V, b), cc = packed_color(V, c);
    TriSetup s;
    tri_coef(A, B, C, s);
    float l1, l2, l3;
    barycentric(s, C.x, C.y, x, y, l1, l2, l3);
    f.col.x = interp(ca.x, cb.x, cc.x, l1, l2, l3);
    f.col.y = interp(ca.y, cb.y, cc.y, l1, l2, l3);
    f.col.z = interp(ca.z, cb.z, cc.z, l1, l2, l3);
    f.depth = interp(A.z, B.z, C.z, l1, l2, l3);
    f.validity = tri_quality_fast(A, B, C, kScaled ? precision : 1.f);
    return f;
}

// Running blend of one pixel: colour and, after view 0, the weight sum
// (view 0: its own quality).
struct BlendAcc {
    float c0, c1, c2, q;
};

// Folds view v's fragment (colour, quality = validity / depth, the quality
// of SynthetisedViewTriangle::transform) into the accumulator.  blend_img
// over {accumulator, new view}: weights quality^exp for quality > 0, colour
// * (1 / sum), quality = sum^(1/exp).  After view 0 the accumulator keeps the
// weight sum itself: the reference re-powers its stored sum^(1/exp) by exp,
// which returns the sum up to a few ulp, and quality > 0 exactly when the
// sum is > 0.
// kIntPow: the exponent is an integer from 2 to 16 (and not by_max).
template <bool kIntPow = false>
__device__ __forceinline__ void blend_view(BlendAcc& a, int v, float3 col, float qv, float blend_exp, int exp_int,
                                           bool by_max) {
    if (v == 0) {
        a.c0 = col.x;
        a.c1 = col.y;
        a.c2 = col.z;
        a.q = qv;
        return;
    }
    if (!kIntPow && by_max) {
        // blend_img_by_max (blending.cpp:293-308): the empty colour and
        // quality 0, replaced by the accumulator where its quality is
        // positive, then by the view where its quality is larger still.
        BlendAcc r = {0.f, 1.f, 0.f, 0.f};
        if (a.q > r.q) r = a;
        if (qv > r.q) {
            r.c0 = col.x;
            r.c1 = col.y;
            r.c2 = col.z;
            r.q = qv;
        }
        a = r;
        return;
    }
    float sum = 0.f, c0 = 0.f, c1 = 0.f, c2 = 0.f;
    if (a.q > 0.f) {
        const float w = v != 1 ? a.q : kIntPow ? int_pow(a.q, exp_int) : blend_pow(a.q, blend_exp, exp_int);
        sum = __fadd_rn(sum, w);
        c0 = __fadd_rn(c0, __fmul_rn(w, a.c0));
        c1 = __fadd_rn(c1, __fmul_rn(w, a.c1));
        c2 = __fadd_rn(c2, __fmul_rn(w, a.c2));
    }
    if (qv > 0.f) {
        const float w = kIntPow ? int_pow(qv, exp_int) : blend_pow(qv, blend_exp, exp_int);
        sum = __fadd_rn(sum, w);
        c0 = __fadd_rn(c0, __fmul_rn(w, col.x));
        c1 = __fadd_rn(c1, __fmul_rn(w, col.y));
        c2 = __fadd_rn(c2, __fmul_rn(w, col.z));
    }
    if (sum == 0.f) {
        a.c0 = 0.f; a.c1 = 1.f; a.c2 = 0.f;
        a.q = 0.f;
    } else {
        const float inv = __frcp_rn(sum);
        a.c0 = __fmul_rn(c0, inv);
        a.c1 = __fmul_rn(c1, inv);
        a.c2 = __fmul_rn(c2, inv);
        a.q = sum;
    }
}

template <bool kIntPow>
__device__ __forceinline__ void blend_view(BlendAcc& a, int v, const Fragment& f, float qv, const DevTarget& T) {
    blend_view<kIntPow>(a, v, f.col, qv, T.blend_exp, T.blend_exp_int, T.blend_max != 0);
}

}  // namespace dev
}  // namespace rvsb
