// Mesh stage: warps every input pixel and rasterises the triangles of its
// quads straight away into the views' z-buffers.
//
// A z-buffer holds one 64-bit key per output pixel of a view,
//   (bits of depth^3 / quality) << 32 | triangle scan index,
// and a fragment is one 64-bit atomicMin on it, so the winner does not depend
// on scheduling.  The buffers live in global memory: the views one launch
// works on at a time take tens of megabytes, which the 126 MB L2 holds, and
// a warp's fragments lie in a few rows of neighbouring pixels.  Against
// z-buffers in shared memory per output tile this needs no binning of the
// triangles into tiles (a count, a scan and a fill pass), sets every triangle
// up once instead of once per tile its 8x4-quad block touches (1.35 times on
// the 4 x 1920x1080 view), holds nothing at block barriers, and takes the
// vertices from registers instead of reading the warped mesh back.  Measured
// for the whole call (shared-memory tiles -> this): 4 x 1920x1080 ->
// 1920x1080 598 -> 457 us, -> 960x540 415 -> 267 us, 4 x ERP 4096x2048 -> ERP
// 3062 -> 2010 us, 2 x 960x540 -> 960x540 132 -> 118 us.
//
// mesh_kernel: one warp takes a strip of 32 vertex columns (31 quads) and
// `rows` rows of quads, a lane one column: it warps the row below, gets the
// right neighbour's vertices by shuffles, and rasterises the two triangles of
// its quad.  Triangles of up to `small` candidate pixels are tested by their
// lane; larger ones (stretched over depth discontinuities) go to the slot's
// list and large_kernel rasterises them, one warp per entry, lanes over the
// pixels of their row spans.
#include <algorithm>

#include "device_common.cuh"
#include "kernels.hpp"

namespace rvsb {
namespace {

using namespace dev;

constexpr int MESH_WARPS = 4;
constexpr int STRIP = 31;              // quads (columns) per warp
constexpr int QUEUE = 64;              // large triangles a warp holds before they go to the list
constexpr int LARGE_THREADS = 128;
// Most pixels of a list entry's box: a larger one is entered as
// several bands of rows, so that one triangle over much of the output does
// not keep a single warp busy after all others are done (ERP to ERP, whose
// poles and seam have such triangles: large_kernel 111 us with 4096, 133 with
// 8192, 178 with 16384, 463 with 65536; the whole call is fastest with 8192).
// A thin diagonal triangle gains nothing from it, and smaller bands cost them
// more: 4 x 1920x1080 29 us with 8192, 31 with 4096, 54 with 1024.
constexpr int kEntryPixels = 8192;

// Adding 1.5 * 2^23 rounds a float to the nearest integer and leaves it in
// the low mantissa bits, and for any float the result's bits, compared as
// int, order as the value does; so pixel coordinates stay in this biased form
// through the clamping and the loop (no conversions).
constexpr float kBias = 12582912.f;
constexpr int kBiasBits = 0x4B400000;

// Reciprocal of a normal number, the same result as rcp_approx.
__device__ __forceinline__ float rcp_normal(float x) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// The view's fields the warp uses per vertex (tab.v[view] is indexed by the
// grid, so each use would otherwise be a load).
struct RegView {
    int w, h, proj;
    float p0, p1;
    float R[9], t[3];
    const uint16_t* pd;
    const float4* depth_lut;
    const float* erp_row;
    const float* erp_col;
    __device__ explicit RegView(const DevView& G) {
        w = G.w; h = G.h; proj = G.proj; p0 = G.p0; p1 = G.p1;
#pragma unroll
        for (int k = 0; k < 9; ++k) R[k] = G.R[k];
#pragma unroll
        for (int k = 0; k < 3; ++k) t[k] = G.t[k];
        pd = G.pd; depth_lut = G.depth_lut; erp_row = G.erp_row; erp_col = G.erp_col;
    }
};

// Whether vertex tile (tx, ty) of an ERP input view lies, with
// its one-pixel ring, wholly beyond one of the output's side planes.  A
// vertex is x = z * d (d within the tile's cone, z within its depth range),
// seen by the virtual camera as y = R x + t; beyond plane a when a . y > 0,
// i.e. z * (b . d) + c > 0 with b = R^T a, c = a . t.  Over the cone
// b . d >= b . dc - |b| rho; the smallest value over z is at the near or far
// end of the range.  A relative margin absorbs the float rounding of the
// vertices, and the planes sit one pixel outside the image.
__device__ __forceinline__ bool tile_culled(const DevView& V, const DevTarget& T, int tx, int ty) {
    const int ntx = (V.w + WARP_TILE - 1) / WARP_TILE;
    const size_t k = (size_t)ty * ntx + tx;
    const float4 cone = V.erp_cone[k];
    const float2 zr = V.tile_depth[k];
    if (!(zr.x > 0.f && zr.x <= zr.y)) return false;
#pragma unroll
    for (int p = 0; p < 4; ++p) {
        const float* a = T.cull_plane[p];
        float b[3];
#pragma unroll
        for (int j = 0; j < 3; ++j) b[j] = a[0] * V.R[j] + a[1] * V.R[3 + j] + a[2] * V.R[6 + j];
        const float c = a[0] * V.t[0] + a[1] * V.t[1] + a[2] * V.t[2];
        const float nb = sqrtf(b[0] * b[0] + b[1] * b[1] + b[2] * b[2]);
        const float m = b[0] * cone.x + b[1] * cone.y + b[2] * cone.z - nb * cone.w;
        const float z = m >= 0.f ? zr.x : zr.y;
        const float L = z * m + c;
        if (L > 1e-3f * (fabsf(c) + z * nb) && isfinite(L)) return true;
    }
    return false;
}

// What the rasterisation of one view's triangles needs beside the triangle.
struct MeshTarget {
    unsigned long long* z;
    int wo;
    uint32_t origin;         // biased index (y * wo + x) of pixel (0, 0)
    int xmin, xmax, ymin, ymax;  // pixel range, biased
    float precision;
};

__device__ __forceinline__ float sq2(float dx, float dy) {
    return __fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy));
}

// Key word of a fragment (see key_invq): bits of d^3 / quality.
__device__ __forceinline__ float small_invq(float m, float precision) {
    float stretch = __fsqrt_rn(m);
    if (precision != 1.f) stretch = __fdiv_rn(stretch, precision);
    return rcp_normal(fminf(10000.f, fmaxf(1.f, __fsub_rn(10000.f, __fmul_rn(1000.f, stretch)))));
}

// The triangles of a lane's quad set up for rasterisation: what differs
// between the two (or is derived per triangle).
struct Tri {
    bool active;
    float b1c1, c0b0, c1a1, a0c0;   // edge coefficients as in tri_coef
    float cx, cy, za, zb, zc;
    float mnx, mxx, mny, mxy;       // bounding box
    float m2;                       // longest edge squared
    int4 box;                       // out: candidate pixels, biased
    bool wide, large;               // out: wider than 4e4 pixels; belongs in the list
};

// N triangles of a lane at once: their arithmetic is independent, so it
// overlaps, and one loop runs over the candidates of both (measured with the
// perspective-only instantiation against one triangle after the other: 164 ->
// 148 M warp instructions on 4 x 1920x1080 -> 1920x1080, the stage 233 -> 196
// us, 200 -> 160 us a view in a batch of 8).  The kernel, since then 139 M
// instructions and 164 us, is bound by instruction issue (87% of cycles); the
// atomics took 5 of the 196 us.
//
// Candidate range: a covered pixel's centre lies within the bounding box
// grown by the tolerance tri_range (device_common.cuh) derives, and
// round(mn - delta) .. round(mx + delta) - 1 holds every such pixel and, for
// delta < 0.5, nothing outside the CPU's box [floor(min), ceil(max)].
// Triangles wider than 4e4 pixels (there the CPU's box and the tolerance
// need care) and those with a nearly zero determinant are left to the list.
//
// Coverage: the test of test_pixel (below) with its error bound
// taken at M = 1.  The bound 24u * M on each coordinate is derived there from
// one of 21u * M, so for M < 24/21 the constant 24u still holds; and since
// the three coordinates add up to 1, M >= 24/21 puts the smallest below
// -(M - 1) / 2 < -0.07, far outside.
template <int N>
__device__ __forceinline__ void raster_small(const MeshTarget& o, Tri (&t)[N], uint32_t tri, int small) {
    const float u = 5.9604645e-8f, eps = 1e-6f;
    float den[N];
    int n[N], nmax = 0;
#pragma unroll
    for (int k = 0; k < N; ++k) {
        den[k] = __fsub_rn(__fmul_rn(t[k].b1c1, t[k].a0c0), __fmul_rn(t[k].c0b0, t[k].c1a1));
        const float L = fmaxf(__fsub_rn(t[k].mxx, t[k].mnx), __fsub_rn(t[k].mxy, t[k].mny));
        t[k].wide = !(L < 4.0e4f);
        const float delta = t[k].wide ? 2.f : __fmaf_rn(1e-5f, L, 4e-3f);
        t[k].box.x = max(o.xmin, __float_as_int(__fadd_rn(__fsub_rn(t[k].mnx, delta), kBias)));
        t[k].box.y = max(o.ymin, __float_as_int(__fadd_rn(__fsub_rn(t[k].mny, delta), kBias)));
        t[k].box.z = min(o.xmax, __float_as_int(__fadd_rn(__fadd_rn(t[k].mxx, delta), kBias)) - 1);
        t[k].box.w = min(o.ymax, __float_as_int(__fadd_rn(__fadd_rn(t[k].mxy, delta), kBias)) - 1);
        const bool some = t[k].active && den[k] > 0.f && t[k].box.x <= t[k].box.z && t[k].box.y <= t[k].box.w;
        const int count = (t[k].box.z - t[k].box.x + 1) * (t[k].box.w - t[k].box.y + 1);
        const bool own = !t[k].wide && count <= small && den[k] >= 1e-30f;
        t[k].large = some && !own;
        n[k] = some && own ? count : 0;
        nmax = max(nmax, n[k]);
    }
    if (nmax == 0) return;
    float rinv[N], invq[N], px0[N], px1[N], px[N], py[N];
    uint32_t at[N], wrap[N];
#pragma unroll
    for (int k = 0; k < N; ++k) {
        rinv[k] = rcp_normal(den[k]);
        invq[k] = small_invq(t[k].m2, o.precision);
        px[k] = px0[k] = __fadd_rn(__fsub_rn(__int_as_float(t[k].box.x), kBias), 0.5f);
        px1[k] = __fadd_rn(__fsub_rn(__int_as_float(t[k].box.z), kBias), 0.5f);
        py[k] = __fadd_rn(__fsub_rn(__int_as_float(t[k].box.y), kBias), 0.5f);
        at[k] = (uint32_t)t[k].box.y * (uint32_t)o.wo + (uint32_t)t[k].box.x - o.origin;
        wrap[k] = (uint32_t)(o.wo - (t[k].box.z - t[k].box.x + 1));
    }
    for (int c = 0; c < nmax; ++c) {
        float l1[N], l2[N], l3[N];
        bool in[N], close = false;
#pragma unroll
        for (int k = 0; k < N; ++k) {
            const float tx = __fsub_rn(px[k], t[k].cx), ty = __fsub_rn(py[k], t[k].cy);
            l1[k] = __fmul_rn(__fadd_rn(__fmul_rn(t[k].b1c1, tx), __fmul_rn(t[k].c0b0, ty)), rinv[k]);
            l2[k] = __fmul_rn(__fadd_rn(__fmul_rn(t[k].c1a1, tx), __fmul_rn(t[k].a0c0, ty)), rinv[k]);
            l3[k] = __fsub_rn(__fsub_rn(1.f, l1[k]), l2[k]);
            const float mn = fminf(fminf(l1[k], l2[k]), l3[k]);
            in[k] = mn >= -eps + 24.f * u && c < n[k];
            close |= !(mn >= -eps + 24.f * u) && mn >= -eps - 24.f * u && c < n[k];
        }
        if (close) {
#pragma unroll
            for (int k = 0; k < N; ++k) {
                const float mn = fminf(fminf(l1[k], l2[k]), l3[k]);
                if (!in[k] && c < n[k] && mn >= -eps - 24.f * u) {
                    const float tx = __fsub_rn(px[k], t[k].cx), ty = __fsub_rn(py[k], t[k].cy);
                    l1[k] = __fdiv_rn(__fadd_rn(__fmul_rn(t[k].b1c1, tx), __fmul_rn(t[k].c0b0, ty)), den[k]);
                    l2[k] = __fdiv_rn(__fadd_rn(__fmul_rn(t[k].c1a1, tx), __fmul_rn(t[k].a0c0, ty)), den[k]);
                    l3[k] = __fsub_rn(__fsub_rn(1.f, l1[k]), l2[k]);
                    in[k] = covered(l1[k], l2[k], l3[k]);
                }
            }
        }
#pragma unroll
        for (int k = 0; k < N; ++k) {
            const float d = interp(t[k].za, t[k].zb, t[k].zc, l1[k], l2[k], l3[k]);
            const float key = __fmul_rn(__fmul_rn(__fmul_rn(d, d), d), invq[k]);
            if (in[k] && !isnan(d))
                atomicMin(o.z + at[k], ((unsigned long long)(d > 0.f ? __float_as_uint(key) : 0u) << 32) | (tri + k));
            px[k] += 1.f;
            ++at[k];
            if (px[k] > px1[k]) {
                px[k] = px0[k];
                py[k] += 1.f;
                at[k] += wrap[k];
            }
        }
    }
}

// A warp's large triangles on their way to the slot's list: at most 31 wait
// in the warp's queue in shared memory; full groups of 32 go out together
// (one atomic on the list's length, coalesced 16-byte stores).
//
// A group that passes the list's capacity is dropped: large_kernel sees the
// length and goes over the whole mesh instead.  The warp enters nothing more
// after it, so the length, a 32-bit number, stays within 32 entries per warp
// of the capacity: at most 2^28 input pixels a view, four views a launch and
// 4 quad rows a warp make 8.7 M warps, 2.8e8 entries, beside a capacity of at
// most 3.9e8.  (One triangle over much of a large output has thousands of
// bands, so that counting them all could pass 2^31.)
struct LargeQueue {
    uint4* q;       // QUEUE entries of this warp
    int n;          // of them waiting; negative: the list is full
    __device__ void flush(const SlotBuffers& B, int lane, int count) {
        __syncwarp();
        int base = 0;
        if (lane == 0) base = atomicAdd(&B.status->n_large, count);
        base = __shfl_sync(0xffffffffu, base, 0);
        if (base > B.large_capacity - count) {
            n = INT_MIN;
            return;
        }
        if (lane < count) B.large[base + lane] = q[lane];
        __syncwarp();
        const uint4 rest = q[32 + lane];
        __syncwarp();
        q[lane] = rest;
        n -= count;
        __syncwarp();
    }
    // Entered by the whole warp; `push` lanes have a triangle with box `b`
    // (biased).  Boxes of more than kEntryPixels pixels become bands of rows.
    __device__ void push(const SlotBuffers& B, int lane, bool push, uint32_t tri, int view, bool general, int4 b) {
        const int w = b.z - b.x + 1;
        const int band = general ? 1 << 20 : max(1, kEntryPixels / max(1, w));
        int y = b.y;
        unsigned m;
        while (n >= 0 && (m = __ballot_sync(0xffffffffu, push))) {
            if (push) {
                const int ye = min(b.w, y + band - 1);
                q[n + __popc(m & ((1u << lane) - 1u))] =
                    make_uint4(tri, (uint32_t)view | (general ? 256u : 0u),
                               (uint32_t)(b.x - kBiasBits) | ((uint32_t)(b.z - kBiasBits) << 16),
                               (uint32_t)(y - kBiasBits) | ((uint32_t)(ye - kBiasBits) << 16));
                y = ye + 1;
                push = y <= b.w;
            }
            n += __popc(m);
            if (n >= 32) flush(B, lane, 32);
        }
    }
};

// Grid (ceil(strips / MESH_WARPS), ceil(max quad rows / rows), slots * gv):
// views g0 .. g0 + gv - 1 of every slot.  ERP outputs wrapping horizontally
// have one more strip, whose lanes take the seam triangles of one row each.
template <int kIn, bool kErpOut, bool kScaled, class Tabs>
__global__ void __launch_bounds__(32 * MESH_WARPS, 8) mesh_kernel(const __grid_constant__ Tabs tabs, int g0, int gv,
                                                                   int rows) {
    __shared__ uint4 s_queue[MESH_WARPS][QUEUE];
    grid_dep_wait();
    const SlotTable& tab = tabs.at(blockIdx.z / gv);
    const int view = g0 + blockIdx.z % gv;
    const DevTarget& T = tab.t;
    if (view >= T.n_views) return;
    const DevView& G = tab.v[view];
    const RegView V(G);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int strip = blockIdx.x * MESH_WARPS + warp, i0 = blockIdx.y * rows;
    const int nstrips = (G.w - 1 + STRIP - 1) / STRIP;
    const bool seam = kErpOut && T.wrap != 0 && strip == nstrips;
    if (i0 >= G.h - 1 || (strip >= nstrips && !seam)) return;
    const int i1 = min(i0 + rows, G.h - 1);  // last vertex row of the warp's quads
    const int j = strip * STRIP + lane;
    bool keep_all = false;
    if (kIn != kPerspectiveIn && T.cull && G.erp_cone) {
        // Quad rows i0 .. i1 - 1 lie in one row of vertex tiles (rows divides
        // WARP_TILE) and the strip's quads in at most two tiles of it; every
        // quad's corners lie in its tile grown by one pixel.
        const int t0 = strip * STRIP / WARP_TILE, t1 = min(strip * STRIP + STRIP - 1, G.w - 2) / WARP_TILE;
        const bool live = t0 + lane <= t1 && !tile_culled(G, T, t0 + lane, i0 / WARP_TILE);
        if (!__any_sync(0xffffffffu, live)) return;
        // The strips right of and below this one may be skipped: the last
        // column and row are stored here as well.
        keep_all = true;
    }
    MeshTarget o;
    o.wo = T.wo;
    o.xmin = o.ymin = kBiasBits;
    o.xmax = kBiasBits + T.wo - 1;
    o.ymax = kBiasBits + T.ho - 1;
    o.z = G.z;
    o.origin = (uint32_t)kBiasBits * (uint32_t)T.wo + (uint32_t)kBiasBits;
    o.precision = kScaled ? T.precision : 1.f;
    float4* vert = G.vert;
    const int shift = G.tri_shift;
    LargeQueue queue{s_queue[warp], 0};
    if (!seam) {
        const bool in_col = j < V.w;
        const bool store = in_col && (lane < STRIP || j == V.w - 1 || keep_all);
        const int jc = min(j, V.w - 1);
        const bool last = i1 == V.h - 1 || keep_all;  // row i1 is stored here
        const InputColumn col = input_column<kIn>(V, jc);
        float4 L = depth_entry(V, i0, jc);
        uint16_t raw = __ldg(V.pd + (size_t)min(i0 + 2, i1) * V.w + jc);
        float4 Ln = depth_entry(V, i0 + 1, jc);
        float4 a = warp_vertex<kIn, kErpOut, kScaled>(V, T, i0, col, L);
        if (store) vert[(size_t)i0 * V.w + j] = a;
        // Emission test (transform.cpp:161-167) per vertex, as masks of the row.
        unsigned ok_a = __ballot_sync(0xffffffffu, a.z > 0.f && a.x > 0.f);
        const unsigned quads = __ballot_sync(0xffffffffu, lane < STRIP && j + 1 < V.w);
        float bx = __shfl_down_sync(0xffffffffu, a.x, 1), by = __shfl_down_sync(0xffffffffu, a.y, 1),
              bz = __shfl_down_sync(0xffffffffu, a.z, 1);
        for (int i = i0; i < i1; ++i) {
            L = Ln;
            Ln = __ldg(V.depth_lut + raw);
            raw = __ldg(V.pd + (size_t)min(i + 3, i1) * V.w + jc);
            const float4 c = warp_vertex<kIn, kErpOut, kScaled>(V, T, i + 1, col, L);
            if (store && (i + 1 < i1 || last)) vert[(size_t)(i + 1) * V.w + j] = c;
            const unsigned ok_c = __ballot_sync(0xffffffffu, c.z > 0.f && c.x > 0.f);
            const float dx = __shfl_down_sync(0xffffffffu, c.x, 1), dy = __shfl_down_sync(0xffffffffu, c.y, 1),
                        dz = __shfl_down_sync(0xffffffffu, c.z, 1);
            const unsigned cond = (ok_a >> 1) & ok_c & quads;
            if (cond) {
                const uint32_t tri = (((uint32_t)i << (shift - 2)) | (uint32_t)j) * 4u;
                // The diagonal b - c belongs to both triangles: its
                // differences, squared length and box serve both (negated
                // exactly for the second).
                const float ey = __fsub_rn(by, c.y), ex = __fsub_rn(c.x, bx);
                const float md = sq2(ex, ey);
                const float nx = fminf(bx, c.x), xx = fmaxf(bx, c.x), ny = fminf(by, c.y), xy = fmaxf(by, c.y);
                Tri t[2];
                t[0].active = (cond & ok_a) >> lane & 1u;
                t[0].b1c1 = ey; t[0].c0b0 = ex;
                t[0].a0c0 = __fsub_rn(a.x, c.x); t[0].c1a1 = __fsub_rn(c.y, a.y);
                t[0].cx = c.x; t[0].cy = c.y;
                t[0].za = a.z; t[0].zb = bz; t[0].zc = c.z;
                t[0].mnx = fminf(nx, a.x); t[0].mxx = fmaxf(xx, a.x);
                t[0].mny = fminf(ny, a.y); t[0].mxy = fmaxf(xy, a.y);
                t[0].m2 = fmaxf(md, fmaxf(sq2(t[0].a0c0, t[0].c1a1), sq2(__fsub_rn(a.x, bx), __fsub_rn(a.y, by))));
                t[1].active = (cond & (ok_c >> 1)) >> lane & 1u;
                t[1].b1c1 = -ey; t[1].c0b0 = -ex;
                t[1].a0c0 = __fsub_rn(dx, bx); t[1].c1a1 = __fsub_rn(by, dy);
                t[1].cx = bx; t[1].cy = by;
                t[1].za = dz; t[1].zb = c.z; t[1].zc = bz;
                t[1].mnx = fminf(nx, dx); t[1].mxx = fmaxf(xx, dx);
                t[1].mny = fminf(ny, dy); t[1].mxy = fmaxf(xy, dy);
                t[1].m2 = fmaxf(md, fmaxf(sq2(t[1].a0c0, t[1].c1a1), sq2(__fsub_rn(dx, c.x), __fsub_rn(dy, c.y))));
                raster_small(o, t, tri, T.small);
                if (__any_sync(0xffffffffu, t[0].large || t[1].large)) {
                    queue.push(tab.b, lane, t[0].large, tri, view, t[0].wide, t[0].box);
                    queue.push(tab.b, lane, t[1].large, tri + 1u, view, t[1].wide, t[1].box);
                }
            }
            a = c;
            bx = dx;
            by = dy;
            bz = dz;
            ok_a = ok_c;
        }
    } else if constexpr (kErpOut) {
        // Seam triangles (transform.cpp:168-175), between columns W - 1 and 0
        // of quad row i0 + lane: emitted where quad (i, 0)'s diagonal is.
        const int i = min(i0 + lane, i1 - 1);
        float4 v[5];  // (i, 0), (i, 1), (i + 1, 0), (i, W - 1), (i + 1, W - 1)
#pragma unroll 1
        for (int k = 0; k < 5; ++k) {
            const int r = i + (k == 2 || k == 4), q = k == 1 ? 1 : k >= 3 ? V.w - 1 : 0;
            v[k] = warp_vertex<kIn, kErpOut, kScaled>(V, T, r, input_column<kIn>(V, q), depth_entry(V, r, q));
        }
        const float4 v00 = v[0], v01 = v[1], v10 = v[2], w0 = v[3], w1 = v[4];
        const bool active = i0 + lane < i1 && v01.z > 0.f && v10.z > 0.f && v01.x > 0.f && v10.x > 0.f;
        const uint32_t tri = ((uint32_t)i << shift) | 2u;
#pragma unroll 1
        for (int t = 0; t < 2; ++t) {
            const float4 A = t ? v10 : w0, B = t ? w1 : v00, C = t ? v00 : w1;
            Tri s[1];
            s[0].active = active;
            s[0].b1c1 = __fsub_rn(B.y, C.y); s[0].c0b0 = __fsub_rn(C.x, B.x);
            s[0].a0c0 = __fsub_rn(A.x, C.x); s[0].c1a1 = __fsub_rn(C.y, A.y);
            s[0].cx = C.x; s[0].cy = C.y;
            s[0].za = A.z; s[0].zb = B.z; s[0].zc = C.z;
            s[0].mnx = fminf(fminf(A.x, B.x), C.x); s[0].mxx = fmaxf(fmaxf(A.x, B.x), C.x);
            s[0].mny = fminf(fminf(A.y, B.y), C.y); s[0].mxy = fmaxf(fmaxf(A.y, B.y), C.y);
            s[0].m2 = fmaxf(sq2(s[0].c0b0, s[0].b1c1), fmaxf(sq2(s[0].a0c0, s[0].c1a1),
                                                             sq2(__fsub_rn(A.x, B.x), __fsub_rn(A.y, B.y))));
            raster_small(o, s, tri + (uint32_t)t, T.small);
            queue.push(tab.b, lane, s[0].large, tri + (uint32_t)t, view, s[0].wide, s[0].box);
        }
    }
    if (queue.n > 0) queue.flush(tab.b, lane, queue.n);
}

// ---------------------------------------------------------------------------
// Large triangles
// ---------------------------------------------------------------------------

// Candidate pixel (x, y) of a set-up triangle: the coverage test of
// transform.cpp:105-114; on success its depth, for the fragment key.
// The CPU keeps, per output pixel, the fragment with the largest
// quality / depth^3 (a later fragment replaces the stored one iff
// (d/D)^3 * Q < q, transform.cpp:119-142), the earliest in scan order on
// ties.  The key holds the bits of depth^3 / quality (smaller is better)
// above the triangle's scan index, so 64-bit atomicMin keeps that winner
// whatever the scheduling order.
//
// The coordinates come from rinv, an approximate reciprocal of den (at most
// 1 ulp off).  Then l1 and l2 are within 4u|l| of the CPU's n / den
// (u = 2^-24: 2u from the reciprocal, one rounding here and one in the
// CPU's division), and l3 = (1 - l1) - l2 within
// u * (4|l1| + 2|1 - l1| + 4|l2| + 2|l3|) of the CPU's, which is below
// 21u * M with M = max(|l1|, |l2|, |l3|, 1).  One bound, 24u * M, therefore
// covers every coordinate: the test is decided when the smallest coordinate
// is farther than the bound from -1e-6; otherwise the coordinates are
// recomputed with the reference's divisions.  The depth in the key uses the
// fast coordinates; the resolve recomputes the winning fragment exactly.
__device__ __forceinline__ bool test_pixel(const TriSetup& s, float cx, float cy, float za, float zb_, float zc,
                                           int x, int y, float& d) {
    const float u = 5.9604645e-8f, eps = 1e-6f;
    const float tx = __fsub_rn(__fadd_rn((float)x, 0.5f), cx);
    const float ty = __fsub_rn(__fadd_rn((float)y, 0.5f), cy);
    const float n1 = __fadd_rn(__fmul_rn(s.b1c1, tx), __fmul_rn(s.c0b0, ty));
    const float n2 = __fadd_rn(__fmul_rn(s.c1a1, tx), __fmul_rn(s.a0c0, ty));
    float l1 = __fmul_rn(n1, s.rinv), l2 = __fmul_rn(n2, s.rinv);
    float l3 = __fsub_rn(__fsub_rn(1.f, l1), l2);
    const float mn = fminf(fminf(l1, l2), l3);
    const float M = fmaxf(fmaxf(fabsf(l1), fabsf(l2)), fmaxf(fabsf(l3), 1.f));
    const float bound = __fmul_rn(24.f * u, M);
    if (__fadd_rn(mn, bound) < -eps) return false;
    if (!(__fsub_rn(mn, bound) >= -eps)) {
        l1 = __fdiv_rn(n1, s.den);
        l2 = __fdiv_rn(n2, s.den);
        l3 = __fsub_rn(__fsub_rn(1.f, l1), l2);
        if (!covered(l1, l2, l3)) return false;
    }
    d = interp(za, zb_, zc, l1, l2, l3);
    return !isnan(d);
}

// Quality of the key only (the resolve recomputes it exactly): the longest
// edge in float, a few ulp from the reference's double evaluation.  The
// squared lengths of an edge shared by two triangles are identical, so
// equal reference qualities stay equal here.
__device__ __forceinline__ float key_invq(float4 A, float4 B, float4 C, float precision) {
    return small_invq(fmaxf(sq2(__fsub_rn(B.x, C.x), __fsub_rn(B.y, C.y)),
                            fmaxf(sq2(__fsub_rn(A.x, B.x), __fsub_rn(A.y, B.y)),
                                  sq2(__fsub_rn(A.x, C.x), __fsub_rn(A.y, C.y)))),
                      precision);
}

__device__ __forceinline__ unsigned long long frag_key(float d, float invq, uint32_t tri) {
    uint32_t hi = 0u;
    if (d > 0.f) hi = __float_as_uint(__fmul_rn(__fmul_rn(__fmul_rn(d, d), d), invq));
    return ((unsigned long long)hi << 32) | tri;
}

// A triangle set up for the warp: its coefficients and candidate box, and what
// a fragment's key needs.
struct Large {
    TriSetup s;
    float cx, cy, za, zb, zc, invq;
    uint32_t tri;
    unsigned long long* z;
};

__device__ __forceinline__ void plot(const Large& t, int wo, int x, int y) {
    float d;
    if (test_pixel(t.s, t.cx, t.cy, t.za, t.zb, t.zc, x, y, d))
        atomicMin(t.z + (size_t)y * wo + x, frag_key(d, t.invq, t.tri));
}

__device__ __forceinline__ int incl_sum(int v, int lane) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int u = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += u;
    }
    return v;
}

// Owner of item `c` of a flattened sequence: the number of lanes whose
// inclusive prefix is at most c (binary search).
__device__ __forceinline__ int owner_of(int incl, int c) {
    int own = 0;
#pragma unroll
    for (int step = 16; step > 0; step >>= 1) {
        const int probe = __shfl_sync(0xffffffffu, incl, own + step - 1);
        if (probe <= c) own += step;
    }
    return own;
}

// The triangle set up by lane `k`.
__device__ __forceinline__ Large from_lane(const Large& t, int k) {
    Large r;
    r.s.b1c1 = __shfl_sync(0xffffffffu, t.s.b1c1, k);
    r.s.c0b0 = __shfl_sync(0xffffffffu, t.s.c0b0, k);
    r.s.c1a1 = __shfl_sync(0xffffffffu, t.s.c1a1, k);
    r.s.a0c0 = __shfl_sync(0xffffffffu, t.s.a0c0, k);
    r.s.den = __shfl_sync(0xffffffffu, t.s.den, k);
    r.s.rinv = __shfl_sync(0xffffffffu, t.s.rinv, k);
    r.s.x0 = __shfl_sync(0xffffffffu, t.s.x0, k);
    r.s.x1 = __shfl_sync(0xffffffffu, t.s.x1, k);
    r.s.y0 = __shfl_sync(0xffffffffu, t.s.y0, k);
    r.s.y1 = __shfl_sync(0xffffffffu, t.s.y1, k);
    r.cx = __shfl_sync(0xffffffffu, t.cx, k);
    r.cy = __shfl_sync(0xffffffffu, t.cy, k);
    r.za = __shfl_sync(0xffffffffu, t.za, k);
    r.zb = __shfl_sync(0xffffffffu, t.zb, k);
    r.zc = __shfl_sync(0xffffffffu, t.zc, k);
    r.invq = __shfl_sync(0xffffffffu, t.invq, k);
    r.tri = __shfl_sync(0xffffffffu, t.tri, k);
    r.z = reinterpret_cast<unsigned long long*>(
        __shfl_sync(0xffffffffu, reinterpret_cast<unsigned long long>(t.z), k));
    return r;
}

// One warp rasterises a triangle: the candidate span of each row, one lane
// per row and 32 rows at a time, then the spans' pixels flattened over the
// warp, 32 candidates per round whatever the shape.
__device__ __forceinline__ void raster_large(const Large& t, int wo, int lane) {
    for (int yb = t.s.y0; yb <= t.s.y1; yb += 32) {
        const int y = yb + lane;
        int xl = 0, xr = -1;
        if (y <= t.s.y1) row_span(t.s, t.cx, t.cy, y, xl, xr);
        const int len = max(0, xr - xl + 1);
        const int incl = incl_sum(len, lane);
        const int excl = incl - len;
        const int total = __shfl_sync(0xffffffffu, incl, 31);
        for (int base = 0; base < total; base += 32) {
            const int c = base + lane;
            const int row = owner_of(incl, c);
            const int rxl = __shfl_sync(0xffffffffu, xl, row);
            const int rex = __shfl_sync(0xffffffffu, excl, row);
            if (c < total) plot(t, wo, rxl + (c - rex), yb + row);
        }
    }
}

// The warp's triangles (one per lane that is `on`) with their boxes flattened
// together, 32 candidates per round.
constexpr int kMediumPixels = 64;
__device__ __forceinline__ void raster_medium(const Large& t, bool on, int wo, int lane) {
    const int bw = t.s.x1 - t.s.x0 + 1;
    const int count = on ? bw * (t.s.y1 - t.s.y0 + 1) : 0;
    const int incl = incl_sum(count, lane);
    const int total = __shfl_sync(0xffffffffu, incl, 31);
    for (int base = 0; base < total; base += 32) {
        const int c = base + lane;
        const int own = owner_of(incl, c) & 31;
        const Large r = from_lane(t, own);
        const int k = c - __shfl_sync(0xffffffffu, incl - count, own), w = __shfl_sync(0xffffffffu, bw, own);
        if (c >= total) continue;
        // k and w are at most 64: (k + 0.5) / w is at least 1/128 from an
        // integer, so the fast quotient truncates to the exact row.
        const int dy = (int)__fdividef((float)k + 0.5f, (float)w);
        plot(r, wo, r.s.x0 + (k - dy * w), r.s.y0 + dy);
    }
}

// Vertices of triangle `tri` of view V from the stored mesh.
__device__ __forceinline__ void load_triangle(const DevView& V, uint32_t tri, float4& A, float4& B, float4& C) {
    const int i = (int)(tri >> V.tri_shift), j = (int)((tri >> 2) & ((1u << (V.tri_shift - 2)) - 1u));
    int ax, ay, bx, by, cx, cy;
    tri_vertices(V.w, i, j, (int)(tri & 3u), ax, ay, bx, by, cx, cy);
    A = __ldg(V.vert + (size_t)ay * V.w + ax);
    B = __ldg(V.vert + (size_t)by * V.w + bx);
    C = __ldg(V.vert + (size_t)cy * V.w + cx);
}

// Triangle `tri` of view V set up for rasterisation.  False when nothing of it
// can be covered.  Its candidate box is (x0, y0) .. (x1, y1) where `box` says
// so, else computed (the whole triangle).
__device__ __forceinline__ bool set_up(const DevView& V, const DevTarget& T, uint32_t tri, bool box, Large& t) {
    float4 A, B, C;
    load_triangle(V, tri, A, B, C);
    const int x0 = t.s.x0, x1 = t.s.x1, y0 = t.s.y0, y1 = t.s.y1;
    if (!tri_coef(A, B, C, t.s)) return false;
    if (box) {
        t.s.x0 = x0; t.s.x1 = x1; t.s.y0 = y0; t.s.y1 = y1;
    } else if (!tri_range(A, B, C, T.wo, T.ho, 0, T.wo - 1, 0, T.ho - 1, t.s)) {
        return false;
    }
    t.s.rinv = rcp_approx(t.s.den);
    t.cx = C.x; t.cy = C.y;
    t.za = A.z; t.zb = B.z; t.zc = C.z;
    t.invq = key_invq(A, B, C, T.precision);
    t.tri = tri;
    t.z = V.z;
    return true;
}

// Whether a list entry is of at most kMediumPixels candidates (its box known).
__device__ __forceinline__ bool is_medium(uint4 q) {
    return !(q.y & 256u) &&
           ((q.z >> 16) - (q.z & 0xffffu) + 1u) * ((q.w >> 16) - (q.w & 0xffffu) + 1u) <= (uint32_t)kMediumPixels;
}

__device__ __forceinline__ bool set_up_entry(const SlotTable& tab, uint4 q, Large& t) {
    t.s.x0 = (int)(q.z & 0xffffu);
    t.s.x1 = (int)(q.z >> 16);
    t.s.y0 = (int)(q.w & 0xffffu);
    t.s.y1 = (int)(q.w >> 16);
    return set_up(tab.v[q.y & 255u], tab.t, q.x, !(q.y & 256u), t);
}

// A triangle of the whole-mesh pass, or one the list holds whole, that covers more
// pixels (about) is huge: its rows go to the warps in kHugeParts parts.  ERP 1024x512 with depth steps into ERP
// 4096x2048: 2560 us with 65536 and 128 parts, 2070 so, 1972 with 4096 and 16, but
// noise 480x270 into 3840x2160 1850, 1840 and 2189.
constexpr int kHugePixels = 16384;
constexpr int kHugeParts = 32;

// A huge triangle's word: its index, its view, kHugeThere once it is there, and
// the parts handed out.  One word, so that nothing has to be ordered by a fence: with
// fences in it, even where they were never reached, the kernel took half as long
// again over its list (4 x ERP 4096x2048 into ERP 125 -> 194 us).
constexpr unsigned long long kHugeThere = 1ull << 40, kHugePart = 1ull << 48;
__device__ __forceinline__ unsigned long long* huge_words(const SlotBuffers& B) {
    return reinterpret_cast<unsigned long long*>(B.large + B.large_capacity);
}

// The warp's huge triangles (the lanes `on`) into their words, for all warps to
// take parts of; returns the lanes whose triangle found none.
__device__ __forceinline__ unsigned offer_huge(const SlotBuffers& B, uint32_t tri, int view, unsigned on, int lane) {
    int base = B.huge_capacity;
    // Words that are all taken are left alone, so that the count stays bounded.
    if (lane == 0 && *reinterpret_cast<volatile int*>(&B.status->n_huge) < B.huge_capacity)
        base = atomicAdd(&B.status->n_huge, __popc(on));
    const int slot = __shfl_sync(0xffffffffu, base, 0) + __popc(on & ((1u << lane) - 1u));
    const bool in = (on >> lane & 1u) && slot < B.huge_capacity;
    if (in) atomicExch(huge_words(B) + slot, kHugeThere | (unsigned long long)view << 32 | tri);
    return on & ~__ballot_sync(0xffffffffu, in);
}

// Parts of the huge triangles that are there, until all are handed out, one of each
// of 32 words at a time.  The warp that offered one comes here after it, so none is
// left over.
__device__ __forceinline__ void take_huge(const SlotTable& tab, int n, int wid, int lane) {
    const unsigned blocks = (unsigned)(n + 31) / 32u;
    for (unsigned k = 0; k < blocks; ++k) {
        // Not all warps at the same words.
        unsigned long long* words = huge_words(tab.b) + ((unsigned)wid * 37u + k) % blocks * 32u;
        const int there = min(32, (int)(huge_words(tab.b) + n - words));
        for (;;) {
            const unsigned long long h =
                lane < there ? *reinterpret_cast<volatile unsigned long long*>(words + lane) : 0ull;
            unsigned m = __ballot_sync(0xffffffffu, (h & kHugeThere) && h / kHugePart < kHugeParts);
            if (!m) break;
            for (; m; m &= m - 1) {
                unsigned long long w = 0;
                if (lane == 0) w = atomicAdd(words + (__ffs(m) - 1), kHugePart);
                w = __shfl_sync(0xffffffffu, w, 0);
                const int part = (int)(w / kHugePart);
                Large t;
                if (part >= kHugeParts || !set_up(tab.v[(int)(w >> 32) & 255], tab.t, (uint32_t)w, false, t)) continue;
                const int rows = (t.s.y1 - t.s.y0 + kHugeParts) / kHugeParts;
                t.s.y0 += part * rows;
                t.s.y1 = min(t.s.y1, t.s.y0 + rows - 1);
                raster_large(t, tab.t.wo, lane);
            }
        }
    }
}

__device__ __forceinline__ int huge_count(const SlotBuffers& B) {
    return min(*reinterpret_cast<volatile int*>(&B.status->n_huge), B.huge_capacity);
}

__device__ __forceinline__ bool is_huge(const Large& t) {
    // den is twice the triangle's area.
    return (t.s.x1 - t.s.x0 + 1) * (t.s.y1 - t.s.y0 + 1) > kHugePixels && t.s.den > 2.f * (float)kHugePixels;
}

// Every triangle of the views g0 .. g0 + gv - 1: the warps claim groups of quads.
// Triangles differ much in work, the stretched ones lie together (a row of quads
// across a depth step, the poles of an equirectangular output), and one can cover
// most of the output.  Rows of 32 quads dealt out in turn, and each triangle left
// to the warp that met it, kept the chip waiting for a few warps (18% of the SMs'
// cycles in use).  So a group is 4 x 4 quads, claimed when a warp is free, the
// outer rows before the inner, and the huge triangles are shared out: 3 x 1186x198
// with bars of 6 rows magnified 3.9 times 3968 -> 591 us, 3 x ERP 1024x512 into ERP
// 4096x2048 with depth steps 4207 -> 1614, with noise 70468 -> 38292, smooth 1213
// -> 1189; 4 x 1920x1080 with bars 2276 -> 1875, with noise 7062 -> 6345.  Groups
// of 8 x 4: 595, 2030, 54869, 1076, 1614 and 6191; of 2 x 4: 615, 1666, 33082,
// 1483, 2400 and 6738.  2 x 480x270 noise into 120x68, whose triangles are all
// small, pays for it: 119 -> 134.
__device__ __forceinline__ void whole_mesh(const SlotTable& tab, int g0, int gv, int wid, int nw, int lane) {
    const DevTarget& T = tab.t;
    const bool wrap = T.wrap != 0;
    auto claim = [&] { return lane == 0 ? atomicAdd(&tab.b.status->n_claimed, 1) : 0; };
    int next = __shfl_sync(0xffffffffu, claim(), 0), first = 0;
    for (int view = g0; view < min(T.n_views, g0 + gv); ++view) {
        const DevView& V = tab.v[view];
        // Fewer rows a group where that leaves some warps without any.
        int rows = 4;
        while (rows > 1 && (long long)(V.w - 1) * (V.h - 1) < 4ll * rows * nw) rows /= 2;
        const int groups = (V.w + 2) / 4, bands = (V.h - 2 + rows) / rows, count = groups * bands;
        while (next < first + count) {
            const int g = next - first, claimed = claim();
            next = __shfl_sync(0xffffffffu, claimed, 0);
            const int r = g / groups, i0 = (r & 1 ? bands - 1 - r / 2 : r / 2) * rows, j0 = g % groups * 4;
            if (T.cull && V.erp_cone && tile_culled(V, T, j0 / WARP_TILE, i0 / WARP_TILE)) continue;
            const int i = i0 + lane / 4, j = j0 + lane % 4;
            for (int t = 0; t < (wrap ? 4 : 2); ++t) {
                const uint32_t tri = ((((uint32_t)i << (V.tri_shift - 2)) | (uint32_t)j) << 2) | (uint32_t)t;
                Large q = {};
                bool on = lane < 4 * rows && i < V.h - 1 && j < V.w - 1 && (t < 2 || j == 0);
                if (on) {
                    // Emission tests of transform.cpp:161-167.
                    const float4 v01 = __ldg(V.vert + (size_t)i * V.w + j + 1);
                    const float4 v10 = __ldg(V.vert + (size_t)(i + 1) * V.w + j);
                    const float4 a = __ldg(V.vert + (size_t)(i + (t & 1)) * V.w + j + (t & 1));
                    on = v01.z > 0.f && v10.z > 0.f && v01.x > 0.f && v10.x > 0.f &&
                         (t >= 2 || (a.z > 0.f && a.x > 0.f)) && set_up(V, T, tri, false, q);
                }
                const int box = (q.s.x1 - q.s.x0 + 1) * (q.s.y1 - q.s.y0 + 1);
                const bool medium = on && box <= kMediumPixels;
                raster_medium(q, medium, T.wo, lane);
                unsigned m = __ballot_sync(0xffffffffu, on && !medium);
                const unsigned huge = __ballot_sync(0xffffffffu, on && is_huge(q));
                if (huge) m = (m & ~huge) | offer_huge(tab.b, tri, view, huge, lane);
                for (; m; m &= m - 1) raster_large(from_lane(q, __ffs(m) - 1), T.wo, lane);
            }
        }
        first += count;
    }
}

// What the list does not hold.  Not inlined: its registers would spill in the
// list's loops.
__device__ __noinline__ void large_rest(const SlotTable& tab, int g0, int gv, bool overflow, int wid, int nw, int lane) {
    if (overflow) whole_mesh(tab, g0, gv, wid, nw, lane);
    take_huge(tab, huge_count(tab.b), wid, lane);
}

// Grid (CTAs, slots), LARGE_THREADS threads, over the slot's list.  Medium
// entries: a warp takes up to 32 consecutive ones (fewer when the list is
// short, so that all warps have some), sets them up one per lane and
// rasterises them together; 2 x 960x540 magnified twice with a threshold of 4
// candidates lists nearly every triangle, 111 us against 995 us with a warp per
// entry.  The others go one by one to the warps, dealt out in turn: they are
// few and differ in size, and neighbours in the list are alike (a warp that
// took 32 in a row kept the kernel waiting: 590 instead of 178 us, ERP to ERP).
//
// When the list overflowed (more large triangles than it holds), the warps
// instead go over all quads of the group's views (whole_mesh) and rasterise every
// triangle; those the mesh kernel has done already only repeat keys that are
// there (atomicMin).
template <class Tabs>
__global__ void __launch_bounds__(LARGE_THREADS, 8) large_kernel(const __grid_constant__ Tabs tabs, int g0, int gv) {
    grid_dep_wait();
    const SlotTable& tab = tabs.at(blockIdx.y);
    const DevTarget& T = tab.t;
    if (g0 >= T.n_views) return;
    const int n = tab.b.status->n_large;
    const int lane = threadIdx.x & 31;
    const int wid = blockIdx.x * (LARGE_THREADS / 32) + (threadIdx.x >> 5), nw = gridDim.x * (LARGE_THREADS / 32);
    if (n <= tab.b.large_capacity) {
        const uint4* list = tab.b.large;
        bool offered = false;
        for (int base = 0; base < n; base += 32 * nw) {
            // Lane k looks at the warp's k-th entry of the round.
            const int e = base + lane * nw + wid;
            uint4 q = make_uint4(0u, 0u, 0u, 0u);
            if (e < n) q = __ldg(list + e);
            for (unsigned m = __ballot_sync(0xffffffffu, e < n && !is_medium(q)); m; m &= m - 1) {
                const int k = __ffs(m) - 1;
                Large t;
                if (set_up_entry(tab,
                                 make_uint4(__shfl_sync(0xffffffffu, q.x, k), __shfl_sync(0xffffffffu, q.y, k),
                                            __shfl_sync(0xffffffffu, q.z, k), __shfl_sync(0xffffffffu, q.w, k)),
                                 t)) {
                    // A triangle wider than 4e4 pixels was entered whole: 6 x ERP
                    // 796x226 magnified 38 times with bars at arm's length 2278 us
                    // with such triangles left to one warp each, 341 shared out.
                    const uint32_t general = __shfl_sync(0xffffffffu, q.y, k);
                    if ((general & 256u) && is_huge(t)) {
                        offered = true;
                        if (!offer_huge(tab.b, t.tri, (int)(general & 255u), 1u, lane)) continue;
                    }
                    raster_large(t, T.wo, lane);
                }
            }
        }
        // One warp in four looks for others' huge triangles (a word that all read
        // takes their reads in turn), under the loop that follows.
        const int huge = threadIdx.x < 32 ? huge_count(tab.b) : 0;
        const int per = min(32, (n + nw - 1) / nw);
        for (int e0 = wid * per; e0 < n; e0 += nw * per) {
            Large t = {};
            bool on = lane < per && e0 + lane < n;
            if (on) {
                const uint4 q = __ldg(list + e0 + lane);
                on = is_medium(q) && set_up_entry(tab, q, t);
            }
            raster_medium(t, on, T.wo, lane);
        }
        if (huge == 0 && !offered) return;
    }
    large_rest(tab, g0, gv, n > tab.b.large_capacity, wid, nw, lane);
}

// Empty keys in the z-buffers of views g0 .. g0 + gv - 1 of every slot, an
// empty list of large triangles and the counters of the pass over the whole mesh.  Grid (CTAs, slots).
template <class Tabs>
__global__ void __launch_bounds__(256) clear_kernel(const __grid_constant__ Tabs tabs, int g0, int gv) {
    grid_dep_wait();
    const SlotTable& tab = tabs.at(blockIdx.y);
    const DevTarget& T = tab.t;
    if (g0 >= T.n_views) return;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        tab.b.status->n_large = 0;
        tab.b.status->n_claimed = 0;
        tab.b.status->n_huge = 0;
    }
    const unsigned some = min(gridDim.x, 32u);
    if (blockIdx.x < some)
        for (int k = blockIdx.x * 256 + threadIdx.x; k < tab.b.huge_capacity; k += some * 256) huge_words(tab.b)[k] = 0ull;
    const size_t n = (size_t)min(gv, T.n_views - g0) * T.wo * T.ho;
    unsigned long long* z = tab.v[g0].z;  // the group's buffers lie back to back from a 16-byte boundary
    if (blockIdx.x == 0 && threadIdx.x == 0 && (n & 1)) z[n - 1] = kEmptyKey;
    for (size_t k = (size_t)blockIdx.x * 256 + threadIdx.x; k < n / 2; k += (size_t)gridDim.x * 256)
        reinterpret_cast<ulonglong2*>(z)[k] = make_ulonglong2(kEmptyKey, kEmptyKey);
}

}  // namespace

// Quad rows per warp, by how many waves of warps (148 SMs x 32) 8 rows each
// would make.  More rows warp fewer vertices twice (one row of 1 + 1 / rows),
// fewer leave shorter warps at the end of the launch (times of the general kernel,
// before launch_mesh_kernels' instantiations).  Below 2 waves 4 rows: 2
// x 960x540 43 us the stage, 49 with 8, 61 with 16.  Below 40 waves 8: 4 x
// 1920x1080 193 us (16 rows: 196), 4 x ERP 4096x2048 into ERP 1076 (16: 1121,
// 32: 1156).  Above, where the end does not matter, 32: 8 poses of the 1080p
// scene 160 us a view (8: 166), 8 views of the ERP scene 122 (16: 128, 8: 145;
// a warp also decides there whether its rows are culled at all).
static int rows_per_warp(const BatchShape& sh, int gv) {
    const long long warps = (long long)sh.slots * gv * ((sh.max_w - 1 + STRIP - 1) / STRIP) * ((sh.max_h + 6) / 8);
    const long long wave = 148 * 32;
    return warps < 2 * wave ? 4 : warps < 40 * wave ? 8 : 32;
}

template <int kIn, bool kErpOut, bool kScaled, class Tabs>
static void launch_mesh_kernel(const Tabs& tabs, const BatchShape& sh, int g0, int gv, cudaStream_t s) {
    const int fixed = kRasterVariants[sh.variant].rows, rows = fixed ? fixed : rows_per_warp(sh, gv);
    const int strips = (sh.max_w - 1 + STRIP - 1) / STRIP + (kErpOut ? 1 : 0);  // and the seam's
    const dim3 grid((strips + MESH_WARPS - 1) / MESH_WARPS, (sh.max_h - 1 + rows - 1) / rows, sh.slots * gv);
    launch_dependent(mesh_kernel<kIn, kErpOut, kScaled, Tabs>, grid, dim3(32 * MESH_WARPS), 0, s, tabs, g0, gv, rows);
}

// The kernel instantiated for what the launch holds (without the projections
// and the scaling that do not occur, and with a column's factors held across its
// rows, it needs fewer registers and constants: 4 x 1920x1080 193 -> 173 us the
// stage, into 960x540 152 -> 134, 8 poses 160 -> 149 us a view); the rarer
// mixtures share general ones.
template <class Tabs>
static void launch_mesh_kernels(const Tabs& tabs, const BatchShape& sh, int g0, int gv, cudaStream_t s) {
    if (sh.erp_out) {
        if (sh.inputs == kErpIn && !sh.rescale)
            launch_mesh_kernel<kErpIn, true, false>(tabs, sh, g0, gv, s);
        else
            launch_mesh_kernel<kAnyIn, true, true>(tabs, sh, g0, gv, s);
    } else if (sh.inputs == kPerspectiveIn) {
        if (sh.rescale)
            launch_mesh_kernel<kPerspectiveIn, false, true>(tabs, sh, g0, gv, s);
        else
            launch_mesh_kernel<kPerspectiveIn, false, false>(tabs, sh, g0, gv, s);
    } else if (sh.inputs == kErpIn && !sh.rescale) {
        launch_mesh_kernel<kErpIn, false, false>(tabs, sh, g0, gv, s);
    } else {
        launch_mesh_kernel<kAnyIn, false, true>(tabs, sh, g0, gv, s);
    }
}

template <class Tabs>
int launch_mesh(const Tabs& tabs, const BatchShape& sh, int g0, cudaStream_t s, cudaEvent_t* ev) {
    const int gv = std::min(sh.vg, sh.max_views - g0);
    const size_t words = (size_t)gv * sh.max_wo * sh.max_ho;
    if (ev) cudaEventRecord(ev[0], s);
    launch_dependent(clear_kernel<Tabs>, dim3((unsigned)std::min<size_t>(2048, (words / 2 + 255) / 256 + 1), sh.slots),
                     dim3(256), 0, s, tabs, g0, gv);
    launch_mesh_kernels(tabs, sh, g0, gv, s);
    if (ev) {
        cudaEventRecord(ev[1], s);
        cudaEventRecord(ev[2], s);
    }
    launch_dependent(large_kernel<Tabs>, dim3(std::max(1, 148 * 8 / sh.slots), sh.slots), dim3(LARGE_THREADS), 0, s,
                     tabs, g0, gv);
    if (ev) cudaEventRecord(ev[3], s);
    return 3;
}

template int launch_mesh<TableParam>(const TableParam&, const BatchShape&, int, cudaStream_t, cudaEvent_t*);
template int launch_mesh<TablePtr>(const TablePtr&, const BatchShape&, int, cudaStream_t, cudaEvent_t*);

}  // namespace rvsb
