// Resolve stage: every view's winning fragment of an output pixel,
// re-evaluated exactly from its z-buffer key (resolve.cuh), blended in view
// order into the output colour, quantised and written as 4:2:0, with the
// packed codes and the hole mask for the inpainting passes.
//
// One thread per pixel; a warp covers 16 x 2 pixels, so a 2x2 chroma block
// is four of its lanes, and a CTA 32 x 8, whose fragments share vertices and
// colours through L1.
//
// Bound by instruction issue and the latency of the gathers (three vertices,
// three colours per pixel and view) together: 4 views of 1920x1080 take 105
// us (8.3 M pixel-views; their keys, vertices and colours, each read once,
// are 265 MB, 41 us), 97 us a view in a batch of 8.  Five CTAs per SM at 48
// registers beat four at 64 (in one kernel for all options: batch 107 against
// 117 us), two views' gathers in flight per thread (116) and six CTAs at 40
// registers (112).
#include <algorithm>

#include "device_common.cuh"
#include "kernels.hpp"
#include "resolve.cuh"

namespace rvsb {
namespace {

using namespace dev;

constexpr int TILE_W = 32, TILE_H = 8;

// The fields of a view the resolve reads.
struct __align__(16) ResolveView {
    const float4* vert;
    const uint64_t* color;
    const unsigned long long* z;
    int w, tri_shift;
    float color_scale;
    int hole;  // of the first: whether the CTA has reported a hole
};

// Grid (ceil(max_wo / 32), ceil(max_ho / 8), slots): views g0 .. g0 + gv - 1
// of every slot; the last group of a slot's views writes its output, earlier
// ones keep the running blend in acc01 / acc23.  Extras: the per-view
// multispectral, auxiliary and debug outputs are written.  kWrap, kScaled: some
// output wraps horizontally (seam triangles), some Precision differs from 1;
// kIntPow: every blending exponent is an integer from 2 to 16.  Without what
// does not occur: 8 poses of the 1080p scene 105 -> 97 us a view.
template <bool Extras, bool kWrap, bool kScaled, bool kIntPow, class Tabs>
__global__ void __launch_bounds__(TILE_W * TILE_H, 5) resolve_kernel(const __grid_constant__ Tabs tabs, int g0, int gv) {
    grid_dep_wait();
    const SlotTable& tab = tabs.at(blockIdx.z);
    const DevTarget& T = tab.t;
    if (g0 >= T.n_views) return;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int x = blockIdx.x * TILE_W + (warp & 1) * 16 + (lane & 15);
    const int y = blockIdx.y * TILE_H + (warp >> 1) * 2 + (lane >> 4);
    if (blockIdx.x * TILE_W >= T.wo || blockIdx.y * TILE_H >= T.ho) return;
    const bool inside = x < T.wo && y < T.ho;
    const int g1 = min(T.n_views, g0 + gv);
    // The views' fields once per CTA, in shared memory: the table is indexed by
    // a loop variable, so each use of it would be a load of its own.
    __shared__ ResolveView s_view[MAX_VIEWS];
    if ((int)threadIdx.x < g1 - g0) {
        const DevView& G = tab.v[g0 + threadIdx.x];
        s_view[threadIdx.x] = ResolveView{G.vert, G.color, G.z, G.w, G.tri_shift, G.color_scale, 0};
    }
    __syncthreads();
    const size_t npo = (size_t)T.wo * T.ho;
    const size_t po = inside ? (size_t)y * T.wo + x : 0;
    BlendAcc a = {0.f, 0.f, 0.f, 0.f};
    uint64_t code = 0;
    bool hole = false;
    if (inside) {
        if (g0 > 0) {
            const float2 p = tab.b.acc01[po], q = tab.b.acc23[po];
            a.c0 = p.x; a.c1 = p.y; a.c2 = q.x; a.q = q.y;
        }
        const bool aux = Extras && tab.aux.on != 0;
        float adepth = 0.f, avalid = 0.f;
        if (aux && g0 > 0) {
            adepth = tab.aux.acc_depth[po];
            avalid = tab.aux.acc_valid[po];
        }
        unsigned long long key = __ldg(s_view[0].z + po);
        for (int v = g0; v < g1; ++v) {
            const unsigned long long cur = key;
            if (v + 1 < g1) key = __ldg(s_view[v + 1 - g0].z + po);
            const Fragment f = resolve_fragment<kWrap, kScaled>(s_view[v - g0], cur, x, y, T.precision);
            const float qv = __fdiv_rn(f.validity, f.depth);
            if (Extras && tab.ms.on) {
                tab.ms.yq[(size_t)v * npo + po] = make_float2(f.col.x, qv);
                tab.ms.uv[(size_t)v * npo + po] = make_float2(f.col.y, f.col.z);
            }
            if (aux) {
                // BlendedView.cpp:205-208: the view's depth where its quality
                // beats the accumulator's before this blend (view 0: its
                // quality; later: (weight sum)^(1/exp)); validity = max.
                if (v == 0) {
                    adepth = f.depth;
                    avalid = f.validity;
                } else {
                    const float qacc =
                        (v == 1 || T.blend_max) ? a.q : (a.q > 0.f ? powf(a.q, T.inv_blend_exp) : a.q);
                    if (qv > qacc) adepth = f.depth;
                    avalid = smax(avalid, f.validity);
                }
            }
            if (Extras) {
                const DebugPtrs& dbg = tab.dbg;
                const size_t o = (size_t)v * npo + po;
                if (dbg.view_color) {
                    float* c = dbg.view_color + o * 3;
                    c[0] = f.col.x; c[1] = f.col.y; c[2] = f.col.z;
                }
                if (dbg.view_depth) dbg.view_depth[o] = f.depth;
                if (dbg.view_validity) dbg.view_validity[o] = f.validity;
            }
            blend_view<kIntPow>(a, v, f, qv, T);
        }
        if (aux) {
            tab.aux.acc_depth[po] = adepth;
            tab.aux.acc_valid[po] = avalid;
        }
    }
    if (g1 < T.n_views) {
        if (inside) {
            tab.b.acc01[po] = make_float2(a.c0, a.c1);
            tab.b.acc23[po] = make_float2(a.c2, a.q);
        }
        return;
    }
    // Quantisation and write (image_writing.cpp:142-180).
    if (inside) {
        hole = !(a.q > 0.f);
        code = (uint64_t)quantize(a.c0, T.max_val) | ((uint64_t)quantize(a.c1, T.max_val) << 16) |
               ((uint64_t)quantize(a.c2, T.max_val) << 32) | (hole ? kHoleBit : 0ull);
        tab.b.codes[po] = code;
        if (kScaled && T.rescale) tab.b.pcolor[po] = make_float4(a.c0, a.c1, a.c2, 0.f);
        if (Extras) {
            const DebugPtrs& dbg = tab.dbg;
            if (dbg.blend_color) {
                dbg.blend_color[po * 3 + 0] = a.c0;
                dbg.blend_color[po * 3 + 1] = a.c1;
                dbg.blend_color[po * 3 + 2] = a.c2;
            }
            if (dbg.blend_quality)
                dbg.blend_quality[po] =
                    (T.n_views == 1 || T.blend_max || !(a.q > 0.f)) ? a.q : powf(a.q, T.inv_blend_exp);
            if (dbg.inpaint_source) {
                dbg.inpaint_source[po * 2 + 0] = x;
                dbg.inpaint_source[po * 2 + 1] = y;
            }
        }
    }
    const unsigned hm = __ballot_sync(0xffffffffu, hole);
    if (!(kScaled && T.rescale)) {
        // 2x2 blocks without holes (the inpainting passes write the others);
        // the output's sides are even, so every block is whole.
        uint32_t su = (uint32_t)(code >> 16) & 0xffffu, sv = (uint32_t)(code >> 32) & 0xffffu;
        su += __shfl_xor_sync(0xffffffffu, su, 1);
        sv += __shfl_xor_sync(0xffffffffu, sv, 1);
        su += __shfl_xor_sync(0xffffffffu, su, 16);
        sv += __shfl_xor_sync(0xffffffffu, sv, 16);
        const unsigned block = 0x00030003u << (lane & 14);
        if (inside && !(hm & block)) {
            tab.out_y[po] = (uint16_t)(code & 0xffff);
            if (!(lane & 17)) {
                const size_t co = (size_t)(y / 2) * (T.wo / 2) + x / 2;
                tab.out_u[co] = quarter_round(su, T.chroma_ties_up);
                tab.out_v[co] = quarter_round(sv, T.chroma_ties_up);
            }
        }
    }
    // Hole bits, 16 columns of each of the warp's two rows; those beyond the
    // width are set.
    const unsigned bits = hm | __ballot_sync(0xffffffffu, x >= T.wo);
    if (!(lane & 15) && y < T.ho) {
        const int words = (T.wo + 31) / 32;
        reinterpret_cast<uint16_t*>(tab.b.holes + (size_t)y * words)[x >> 4] = (uint16_t)(bits >> (lane & 16));
    }
    // Once per CTA: the stores of all warps to one address take their turns, half
    // of the kernel's time where most of a large view is a hole (2 x 640x360 into
    // 3840x2160 looking away 240 -> 130 us, into ERP 4096x2048 267 -> 142).
    if (hm && lane == 0 && atomicExch(&s_view[0].hole, 1) == 0) tab.b.status->n_holes = 1;
}

}  // namespace

template <class Tabs>
void launch_resolve(const Tabs& tabs, const BatchShape& sh, int g0, cudaStream_t s) {
    const int gv = std::min(sh.vg, sh.max_views - g0);
    const dim3 grid((sh.max_wo + TILE_W - 1) / TILE_W, (sh.max_ho + TILE_H - 1) / TILE_H, sh.slots);
    auto go = [&](auto kernel) { launch_dependent(kernel, grid, dim3(TILE_W * TILE_H), 0, s, tabs, g0, gv); };
    if (sh.extras)
        go(resolve_kernel<true, true, true, false, Tabs>);
    else if (sh.erp_out || sh.rescale)
        go(resolve_kernel<false, true, true, false, Tabs>);
    else if (sh.int_pow)
        go(resolve_kernel<false, false, false, true, Tabs>);
    else
        go(resolve_kernel<false, false, false, false, Tabs>);
}

template void launch_resolve<TableParam>(const TableParam&, const BatchShape&, int, cudaStream_t);
template void launch_resolve<TablePtr>(const TablePtr&, const BatchShape&, int, cudaStream_t);

}  // namespace rvsb
