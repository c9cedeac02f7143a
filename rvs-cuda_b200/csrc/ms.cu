// Multispectral blending (BlendedViewMultiSpec, rvs/src/BlendedView.cpp:63-88),
// after the resolve has stored every view's resolved colour and quality:
// split_frequencies (blending.cpp:371-395; YUV: only luma is blurred) with
// calcBlurring (blending.cpp:62-105: box mean over the masked pixels of a
// (2r+1)^2 window clipped to the image, r = max(W, H) / 20, the window sum
// truncated to an integer before the division by the count, 0 outside the
// mask of quality > 0), then the low band (blur(Y), U, V) and the high band
// (Y - blur(Y), 0, 0) blended separately with their own factors and added.
// The window sums are accumulated in double as the reference's integral
// image is; only their order differs, which can change a truncated sum only
// when it lies within about 1e-10 of an integer.
#include "device_common.cuh"
#include "kernels.hpp"
#include "resolve.cuh"

namespace rvsb {
namespace {

using namespace dev;

constexpr int MS_THREADS = 512;
constexpr int MS_WARPS = MS_THREADS / 32;
constexpr int MS_CHUNKS = 4;   // 32-column chunks a warp holds at once
constexpr int MS_COLS = 128;   // columns per CTA of the column windows
constexpr int MS_ROWS = 64;    // rows a thread of it slides over
constexpr int MS_BATCH = 8;    // of them loaded together

// Row-window sums of masked luma: one CTA per (row, view, slot).  The row's
// exclusive prefix (double sums, integer counts) is built in shared memory:
// each warp scans MS_CHUNKS chunks of 32 columns, loaded together and
// coalesced, the warps' totals are added, and wide rows take several rounds.
// Bound by latency between its barriers: 54 us on 4 views of 1920x1080 (66 MB
// in, 100 out) with four 512-thread CTAs per SM, 60 with three, 62 with four
// of 256 threads and twice the chunks; a run of consecutive columns per
// thread, read twice, 16 bytes every 128, took 162.
template <class Tabs>
__global__ void __launch_bounds__(MS_THREADS, 4) ms_rows_kernel(const __grid_constant__ Tabs tabs) {
    grid_dep_wait();
    extern __shared__ __align__(16) unsigned char s_raw[];
    const SlotTable& tab = tabs.at(blockIdx.z);
    const MsPtrs& M = tab.ms;
    if (!M.on) return;
    const DevTarget& T = tab.t;
    const int v = blockIdx.y, y = blockIdx.x;
    if (v >= T.n_views || y >= T.ho) return;
    const int w = T.wo;
    double* P = reinterpret_cast<double*>(s_raw);                     // w + 1 prefix sums
    int* C = reinterpret_cast<int*>(s_raw + sizeof(double) * (w + 1));  // w + 1 prefix counts
    __shared__ double s_wsum[MS_WARPS];
    __shared__ int s_wcnt[MS_WARPS];
    const size_t npo = (size_t)T.wo * T.ho;
    const float2* row = M.yq + (size_t)v * npo + (size_t)y * w;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double base = 0.0;
    int cbase = 0;
    if (threadIdx.x == 0) {
        P[0] = 0.0;
        C[0] = 0;
    }
    for (int r0 = 0; r0 < w; r0 += MS_THREADS * MS_CHUNKS) {
        const int x0 = r0 + warp * 32 * MS_CHUNKS + lane;
        double s[MS_CHUNKS];
        unsigned mask[MS_CHUNKS];
#pragma unroll
        for (int k = 0; k < MS_CHUNKS; ++k) {
            const int x = x0 + 32 * k;
            float2 c = make_float2(0.f, 0.f);
            if (x < w) c = row[x];
            const bool in = c.y > 0.f && isfinite(c.x);
            mask[k] = __ballot_sync(0xffffffffu, in);
            s[k] = in ? (double)c.x : 0.0;
        }
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
#pragma unroll
            for (int k = 0; k < MS_CHUNKS; ++k) {
                const double a = __shfl_up_sync(0xffffffffu, s[k], o);
                if (lane >= o) s[k] += a;
            }
        }
        double run = 0.0;
        int crun = 0;
        int cnt[MS_CHUNKS];
#pragma unroll
        for (int k = 0; k < MS_CHUNKS; ++k) {
            const double t = __shfl_sync(0xffffffffu, s[k], 31);
            s[k] += run;
            cnt[k] = crun + __popc(mask[k] & (0xffffffffu >> (31 - lane)));
            run += t;
            crun += __popc(mask[k]);
        }
        if (lane == 0) {
            s_wsum[warp] = run;
            s_wcnt[warp] = crun;
        }
        __syncthreads();
        double before = base;
        int cbefore = cbase;
#pragma unroll
        for (int k = 0; k < MS_WARPS; ++k) {
            if (k < warp) {
                before += s_wsum[k];
                cbefore += s_wcnt[k];
            }
            base += s_wsum[k];
            cbase += s_wcnt[k];
        }
#pragma unroll
        for (int k = 0; k < MS_CHUNKS; ++k) {
            const int x = x0 + 32 * k;
            if (x < w) {
                P[x + 1] = before + s[k];
                C[x + 1] = cbefore + cnt[k];
            }
        }
        __syncthreads();
    }
    const int rad = M.rad;
    double* hs = M.hsum + (size_t)v * npo + (size_t)y * w;
    int* hc = M.hcnt + (size_t)v * npo + (size_t)y * w;
    for (int x = threadIdx.x; x < w; x += MS_THREADS) {
        const int a = max(0, x - rad), b = min(w, x - rad + 2 * rad + 1);
        hs[x] = P[b] - P[a];
        hc[x] = C[b] - C[a];
    }
}

// Column windows of the row sums: a thread per column and view slides over
// MS_ROWS rows, from a window summed up anew.  At 1080 rows and a radius of
// 54 that reads each row sum 3.7 times instead of twice, but runs 17 times as
// many threads, and the loads of MS_BATCH rows are in flight together: 54 us
// on 4 views of 1920x1080 against 827 us with one thread per whole column
// (60 CTAs of 128 threads on 148 SMs); 32 and 128 rows: 64 and 62 us, 4 rows
// in flight and 12 CTAs per SM 79.
// Writes the blurred luma.
// Grid (ceil(max_wo / MS_COLS) * segments, views, slots).
template <class Tabs>
__global__ void __launch_bounds__(MS_COLS, 7) ms_cols_kernel(const __grid_constant__ Tabs tabs, int segments) {
    grid_dep_wait();
    const SlotTable& tab = tabs.at(blockIdx.z);
    const MsPtrs& M = tab.ms;
    if (!M.on) return;
    const DevTarget& T = tab.t;
    const int v = blockIdx.y, x = blockIdx.x / segments * MS_COLS + threadIdx.x;
    const int w = T.wo, h = T.ho, rad = M.rad;
    const int y0 = (int)(blockIdx.x % segments) * MS_ROWS, y1 = min(h, y0 + MS_ROWS);
    if (v >= T.n_views || x >= w || y0 >= h) return;
    const size_t npo = (size_t)w * h;
    const double* hs = M.hsum + (size_t)v * npo + x;
    const int* hc = M.hcnt + (size_t)v * npo + x;
    float* out = M.blur + (size_t)v * npo + x;
    double s = 0.0;
    int c = 0;
    const int ya = max(0, y0 - rad), yb = min(h - 1, y0 + rad);
#pragma unroll 8
    for (int y = ya; y <= yb; ++y) {
        s += __ldg(hs + (size_t)y * w);
        c += __ldg(hc + (size_t)y * w);
    }
    // The rows entering and leaving the window, MS_BATCH at a time, before
    // the sums that wait for them.
    for (int yb0 = y0; yb0 < y1; yb0 += MS_BATCH) {
        double sin[MS_BATCH], sout[MS_BATCH];
        int cin[MS_BATCH], cout[MS_BATCH];
#pragma unroll
        for (int k = 0; k < MS_BATCH; ++k) {
            const int yin = yb0 + k + rad + 1, yout = yb0 + k - rad;
            const bool i = yin < h, o = yout >= 0 && yout < h;
            sin[k] = i ? __ldg(hs + (size_t)yin * w) : 0.0;
            cin[k] = i ? __ldg(hc + (size_t)yin * w) : 0;
            sout[k] = o ? __ldg(hs + (size_t)yout * w) : 0.0;
            cout[k] = o ? __ldg(hc + (size_t)yout * w) : 0;
        }
#pragma unroll
        for (int k = 0; k < MS_BATCH; ++k) {
            if (yb0 + k < y1) out[(size_t)(yb0 + k) * w] = c > 0 ? __fdiv_rn((float)(unsigned)(int)s, (float)c) : 0.f;
            s += sin[k];
            c += cin[k];
            s -= sout[k];
            c -= cout[k];
        }
    }
}

constexpr int MS_TILE_W = 32, MS_TILE_H = 8;
constexpr int MS_VIEWS = 4;

// The two bands' blends per pixel, added: rewrites the colour part of the
// codes (the holes stay the raster's) and the output samples of hole-free 2x2
// blocks.  One thread per pixel, a warp 16 x 2 of them (the lanes of a chroma
// block exchange its samples).  Bound by the latency of its loads: with
// MS_VIEWS views' values loaded together 54 us on 4 views of 1920x1080 (180
// MB, 28 us at the copy rate), one or two at a time 95.
// Grid (ceil(max_wo / 32), ceil(max_ho / 8), slots).
template <class Tabs>
__global__ void __launch_bounds__(MS_TILE_W * MS_TILE_H, 6) ms_blend_kernel(const __grid_constant__ Tabs tabs) {
    grid_dep_wait();
    const SlotTable& tab = tabs.at(blockIdx.z);
    const MsPtrs& M = tab.ms;
    if (!M.on) return;
    const DevTarget& T = tab.t;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int x = blockIdx.x * MS_TILE_W + (warp & 1) * 16 + (lane & 15);
    const int y = blockIdx.y * MS_TILE_H + (warp >> 1) * 2 + (lane >> 4);
    const bool inside = x < T.wo && y < T.ho;
    const size_t npo = (size_t)T.wo * T.ho, o = inside ? (size_t)y * T.wo + x : 0;
    uint64_t code = 0;
    bool hole = false;
    if (inside) {
        BlendAcc lo = {0.f, 0.f, 0.f, 0.f}, hi = {0.f, 0.f, 0.f, 0.f};
        // The views' values MS_VIEWS at a time, before the blends that wait
        // for them.
        for (int v0 = 0; v0 < T.n_views; v0 += MS_VIEWS) {
            float2 yq[MS_VIEWS], uv[MS_VIEWS];
            float blur[MS_VIEWS];
#pragma unroll
            for (int k = 0; k < MS_VIEWS; ++k) {
                const size_t q = (size_t)min(v0 + k, T.n_views - 1) * npo + o;
                yq[k] = M.yq[q];
                uv[k] = M.uv[q];
                blur[k] = M.blur[q];
            }
#pragma unroll
            for (int k = 0; k < MS_VIEWS; ++k) {
                if (v0 + k >= T.n_views) break;
                // 0 outside the mask of quality > 0
                const float b = yq[k].y > 0.f ? blur[k] : 0.f;
                const float3 lowc = make_float3(b, uv[k].x, uv[k].y);
                const float3 highc = make_float3(__fsub_rn(yq[k].x, b), __fsub_rn(uv[k].x, uv[k].x),
                                                 __fsub_rn(uv[k].y, uv[k].y));
                blend_view(lo, v0 + k, lowc, yq[k].y, M.low_exp, M.low_int, M.low_exp < 0.f);
                blend_view(hi, v0 + k, highc, yq[k].y, M.high_exp, M.high_int, M.high_exp < 0.f);
            }
        }
        const float f0 = __fadd_rn(lo.c0, hi.c0), f1 = __fadd_rn(lo.c1, hi.c1), f2 = __fadd_rn(lo.c2, hi.c2);
        if (T.rescale) tab.b.pcolor[o] = make_float4(f0, f1, f2, 0.f);
        hole = tab.b.holes[(size_t)y * ((T.wo + 31) / 32) + (x >> 5)] >> (x & 31) & 1u;
        code = (uint64_t)quantize(f0, T.max_val) | ((uint64_t)quantize(f1, T.max_val) << 16) |
               ((uint64_t)quantize(f2, T.max_val) << 32) | (hole ? kHoleBit : 0ull);
        tab.b.codes[o] = code;
        if (tab.dbg.blend_color) {
            tab.dbg.blend_color[o * 3 + 0] = f0;
            tab.dbg.blend_color[o * 3 + 1] = f1;
            tab.dbg.blend_color[o * 3 + 2] = f2;
        }
    }
    if (T.rescale) return;  // written by the resize
    const unsigned hm = __ballot_sync(0xffffffffu, hole);
    uint32_t su = (uint32_t)(code >> 16) & 0xffffu, sv = (uint32_t)(code >> 32) & 0xffffu;
    su += __shfl_xor_sync(0xffffffffu, su, 1);
    sv += __shfl_xor_sync(0xffffffffu, sv, 1);
    su += __shfl_xor_sync(0xffffffffu, su, 16);
    sv += __shfl_xor_sync(0xffffffffu, sv, 16);
    // Blocks with holes are the inpainting's.
    if (!inside || (hm & (0x00030003u << (lane & 14)))) return;
    tab.out_y[o] = (uint16_t)(code & 0xffff);
    if (!(lane & 17)) {
        const size_t co = (size_t)(y / 2) * (T.wo / 2) + x / 2;
        tab.out_u[co] = quarter_round(su, T.chroma_ties_up);
        tab.out_v[co] = quarter_round(sv, T.chroma_ties_up);
    }
}

}  // namespace

template <class Tabs>
int launch_ms(const Tabs& tabs, const BatchShape& sh, cudaStream_t s) {
    const size_t smem = (sizeof(double) + sizeof(int)) * (size_t)(sh.max_wo + 1);
    launch_dependent(ms_rows_kernel<Tabs>, dim3(sh.max_ho, sh.max_views, sh.slots), dim3(MS_THREADS), smem, s, tabs);
    const int segments = (sh.max_ho + MS_ROWS - 1) / MS_ROWS;
    launch_dependent(ms_cols_kernel<Tabs>, dim3((sh.max_wo + MS_COLS - 1) / MS_COLS * segments, sh.max_views, sh.slots),
                     dim3(MS_COLS), 0, s, tabs, segments);
    launch_dependent(ms_blend_kernel<Tabs>, dim3((sh.max_wo + MS_TILE_W - 1) / MS_TILE_W, (sh.max_ho + MS_TILE_H - 1) / MS_TILE_H, sh.slots),
                     dim3(MS_TILE_W * MS_TILE_H), 0, s, tabs);
    return 3;
}

void prepare_ms_kernels(int max_wo) {
    const int smem = (int)((sizeof(double) + sizeof(int)) * (size_t)(max_wo + 1));
    if (smem > 48 * 1024) {
        cudaFuncSetAttribute(ms_rows_kernel<TableParam>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        cudaFuncSetAttribute(ms_rows_kernel<TablePtr>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    }
}

template int launch_ms<TableParam>(const TableParam&, const BatchShape&, cudaStream_t);
template int launch_ms<TablePtr>(const TablePtr&, const BatchShape&, cudaStream_t);

}  // namespace rvsb
