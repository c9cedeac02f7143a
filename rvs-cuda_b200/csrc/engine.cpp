// Host engine: device memory, slot workspaces, slot tables and batch launches.
#include "engine.hpp"

#include <algorithm>
#include <climits>
#include <cmath>
#include <cstring>

#include "camera.hpp"
#include "frontend.hpp"

namespace rvsb {

void check(cudaError_t e, const char* what) {
    if (e != cudaSuccess) throw CudaError(std::string(what) + ": " + cudaGetErrorString(e));
}

void DevMem::alloc(rvsb_context* c, size_t n) {
    release();
    if (n == 0) n = 16;
    {
        std::lock_guard<std::mutex> lock(c->mem_mu);
        if (c->in_use + n > c->budget)
            throw BudgetError("request of " + std::to_string(n) + " bytes exceeds the HBM budget (" +
                              std::to_string(c->in_use) + " of " + std::to_string(c->budget) + " in use)");
        c->in_use += n;
    }
    const cudaError_t e = cudaMalloc(&ptr, n);
    if (e != cudaSuccess) {
        ptr = nullptr;
        std::lock_guard<std::mutex> lock(c->mem_mu);
        c->in_use -= n;
        check(e, "cudaMalloc");
    }
    ctx = c;
    bytes = n;
}

void DevMem::release() {
    if (ptr) {
        cudaFree(ptr);
        std::lock_guard<std::mutex> lock(ctx->mem_mu);
        ctx->in_use -= bytes;
    }
    ptr = nullptr;
    bytes = 0;
}

RasterDims raster_dims(const rvsb_camera& virt, const rvsb_synth_params& p) {
    if (!std::isfinite(p.precision) || !(p.precision > 0.f)) throw Unsupported("Precision must be positive");
    if (p.precision == 1.f) return {virt.width, virt.height, false};
    const int w = (int)(0.5f + (float)virt.width * p.precision);
    const int h = (int)(0.5f + (float)virt.height * p.precision);
    if (w < 2 || h < 2 || w > 32768 || h > 32768)
        throw Unsupported("Precision " + std::to_string(p.precision) + " gives a raster size of " +
                          std::to_string(w) + "x" + std::to_string(h) +
                          "; only sizes of at least 2 and at most 32768 are supported");
    return {w, h, true};
}

namespace {

struct SlotNeeds {
    size_t vert, out, large, hole_words, sum_words;
};

SlotNeeds needs_of(const rvsb_scene* sc, int wo, int ho) {
    SlotNeeds n{};
    for (const auto& c : sc->cams) n.vert += (size_t)c.width * c.height;
    n.out = (size_t)wo * ho;
    n.hole_words = (size_t)((wo + 31) / 32) * ho;
    n.sum_words = inpaint_sum_words(wo, ho);
    // About 1% of the triangles of an unmagnified view are large; when they
    // do not fit, large_kernel goes over the whole mesh.
    n.large = std::min<size_t>(INT32_MAX / 2, std::max<size_t>(1 << 14, n.vert / 11));
    return n;
}

}  // namespace

size_t SlotWorkspace::bytes_for(const rvsb_scene* sc, int wo, int ho, bool rescale) {
    const SlotNeeds n = needs_of(sc, wo, ho);
    return sizeof(DevStatus) + n.vert * sizeof(float4) + n.large * sizeof(uint4) + n.out * sizeof(uint64_t) * 5 +
           n.hole_words * sizeof(uint32_t) + n.sum_words * sizeof(uint64_t) + (rescale ? n.out * (sizeof(float4) + 2 * sizeof(int32_t)) : 0);
}

// Grows `m` to at least n bytes.  What it holds is its allocation's own size, so
// that a buffer whose growth failed counts as empty in the calls that follow.
static void grow(rvsb_context* ctx, DevMem& m, size_t n) {
    if (m.bytes < n) m.alloc(ctx, n);
}

void SlotWorkspace::ensure_rescale(rvsb_context* ctx, int wo, int ho) {
    const size_t n = (size_t)wo * ho;
    grow(ctx, pcolor, n * sizeof(float4));
    grow(ctx, psrc, n * 2 * sizeof(int32_t));
}

void SlotWorkspace::ensure(rvsb_context* ctx, const rvsb_scene* sc, int wo, int ho) {
    const SlotNeeds n = needs_of(sc, wo, ho);
    grow(ctx, status, sizeof(DevStatus));
    grow(ctx, vert, n.vert * sizeof(float4));
    grow(ctx, large, n.large * sizeof(uint4));
    grow(ctx, holes, n.hole_words * sizeof(uint32_t));
    grow(ctx, inpaint_sum, n.sum_words * sizeof(uint64_t));
    grow(ctx, codes, n.out * sizeof(uint64_t));
    grow(ctx, scan, 4 * n.out * sizeof(uint64_t));
}

void SlotWorkspace::ensure_aux(rvsb_context* ctx, int wo, int ho) {
    const size_t n = (size_t)wo * ho;
    grow(ctx, aux_depth, n * sizeof(float));
    grow(ctx, aux_valid, n * sizeof(float));
}

void SlotWorkspace::ensure_ms(rvsb_context* ctx, int n_views, int wo, int ho) {
    const size_t n = (size_t)n_views * wo * ho;
    grow(ctx, ms_view, n * sizeof(float4));
    grow(ctx, ms_hsum, n * sizeof(double));
    grow(ctx, ms_hcnt, n * sizeof(int));
    grow(ctx, ms_blur, n * sizeof(float));
}

BatchCore::BatchCore(rvsb_context* ctx, int slots) : ctx_(ctx), slots_(slots) {
    if (slots <= 0) throw ArgError("a batch needs at least one slot");
    for (int k = 0; k < slots; ++k) ws_.push_back(std::make_unique<SlotWorkspace>());
    tables_.alloc(ctx, sizeof(SlotTable) * (size_t)slots);
    for (int b = 0; b < 2; ++b) {
        void* p = nullptr;
        check(cudaHostAlloc(&p, sizeof(SlotTable) * (size_t)slots, cudaHostAllocDefault), "cudaHostAlloc");
        staging_[b] = static_cast<SlotTable*>(p);
        check(cudaEventCreateWithFlags(&copied_[b], cudaEventDisableTiming), "cudaEventCreate");
    }
    check(cudaStreamCreateWithFlags(&capture_, cudaStreamNonBlocking), "cudaStreamCreate");
    for (auto& e : tune_ev_) check(cudaEventCreate(&e), "cudaEventCreate");
}

BatchCore::~BatchCore() {
    for (auto& g : graphs_) cudaGraphExecDestroy(g.second.exec);
    for (int b = 0; b < 2; ++b) {
        if (copied_[b]) {
            cudaEventSynchronize(copied_[b]);
            cudaEventDestroy(copied_[b]);
        }
        if (staging_[b]) cudaFreeHost(staging_[b]);
    }
    for (auto& e : events_)
        if (e) cudaEventDestroy(e);
    if (capture_) cudaStreamDestroy(capture_);
    for (auto& e : tune_ev_)
        if (e) cudaEventDestroy(e);
}

void BatchCore::set_profiling(bool on) {
    if (on && !events_[0])
        for (auto& e : events_) check(cudaEventCreate(&e), "cudaEventCreate");
    profiling_ = on;
}

int BatchCore::stage_times(float* ms, int max_stages) const {
    if (!profiled_ || !ms) return -1;
    const int n = std::min(max_stages, (int)NUM_STAGES);
    for (int k = 0; k < n; ++k) {
        if (cudaEventElapsedTime(&ms[k], events_[2 * k], events_[2 * k + 1]) != cudaSuccess) {
            cudaGetLastError();
            return -1;
        }
    }
    return n;
}

namespace {

// Pixels per radian at the centre of a camera: the focal length of a
// perspective camera, the width over the horizontal range of an
// equirectangular one.
float pixels_per_radian(const rvsb_camera& c) {
    if (c.projection == RVSB_PROJ_EQUIRECTANGULAR) {
        const float range = (c.hor_range[1] - c.hor_range[0]) * (3.14159265f / 180.f);
        return range > 0.f ? (float)c.width / range : 0.f;
    }
    return c.focal[0];
}

// Magnification of a synthesis: output pixels per radian at the raster size
// over the densest input's.  An equirectangular output stretches its rows by
// 1 / cos(latitude), sqrt(2) at the median row, which its m includes.
float magnification(const SlotRequest& r) {
    float in = 0.f;
    for (const rvsb_camera& c : r.scene->cams) in = std::max(in, pixels_per_radian(c));
    const RasterDims rd = raster_dims(r.virt, r.params);
    float out = pixels_per_radian(r.virt) * (float)rd.w / (float)r.virt.width;
    if (r.virt.projection == RVSB_PROJ_EQUIRECTANGULAR) out *= 1.41421356f;
    return in > 0.f ? out / in : 0.f;
}
// Above it the ordinary triangles have more than the 4 candidates of the
// unmagnified threshold.
constexpr float kMagnified = 1.1f;

// Candidate pixels up to which a view's triangles stay with their lanes.  An
// input pixel spacing seen m times magnified gives candidate boxes of about m + 1
// pixels a side, somewhat more where the surface is slanted.  A threshold below
// that lists nearly every triangle, which overflows the list: 3 x ERP 1102x550
// into ERP 3890x1944 (m = 5) 1303 us with 16, 724 with 49; 2 x 480x270 into
// 1920x1080 (m = 4) 211 with 16, 146 with 25, 149 with 36.  One far above it
// leaves stretched triangles to single lanes: m = 2, 193 us with 9 and 16, 211
// with 36, 270 with 120.  Below 16 nothing is gained (m = 1.5, 224 us with 4 to
// 16).
//
// The more a view is magnified, the fewer of its triangles are in sight (two per
// m x m output pixels and view): a few warps then walk through large boxes while
// the rest of the chip has nothing to do.  Past kFewInSight they go to the list,
// which all warps share, where it holds them: 3 x 960x540 into the same size at m
// = 5 124 -> 101 us, at m = 10 215 -> 96, at m = 20 410 -> 87; 16 x 1920x1080 at
// m = 20 4735 -> 995.  At m = 4 that gains as often as it loses (16 x 1920x1080
// 1802 -> 1525, 4 x ERP 4096x2048 into 1920x1080 342 -> 349).  Where the list
// cannot hold them the pass over the whole mesh shares them out as well, which
// pays past kShared: 2 x 192x108 into 1920x1080 (m = 10) 237 -> 158 us, 2 x 96x54
// (m = 20) 463 -> 170, but 2 x 400x225 (m = 4.8) 161 -> 187.
constexpr float kFewInSight = 4.5f, kShared = 10.f;

int candidate_threshold(const SlotRequest& r) {
    const float m = magnification(r);
    if (!(m > kMagnified) || m > kShared) return 4;
    if (m > kFewInSight) {
        const RasterDims rd = raster_dims(r.virt, r.params);
        double in_sight = 0.0;
        const size_t group = std::min<size_t>(4, r.scene->cams.size());
        for (size_t v = 0; v < group; ++v) {
            const rvsb_camera& c = r.scene->cams[v];
            in_sight += 2.0 * std::min((double)c.width * c.height, (double)rd.w * rd.h / ((double)m * m));
        }
        if (in_sight <= 0.75 * (double)needs_of(r.scene, rd.w, rd.h).large) return 4;
    }
    const int side = (int)std::max(4.f, std::ceil(m + 1.2f));
    return side * side;
}

}  // namespace

void BatchCore::fill(SlotTable& T, int k, const SlotRequest& r, const BatchShape& sh) {
    std::memset(&T, 0, sizeof(T));
    const rvsb_scene* sc = r.scene;
    SlotWorkspace& ws = *ws_[k];
    const rvsb_camera& virt = r.virt;
    const rvsb_synth_params& p = r.params;
    const int n = (int)sc->cams.size();
    const RasterDims rd = raster_dims(virt, p);
    const size_t npix = (size_t)rd.w * rd.h;
    size_t voff = 0;
    for (int v = 0; v < n; ++v) {
        const rvsb_camera& c = sc->cams[v];
        DevView& V = T.v[v];
        V.w = c.width;
        V.h = c.height;
        V.proj = c.projection;
        V.bits_color = c.bit_depth_color;
        V.f0 = c.focal[0];
        V.f1 = c.focal[1];
        V.p0 = c.principle_point[0];
        V.p1 = c.principle_point[1];
        V.near_ = c.depth_range[0];
        V.far_ = c.depth_range[1];
        V.depth_scale = 1.0f / (float)((1u << c.bit_depth_depth) - 1u);
        V.has_invalid = c.has_invalid_depth;
        V.color_scale = 1.0f / (float)((1u << c.bit_depth_color) - 1u);
        V.cw = c.width / 2;
        V.ch = c.height / 2;
        V.chroma_sx = (float)V.cw / c.width;
        V.chroma_sy = (float)V.ch / c.height;
        relative_pose(c, virt, V.R, V.t);
        V.py = sc->plane(v, 0);
        V.pu = sc->plane(v, 1);
        V.pv = sc->plane(v, 2);
        V.pd = r.frame ? r.frame[v].depth : sc->plane(v, 3);
        if (c.projection == RVSB_PROJ_EQUIRECTANGULAR) {
            V.erp_row = sc->erp[v * 2 + 0]->as<float>();
            V.erp_col = sc->erp[v * 2 + 1]->as<float>();
            V.erp_cone = sc->erp_cone[v]->as<float4>();
            V.tile_depth = sc->tile_depth[v]->as<float2>();
        }
        V.color = sc->color[v]->as<uint64_t>();
        V.depth_lut = sc->depth_lut[v]->as<float4>();
        V.vert = ws.vert.as<float4>() + voff;
        V.z = ws.scan.as<unsigned long long>() + (size_t)(v % sh.vg) * npix;
        V.tri_shift = 2;
        while ((1 << (V.tri_shift - 2)) < c.width - 1) ++V.tri_shift;
        voff += (size_t)c.width * c.height;
    }
    DevTarget& D = T.t;
    D.wo = rd.w;
    D.ho = rd.h;
    D.out_w = virt.width;
    D.out_h = virt.height;
    D.precision = p.precision;
    D.small = kRasterVariants[sh.variant].small;
    if (D.small == 0) D.small = candidate_threshold(r);
    if (rd.rescale) {
        D.rescale = 1;
        D.uv_sx = (float)rd.w / (float)virt.width;
        D.uv_sy = (float)rd.h / (float)virt.height;
        // cv::resize from the raster size to W x H: an exact 2x reduction
        // is an area mean, everything else bilinear.
        D.rs_scale_x = 1.0 / ((double)virt.width / rd.w);
        D.rs_scale_y = 1.0 / ((double)virt.height / rd.h);
        const int ix = (int)std::lrint(D.rs_scale_x), iy = (int)std::lrint(D.rs_scale_y);
        D.rs_area = std::fabs(D.rs_scale_x - ix) < 2.220446049250313e-16 &&
                    std::fabs(D.rs_scale_y - iy) < 2.220446049250313e-16 && ix == 2 && iy == 2;
    }
    D.proj = virt.projection;
    D.wrap = (virt.projection == RVSB_PROJ_EQUIRECTANGULAR && virt.full_hor_range) ? 1 : 0;
    D.f0 = virt.focal[0];
    D.f1 = virt.focal[1];
    D.p0 = virt.principle_point[0];
    D.p1 = virt.principle_point[1];
    if (virt.projection == RVSB_PROJ_EQUIRECTANGULAR) erp_projector_constants(virt, D.u0, D.v0, D.du_dphi, D.dv_dtheta);
    // ERP input tiles wholly beyond a side of a perspective output are
    // skipped, except when the warped vertices themselves are asked for.
    if (virt.projection == RVSB_PROJ_PERSPECTIVE && p.precision == 1.f && !r.dbg.warped_uvz) {
        const float f0 = virt.focal[0], f1 = virt.focal[1], p0 = virt.principle_point[0], p1 = virt.principle_point[1];
        const float W = (float)virt.width, H = (float)virt.height;
        const float planes[4][3] = {{-(p0 + 1.f), f0, 0.f},      // u < -1
                                    {p0 - W - 1.f, -f0, 0.f},    // u > W + 1
                                    {-(p1 + 1.f), 0.f, f1},      // v < -1
                                    {p1 - H - 1.f, 0.f, -f1}};   // v > H + 1
        std::memcpy(D.cull_plane, planes, sizeof(planes));
        D.cull = 1;
    }
    D.bits = virt.bit_depth_color;
    D.max_val = (1u << virt.bit_depth_color) - 1u;
    D.blend_exp = p.blending_factor;
    D.inv_blend_exp = 1.0f / p.blending_factor;
    D.blend_exp_int = 0;
    if (p.blending_factor == std::floor(p.blending_factor) && p.blending_factor >= 2.f && p.blending_factor <= 16.f)
        D.blend_exp_int = (int)p.blending_factor;
    D.chroma_ties_up = p.chroma_rounding == RVSB_CHROMA_TIES_UP;
    D.blend_max = p.blending_factor < 0.f ? 1 : 0;
    auto exp_int = [](float e) {
        return (e == std::floor(e) && e >= 2.f && e <= 16.f) ? (int)e : 0;
    };
    if (p.blending_method == RVSB_BLEND_MULTISPECTRAL) {
        // The raster's own blend follows the low band: its quality, holes,
        // depth and validity are the multispectral blender's.
        D.blend_exp = p.low_freq_factor;
        D.inv_blend_exp = 1.0f / p.low_freq_factor;
        D.blend_exp_int = exp_int(p.low_freq_factor);
        D.blend_max = p.low_freq_factor < 0.f ? 1 : 0;
        MsPtrs& M = T.ms;
        M.yq = ws.ms_view.as<float2>();
        M.uv = M.yq + (size_t)n * npix;
        M.hsum = ws.ms_hsum.as<double>();
        M.hcnt = ws.ms_hcnt.as<int>();
        M.blur = ws.ms_blur.as<float>();
        M.on = 1;
        M.rad = std::max(rd.w, rd.h) / 20;
        M.low_exp = p.low_freq_factor;
        M.high_exp = p.high_freq_factor;
        M.low_int = exp_int(p.low_freq_factor);
        M.high_int = exp_int(p.high_freq_factor);
    }
    D.n_views = n;
    SlotBuffers& B = T.b;
    B.status = ws.status.as<DevStatus>();
    B.large = ws.large.as<uint4>();
    // The last of the list's memory holds the huge triangles, two words an entry.
    const int entries = (int)std::min<size_t>(INT32_MAX / 2, ws.large.bytes / sizeof(uint4));
    B.huge_capacity = std::min(8192, entries / 16) / 2 * 2;
    B.large_capacity = entries - B.huge_capacity / 2;
    B.codes = ws.codes.as<uint64_t>();
    B.holes = ws.holes.as<uint32_t>();
    for (int s = 0; s < 4; ++s) B.scan[s] = ws.scan.as<uint64_t>() + (size_t)s * npix;
    B.acc01 = reinterpret_cast<float2*>(B.scan[3]);
    B.acc23 = reinterpret_cast<float2*>(B.codes);
    B.inpaint_sum = ws.inpaint_sum.as<uint64_t>();
    if (rd.rescale) {
        B.pcolor = ws.pcolor.as<float4>();
        B.psrc = r.dbg.inpaint_source ? r.dbg.inpaint_source : ws.psrc.as<int32_t>();
    }
    T.out_y = r.out.y;
    T.out_u = r.out.u;
    T.out_v = r.out.v;
    T.dbg = r.dbg;
    if (r.aux) {
        AuxPtrs& A = T.aux;
        A.mask = r.aux->mask;
        A.masked_y = r.aux->masked.y;
        A.masked_u = r.aux->masked.u;
        A.masked_v = r.aux->masked.v;
        A.depth = r.aux->depth;
        A.masked_depth = r.aux->masked_depth;
        A.acc_depth = ws.aux_depth.as<float>();
        A.acc_valid = ws.aux_valid.as<float>();
        A.threshold = r.aux->validity_threshold;
        A.on = 1;
        A.depth_near = virt.depth_range[0];
        A.depth_far = virt.depth_range[1];
        A.depth_max = (1u << virt.bit_depth_depth) - 1u;
    }
}

BatchShape BatchCore::shape_of(const SlotRequest* reqs, int n, int variant) const {
    BatchShape sh;
    sh.slots = n;
    sh.variant = variant;
    bool persp = false, erp = false;
    for (int k = 0; k < n; ++k) {
        const SlotRequest& r = reqs[k];
        if (r.aux) sh.aux = 1;
        if (r.params.blending_method == RVSB_BLEND_MULTISPECTRAL) sh.ms = 1;
        if (r.params.precision != 1.f) sh.rescale = 1;
        const float e = r.params.blending_factor;
        if (!(e == std::floor(e) && e >= 2.f && e <= 16.f)) sh.int_pow = 0;
        if (r.virt.projection == RVSB_PROJ_EQUIRECTANGULAR) sh.erp_out = 1;
        if (r.aux || r.dbg.any() || r.params.blending_method == RVSB_BLEND_MULTISPECTRAL) sh.extras = 1;
        sh.max_views = std::max(sh.max_views, (int)r.scene->cams.size());
        for (const auto& c : r.scene->cams) {
            sh.max_w = std::max(sh.max_w, c.width);
            sh.max_h = std::max(sh.max_h, c.height);
            (c.projection == RVSB_PROJ_EQUIRECTANGULAR ? erp : persp) = true;
        }
        const RasterDims rd = raster_dims(r.virt, r.params);
        sh.max_wo = std::max(sh.max_wo, rd.w);
        sh.max_ho = std::max(sh.max_ho, rd.h);
        sh.max_out_w = std::max(sh.max_out_w, r.virt.width);
        sh.max_out_h = std::max(sh.max_out_h, r.virt.height);
    }
    sh.inputs = erp ? (persp ? 2 : 1) : 0;
    // The four words per pixel that the inpainting scans use later hold the
    // z-buffers of up to four views, or, for more views, of three at a time
    // and half of the running blend (its other half takes the codes').
    sh.vg = sh.max_views <= 4 ? 4 : 3;
    return sh;
}

int BatchCore::launch_variant(const SlotRequest* reqs, int n, int variant, cudaStream_t s,
                              const std::function<void()>& before_resolve) {
    const BatchShape sh = shape_of(reqs, n, variant);
    if (n == 1 && (!use_graphs_ || before_resolve)) {
        // A single synthesis: the table travels as a kernel parameter.
        TableParam tp;
        fill(tp.t, 0, reqs[0], sh);
        const int launches = launch_batch(tp, sh, s, profiling_ ? events_ : nullptr, before_resolve);
        if (launches < 0) check(cudaGetLastError(), "kernel launch");
        return launches;
    }
    // The staging buffer is reused every other call: its previous copy must
    // have been consumed.
    check(cudaEventSynchronize(copied_[cur_]), "wait for table staging");
    for (int k = 0; k < n; ++k) fill(staging_[cur_][k], k, reqs[k], sh);
    check(cudaMemcpyAsync(tables_.ptr, staging_[cur_], sizeof(SlotTable) * (size_t)n, cudaMemcpyHostToDevice, s),
          "upload slot tables");
    check(cudaEventRecord(copied_[cur_], s), "record table upload");
    cur_ ^= 1;
    const TablePtr tabs{tables_.as<SlotTable>()};
    if (use_graphs_ && !profiling_) {
        const std::vector<int> key = {sh.slots, sh.variant, sh.vg, sh.max_views, sh.max_w, sh.max_h, sh.max_wo,
                                      sh.max_ho, sh.aux, sh.ms, sh.extras, sh.erp_out, sh.int_pow, sh.inputs, sh.rescale, sh.max_out_w, sh.max_out_h};
        auto it = graphs_.find(key);
        if (it == graphs_.end()) {
            cudaGraph_t g = nullptr;
            check(cudaStreamBeginCapture(capture_, cudaStreamCaptureModeThreadLocal), "begin capture");
            const int nl = launch_batch(tabs, sh, capture_, nullptr);
            const cudaError_t ec = cudaStreamEndCapture(capture_, &g);
            if (nl < 0) check(cudaGetLastError(), "kernel launch (capture)");
            check(ec, "end capture");
            cudaGraphExec_t exec = nullptr;
            const cudaError_t ei = cudaGraphInstantiate(&exec, g, 0);
            cudaGraphDestroy(g);
            check(ei, "graph instantiate");
            it = graphs_.emplace(key, Graph{exec, nl}).first;
        }
        check(cudaGraphLaunch(it->second.exec, s), "graph launch");
        return it->second.launches;
    }
    const int launches = launch_batch(tabs, sh, s, profiling_ ? events_ : nullptr);
    if (launches < 0) check(cudaGetLastError(), "kernel launch");
    return launches;
}

namespace {

// Raster variant of a run that is neither pinned nor tuned.  At a magnification
// of m = 1 a triangle has one or two candidates, and the few above 4 go to the
// list of large triangles; past m of about 1.1 the threshold follows m
// (candidate_threshold), so that the ordinary triangles stay with their lanes:
// 2 x 960x540 into 1920x1080 (m = 2) 158 us against 249 with 4, 8 views of 4
// ERP 4096x2048 inputs (m = 1.47) 2.06 ms against 2.75, 4 x ERP 4096x2048 into
// the same 1.67 ms against 1.81.  At m <= 1 a threshold of 16 costs up to 6%
// (4 x 1920x1080 into 960x540 245 us against 232).  The unmagnified classes
// (one view, one minified to m <= 0.6, a batch of 8 or more) share their
// parameters; the rows per warp follow the launch's size (mesh.cu).
constexpr int kMagnifiedVariant = 7;
constexpr int kDefaultVariant = 4;
constexpr int kMinifiedVariant = 2;
constexpr int kBatchVariant = 1;
constexpr int kBatchVariantMinSlots = 8;

int default_variant(const SlotRequest* reqs, int n) {
    float m = 0.f;
    bool erp_out = false;
    for (int k = 0; k < n; ++k) {
        m = std::max(m, magnification(reqs[k]));
        if (reqs[k].virt.projection == RVSB_PROJ_EQUIRECTANGULAR) erp_out = true;
    }
    if (m > kMagnified) return kMagnifiedVariant;
    if (!erp_out && m <= 0.6f) return kMinifiedVariant;
    return n >= kBatchVariantMinSlots ? kBatchVariant : kDefaultVariant;
}

}  // namespace

int BatchCore::tune(const SlotRequest* reqs, int n, cudaStream_t s) {
    const bool graphs = use_graphs_, prof = profiling_;
    use_graphs_ = false;
    profiling_ = false;
    // A warm-up run of every variant (first use of its module), then five
    // rounds that time each variant once, in turn, so that a drift of the
    // device's state affects them alike; the variant with the smallest median
    // wins if it beats the untuned default's median by at least 2%, else the
    // default stays.  One run alone is too noisy to rank variants a few
    // percent apart, and among variants within the noise of each other the
    // pick would otherwise be arbitrary (measured: a 1.7% slower one picked
    // for the plain 1080p view).
    // Variants whose launch is that of an earlier one (same rows, and the same
    // threshold in every slot) take its time.
    constexpr int kRounds = 5;
    bool magnified = false;
    for (int k = 0; k < n; ++k) magnified = magnified || candidate_threshold(reqs[k]) != 4;
    int same[NUM_RASTER_VARIANTS];
    std::vector<int> timed;
    for (int v = 0; v < NUM_RASTER_VARIANTS; ++v) {
        auto small_of = [&](int w) {
            const int small = kRasterVariants[w].small;
            return small == 0 && !magnified ? 4 : small;
        };
        same[v] = v;
        for (int u : timed)
            if (kRasterVariants[u].rows == kRasterVariants[v].rows && small_of(u) == small_of(v)) same[v] = u;
        if (same[v] == v) timed.push_back(v);
    }
    for (int v : timed) launch_variant(reqs, n, v, s);
    float t[NUM_RASTER_VARIANTS][kRounds];
    for (int r = 0; r < kRounds; ++r)
        for (int v : timed) {
            check(cudaEventRecord(tune_ev_[0], s), "record");
            launch_variant(reqs, n, v, s);
            check(cudaEventRecord(tune_ev_[1], s), "record");
            check(cudaEventSynchronize(tune_ev_[1]), "synchronize");
            check(cudaEventElapsedTime(&t[v][r], tune_ev_[0], tune_ev_[1]), "elapsed");
        }
    int best = 0;
    float best_ms = 0.f, med[NUM_RASTER_VARIANTS];
    for (int v : timed) {
        std::sort(t[v], t[v] + kRounds);
        med[v] = t[v][kRounds / 2];
        if (v == 0 || med[v] < best_ms) {
            best = v;
            best_ms = med[v];
        }
    }
    const int fallback = default_variant(reqs, n);
    if (best_ms > 0.98f * med[same[fallback]]) best = fallback;
    use_graphs_ = graphs;
    profiling_ = prof;
    return best;
}

int BatchCore::run(const SlotRequest* reqs, int n, cudaStream_t s, const std::function<void()>& before_resolve) {
    HostRange range("rvsb: batch (tables, launches)");
    if (n <= 0 || n > slots_) throw ArgError("batch of " + std::to_string(n) + " requests for " +
                                             std::to_string(slots_) + " slots");
    int ms_wo = 0;
    for (int k = 0; k < n; ++k) {
        const SlotRequest& r = reqs[k];
        const RasterDims rd = raster_dims(r.virt, r.params);
        if (rd.rescale && r.aux && r.aux->masked.y)
            throw Unsupported("MaskedOutputFiles needs Precision 1: the reference masks the raster-sized colour "
                              "with the mask resized to the output size (Pipeline.cpp:314-318), which OpenCV "
                              "rejects");
        ws_[k]->ensure(ctx_, r.scene, rd.w, rd.h);
        if (r.aux) ws_[k]->ensure_aux(ctx_, rd.w, rd.h);
        if (rd.rescale) ws_[k]->ensure_rescale(ctx_, rd.w, rd.h);
        if (r.params.blending_method == RVSB_BLEND_MULTISPECTRAL) {
            ws_[k]->ensure_ms(ctx_, (int)r.scene->cams.size(), rd.w, rd.h);
            ms_wo = std::max(ms_wo, rd.w);
        }
    }
    if (ms_wo > 0) prepare_ms_kernels(ms_wo);
    int variant = default_variant(reqs, n);
    if (forced_variant_ >= 0) {
        variant = forced_variant_;
    } else if (autotune_) {
        // The shape the tuner keys on: the batch size bucket and, over the
        // batch, the largest input set and output, the projections and the
        // magnified thresholds (a fixed threshold that suits unmagnified
        // triangles lists nearly every magnified one; 1: magnified, and all
        // listed).
        const BatchShape sh = shape_of(reqs, n, 0);
        int proj_in = 0, proj_out = 0, small_lo = INT_MAX, small_hi = 0;
        for (int k = 0; k < n; ++k) {
            proj_in |= 1 << reqs[k].scene->cams[0].projection;
            proj_out |= 1 << reqs[k].virt.projection;
            const int t = candidate_threshold(reqs[k]);
            const int small = t == 4 && magnification(reqs[k]) > kMagnified ? 1 : t;
            small_lo = std::min(small_lo, small);
            small_hi = std::max(small_hi, small);
        }
        const int bucket = n == 1 ? 1 : n <= 4 ? 4 : n <= 16 ? 16 : 64;
        const std::vector<int> sig = {bucket, sh.max_views, sh.max_w, sh.max_h, sh.max_wo, sh.max_ho,
                                      proj_in, proj_out, sh.max_out_w, sh.max_out_h, small_lo, small_hi};
        auto it = tuned_.find(sig);
        if (it == tuned_.end()) it = tuned_.emplace(sig, tune(reqs, n, s)).first;
        variant = it->second;
    }
    const int launches = launch_variant(reqs, n, variant, s, before_resolve);
    profiled_ = profiling_;
    last_launches_ = launches;
    last_variant_ = variant;
    return launches;
}

}  // namespace rvsb
