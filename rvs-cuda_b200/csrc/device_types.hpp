// Parameter blocks shared by the host launch code and the kernels.
#pragma once

#include <cstdint>

namespace rvsb {

// Vertex tile of the ERP input culling tables (WARP_TILE x WARP_TILE input
// pixels).
constexpr int WARP_TILE = 32;

// Per input view parameters of one synthesis (device copy in a table).
struct DevView {
    int w, h;          // input size
    int proj;          // 0 perspective, 1 equirectangular
    int bits_color;
    float f0, f1, p0, p1;                 // perspective intrinsics
    float near_, far_, depth_scale;       // depth decode (process_input_frame.cu:369-376)
    int has_invalid;
    float color_scale;                    // 1 / (2^bits - 1)
    float chroma_sx, chroma_sy;           // (w/2)/w, (h/2)/h as float
    int cw, ch;                           // chroma plane size
    float R[9], t[3];                     // relative pose (SpaceTransformer.cpp:77-92)
    const uint16_t* py;
    const uint16_t* pu;
    const uint16_t* pv;
    const uint16_t* pd;
    const float4* depth_lut;              // 65536 (d, -d/f0, -d/f1, 0), indexed by the raw sample
    const float* erp_row;                 // ERP: per row (cos theta, sin theta), 2*h floats
    const float* erp_col;                 // ERP: per column (cos phi, sin phi), 2*w floats
    // ERP inputs, per WARP_TILE x WARP_TILE vertex tile grown by one pixel:
    // the unit direction of its centre and an angle bounding every vertex
    // direction from it (x, y, z, radius), and the range of its decoded
    // depths (min, max); used to skip tiles no output pixel can come from.
    const float4* erp_cone;
    const float2* tile_depth;
    const uint64_t* color;                // h*w decoded colour: Y | 4U << 18 | 4V << 36
    float4* vert;                         // h*w warped vertices (u, v, z, 0)
    unsigned long long* z;                // wo*ho fragment keys (shared by the views of one group each)
    int tri_shift;                        // triangle index = i << tri_shift | j << 2 | t
    int pad;
};

// Virtual camera of one synthesis.
struct DevTarget {
    int wo, ho;
    int proj;
    int wrap;                             // horizontal wrap (ERP output, full range)
    // Perspective output: the planes u = -1, u = W + 1, v = -1, v = H + 1 in
    // the virtual camera's frame (a . y > 0 beyond each, for y0 > 0); cull
    // enables skipping ERP input tiles wholly beyond one of them.
    int cull;
    float cull_plane[4][3];
    float f0, f1, p0, p1;                 // perspective
    float u0, v0, du_dphi, dv_dtheta;     // equirectangular
    int bits;                             // output bit depth
    unsigned max_val;                     // 2^bits - 1
    float blend_exp;                      // BlendingFactor
    float inv_blend_exp;                  // 1.0f / BlendingFactor
    int blend_exp_int;                    // BlendingFactor when it is an integer in [2, 16], else 0
    int chroma_ties_up;                   // output chroma mean: 1 rounds ties up, 0 to even
    int blend_max;                        // BlendingFactor < 0: blend by maximum quality
    // Precision P != 1 (SynthesizedView.cpp:325-333): wo x ho is the raster
    // size int(0.5 + W * P) x int(0.5 + H * P); the output W x H is resized
    // from it (image_writing.cpp:188-190).
    int rescale;
    int out_w, out_h;
    float uv_sx, uv_sy;                   // raster size / output size (float)
    float precision;
    int small;                            // candidate pixels above which a triangle is a large one
    int rs_area;                          // the resize is an exact 2x reduction (area mean)
    double rs_scale_x, rs_scale_y;        // raster size / output size (double), bilinear
    int n_views;
};

// Largest number of input views of one synthesis.
constexpr int MAX_VIEWS = 16;

// Status words written by the kernels (device memory, reset per call).
struct DevStatus {
    int n_large;        // large triangles entered in the list (may exceed its capacity)
    int n_holes;        // nonzero when some pixel is a hole
    int n_claimed;      // groups of quads claimed by the pass over the whole mesh
    int n_huge;         // huge triangles that are shared out (may exceed their words)
};

// Optional intermediate outputs (device pointers, may be null).
struct DebugPtrs {
    float* warped_uvz = nullptr;
    float* view_color = nullptr;
    float* view_depth = nullptr;
    float* view_validity = nullptr;
    float* blend_color = nullptr;
    float* blend_quality = nullptr;
    int32_t* inpaint_source = nullptr;
    bool any() const {
        return warped_uvz || view_color || view_depth || view_validity || blend_color ||
               blend_quality || inpaint_source;
    }
};

// Auxiliary outputs of a synthesis (Pipeline.cpp:303-336, CPU mode): any
// pointer may be null.  acc_depth / acc_valid are the slot's per-pixel
// blended depth and validity (workspace buffers, set when any output is on).
struct AuxPtrs {
    uint8_t* mask;            // 255 where the blended validity is not above threshold
    uint16_t* masked_y;       // YUV420 colour with masked pixels set to 0.5
    uint16_t* masked_u;
    uint16_t* masked_v;
    uint16_t* depth;          // encoded blended depth
    uint16_t* masked_depth;   // the same, 0 where masked
    float* acc_depth;
    float* acc_valid;
    float threshold;          // "ValidityThreshold"
    int on;                   // any output requested
    float depth_near, depth_far;  // virtual camera's depth range
    unsigned depth_max;       // 2^BitDepthDepth - 1
    int pad;
};

// Multispectral blending (BlendedViewMultiSpec, BlendedView.cpp:63-88): the
// raster stores every view's resolved colour and quality, the blur kernels
// the masked box mean of each view's luma, and the blend kernel the two
// frequency bands' blends.  Per view, npix = Wo*Ho entries each.
struct MsPtrs {
    float2* yq;         // (Y, quality) per view and pixel: all the blur reads
    float2* uv;         // (U, V) per view and pixel
    double* hsum;       // row-window sums of masked luma
    int* hcnt;          // row-window counts of masked pixels
    float* blur;        // blurred luma (0 outside the mask)
    int on;
    int rad;            // window radius: max(Wo, Ho) / 20
    float low_exp, high_exp;
    int low_int, high_int;  // integer exponents in [2, 16] (0 otherwise)
};

// Device buffers of one slot's workspace.
struct SlotBuffers {
    DevStatus* status;   // 1 entry
    uint4* large;        // large triangles of the view group, `large_capacity` entries
    int large_capacity;
    int huge_capacity;   // words after the list, one per huge triangle that is shared out
    // Running blend between view groups: (c0, c1) and (c2, weight sum) per
    // pixel; they share the memory of the last scan buffer and the codes,
    // which are written later.
    float2* acc01;
    float2* acc23;
    uint64_t* codes;     // Wo*Ho packed output codes + hole bit
    uint32_t* holes;     // hole mask, one bit per pixel (1 = no view covers it), (Wo + 31) / 32 words a row
    uint64_t* scan[4];   // Wo*Ho inpainting scratch each
    uint64_t* inpaint_sum;  // column minima of the inpainting's row groups
    float4* pcolor;      // Precision != 1: blended colour per raster pixel
    int32_t* psrc;       // Precision != 1: inpainting source of every hole
};

// Everything one synthesis (one virtual view) needs on the device.  A batch
// keeps one table per slot in device memory; every kernel of the batch reads
// the table of its slot (a grid dimension), so the launch sequence of a
// batch is fixed and the per-call data travels in one copy of the tables.
struct SlotTable {
    DevTarget t;
    SlotBuffers b;
    uint16_t* out_y;
    uint16_t* out_u;
    uint16_t* out_v;
    DebugPtrs dbg;
    AuxPtrs aux;
    MsPtrs ms;
    DevView v[MAX_VIEWS];
};

}  // namespace rvsb
