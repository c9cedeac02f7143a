// Tables of the input views: the decoded depth of every raw sample, and the
// depth range of every vertex tile of an equirectangular view.
#include "device_common.cuh"
#include "kernels.hpp"

namespace rvsb {
namespace {

using namespace dev;

// Range of the decoded depths of one vertex tile grown by one pixel (NaN
// samples ignored).  Grid (tiles x, tiles y, views), 256 threads.
__global__ void tile_depth_kernel(const __grid_constant__ TileDepthJobs jobs) {
    const TileDepthJob& J = jobs.v[blockIdx.z];
    const int ntx = (J.w + WARP_TILE - 1) / WARP_TILE, nty = (J.h + WARP_TILE - 1) / WARP_TILE;
    if ((int)blockIdx.x >= ntx || (int)blockIdx.y >= nty) return;
    const int r0 = max(0, (int)blockIdx.y * WARP_TILE - 1), r1 = min(J.h - 1, (int)blockIdx.y * WARP_TILE + WARP_TILE);
    const int c0 = max(0, (int)blockIdx.x * WARP_TILE - 1), c1 = min(J.w - 1, (int)blockIdx.x * WARP_TILE + WARP_TILE);
    const int cols = c1 - c0 + 1, n = (r1 - r0 + 1) * cols;
    float mn = INFINITY, mx = -INFINITY;
    for (int k = threadIdx.x; k < n; k += blockDim.x) {
        const int i = r0 + k / cols, j = c0 + k % cols;
        const float z = __ldg(&J.lut[__ldg(J.depth + (size_t)i * J.w + j)].x);
        mn = fminf(mn, z);
        mx = fmaxf(mx, z);
    }
    __shared__ float s_mn[8], s_mx[8];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        mn = fminf(mn, __shfl_xor_sync(0xffffffffu, mn, o));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0) {
        s_mn[warp] = mn;
        s_mx[warp] = mx;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int k = 1; k < (int)(blockDim.x >> 5); ++k) {
            mn = fminf(mn, s_mn[k]);
            mx = fmaxf(mx, s_mx[k]);
        }
        J.out[blockIdx.y * ntx + blockIdx.x] = make_float2(mn, mx);
    }
}

// Decoded depth d of every possible 16-bit sample of one view, with the
// two per-sample factors of the perspective unprojection, -(d / f0) and
// -(d / f1) (PerspectiveUnprojector.cpp:75-77), so that the warp reads them
// instead of dividing per pixel.
__global__ void depth_lut_kernel(float near_, float far_, float depth_scale, int has_invalid, float f0, float f1,
                                 float4* out) {
    const uint32_t raw = blockIdx.x * blockDim.x + threadIdx.x;
    if (raw >= 65536u) return;
    const float d = decode_depth_raw(near_, far_, depth_scale, has_invalid, raw);
    out[raw] = make_float4(d, -__fdiv_rn(d, f0), -__fdiv_rn(d, f1), 0.f);
}

}  // namespace

void launch_tile_depth(const TileDepthJobs& jobs, int n, int max_w, int max_h, cudaStream_t s) {
    tile_depth_kernel<<<dim3((max_w + WARP_TILE - 1) / WARP_TILE, (max_h + WARP_TILE - 1) / WARP_TILE, n), 256, 0, s>>>(
        jobs);
}

void launch_depth_lut(float near_, float far_, float depth_scale, int has_invalid, float f0, float f1, float4* out,
                      cudaStream_t s) {
    depth_lut_kernel<<<256, 256, 0, s>>>(near_, far_, depth_scale, has_invalid, f0, f1, out);
}

}  // namespace rvsb
