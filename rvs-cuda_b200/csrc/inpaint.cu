// Inpainting stage: compute_nearest (rvs/src/inpainting.cpp:104-136) as two
// sweeps of min-plus scans over the holes, then the fill of inpaint_color
// (inpainting.cpp:191-198) and the write of the 2x2 output blocks that held
// holes.
//
// Why two sweeps of scans are exact: the reference alternates column-major
// Gauss-Seidel sweeps (forward, then reverse) until one changes nothing.
// After the forward sweep 0 and the reverse sweep 1 every distance equals
// the L1 distance transform, so sweep 2 never changes anything and the
// result is the state after sweep 1.  Each sweep is a min-plus recurrence
// over left/up (or right/down) neighbours with a fixed neighbour priority:
//  sweep 0: (D0, S0)(p) = lexmin over q with q.x <= p.x, q.y <= p.y of
//           (C(q).d + |p - q|, C(q).source), C(q) = (0, q) for a non-hole,
//           (1, down(q)) or else (1, right(q)) for a hole whose down/right
//           neighbour is a non-hole;
//  sweep 1: seeds T(q) = best of stay (D0, S0), left (D0 + 1, S0 of left),
//           up (D0 + 1, S0 of up), in that priority (T'(q) without stay);
//           a hole p takes the best seed of its lower-right quadrant, from
//           its own column (smallest y) when the column holds a minimum,
//           otherwise the minimum with the largest y, then smallest x, and
//           changes only on strict improvement.
//
// Only holes cost memory traffic.  The hole mask is one bit per pixel (32
// columns, a strip, per word), and what a scan would hold at a non-hole
// follows from the mask: distance 0, itself.  A hole's row term is the
// nearest event to its left -- a non-hole, or a hole with C = 1 -- so it
// comes from the mask words and one prefix per (row, word), not from a scan
// of the row; a non-hole ends every column and row recurrence, being better
// than all that lies behind it.  So the 8-byte words of a sweep are written
// and read at holes alone, and strips without holes cost one mask word per
// row.  Columns are split into groups of rows; a group starts from the
// minimum of the groups' minima before it.  The stage is a chain of five
// short kernels, bound by their latency at one image: against scans over
// every pixel of the holes' bounding box (seven kernels, about 100 bytes a
// pixel) a 1920x1080 view with holes along its borders takes 37 us instead of
// 79, a 960x540 one 26 instead of 38, an equirectangular 4096x2048 one 52
// instead of 214, and a batch of 8 1920x1080 views 21 us a view instead of 60.
#include <algorithm>

#include "device_common.cuh"
#include "kernels.hpp"

namespace rvsb {
namespace {

using namespace dev;

constexpr int kScanBias = 1 << 20;
// A hole's sweep-1 choice stored in its D0/S0 word by the last column
// scan: with this bit, (x << 16 | y) of the seed T(q) whose source it
// takes; without, its source itself (x << 16 | y in the low 32 bits).
constexpr uint64_t kSeedRef = 1ull << 63;

// The buffers of one image the passes work on.
struct InpaintImage {
    int wo, ho;
    int words;                 // mask words per row
    const DevStatus* st;       // whether there are holes
    const uint32_t* holes;     // hole bits; bits beyond the width are set
    uint64_t* codes;           // wo*ho packed codes (null: only sources are wanted)
    // Words per pixel, at holes only: RR, (D0, S0), T and T'.
    uint64_t* rr;
    uint64_t* ds;
    uint64_t* tq;
    uint64_t* tp;
    uint64_t* before;          // per (row, word): the row's best event before the word (in rr's memory)
    uint64_t* sum;             // 3 * groups * wo: minima of the row groups, per column
    int32_t* sources;          // optional: (x, y) source of every hole
    uint16_t* out_y;
    uint16_t* out_u;
    uint16_t* out_v;
    int ties_up;               // output chroma rounding
    int no_write;              // Precision != 1: the resize writes the output
};

// Image of slot blockIdx.z of a batch.
template <class Tabs>
struct FromTables {
    Tabs tabs;
    __device__ InpaintImage operator()() const {
        const SlotTable& t = tabs.at(blockIdx.z);
        InpaintImage im;
        im.wo = t.t.wo;
        im.ho = t.t.ho;
        im.words = (t.t.wo + 31) / 32;
        im.st = t.b.status;
        im.holes = t.b.holes;
        im.codes = t.b.codes;
        im.rr = im.before = t.b.scan[0];
        im.ds = t.b.scan[1];
        im.tq = t.b.scan[2];
        im.tp = t.b.scan[3];
        im.sum = t.b.inpaint_sum;
        im.sources = t.t.rescale ? t.b.psrc : t.dbg.inpaint_source;
        im.no_write = t.t.rescale;
        im.out_y = t.out_y;
        im.out_u = t.out_u;
        im.out_v = t.out_v;
        im.ties_up = t.t.chroma_ties_up;
        return im;
    }
};

// One image given directly (kernel parameter).
struct Direct {
    InpaintImage im;
    __device__ InpaintImage operator()() const { return im; }
};

// Row groups of the column passes.  A CTA takes one group of one strip, a
// warp 4 rows of it, so that no thread's serial chain is longer than that
// (one warp over 32 rows took five times as long: 24 us instead of 5 for the
// forward columns of a 1920x1080 view).
constexpr int GROUP = 32;
constexpr int COL_WARPS = 8;
constexpr int WROWS = GROUP / COL_WARPS;
__host__ __device__ __forceinline__ int group_count(int ho) { return (ho + GROUP - 1) / GROUP; }

__device__ __forceinline__ uint64_t pack_dxy(uint32_t d, int x, int y) {
    return ((uint64_t)d << 32) | ((uint64_t)(uint32_t)x << 16) | (uint64_t)(uint32_t)y;
}

__device__ __forceinline__ unsigned long long umin64(unsigned long long a, unsigned long long b) {
    return b < a ? b : a;
}

// The mask words a row of 32 columns needs: its own, the one to its right
// and the one below (set bits where there is no neighbour).
struct MaskWords {
    uint32_t own, right, below;
};
__device__ __forceinline__ MaskWords mask_words(const InpaintImage& im, int y, int w) {
    const uint32_t* p = im.holes + (size_t)y * im.words + w;
    MaskWords m;
    m.own = __ldg(p);
    m.right = w + 1 < im.words ? __ldg(p + 1) : 0xffffffffu;
    m.below = y + 1 < im.ho ? __ldg(p + im.words) : 0xffffffffu;
    return m;
}

// Columns of word w inside the image.
__device__ __forceinline__ uint32_t word_columns(const InpaintImage& im, int w) {
    return w + 1 < im.words || !(im.wo & 31) ? 0xffffffffu : (1u << (im.wo & 31)) - 1u;
}

// Events of a word: non-holes, and holes whose right or lower neighbour is
// a non-hole (C = 1).
__device__ __forceinline__ uint32_t events(const MaskWords& m) {
    return ~m.own | ~m.below | ~((m.own >> 1) | (m.right << 31));
}

// Row key (C(q).d - q.x, source) of the last event in `ev`, a nonempty part
// of the word's events up to some column; smaller keys are better for every
// pixel to the right.  A hole next to a non-hole on its left gives the same
// distance as that non-hole, whose column is smaller, and the earlier
// events give larger ones.
__device__ __forceinline__ unsigned long long event_key(const MaskWords& m, uint32_t ev, int x0, int y) {
    int e = 31 - __clz(ev);
    if ((m.own >> e & 1u) && e > 0 && !(m.own >> (e - 1) & 1u)) --e;
    const int x = x0 + e;
    if (!(m.own >> e & 1u)) return pack_dxy((uint32_t)(kScanBias - x), x, y);
    if (!(m.below >> e & 1u)) return pack_dxy((uint32_t)(kScanBias + 1 - x), x, y + 1);
    return pack_dxy((uint32_t)(kScanBias + 1 - x), x + 1, y);
}

// Column key (R(p).d - y, source) of pixel (x0 + lane, y), R from the row's
// events; empty when there is none to its left.
__device__ __forceinline__ unsigned long long column_key(const MaskWords& m, unsigned long long before, int x0, int y,
                                                         int lane) {
    unsigned long long k = before;
    const uint32_t ev = events(m) & (0xffffffffu >> (31 - lane));
    if (ev) k = umin64(k, event_key(m, ev, x0, y));
    if (k == kEmptyKey) return k;
    return k + ((unsigned long long)(uint32_t)(x0 + lane - y) << 32);
}

__device__ __forceinline__ unsigned long long non_hole_key(int x, int y) {
    return pack_dxy((uint32_t)(kScanBias - y), x, y);
}

// Sweep 0, rows: the best event of the row before every word.  Grid
// (ceil(max_ho / 8), 1, images), one warp per row.
template <class Src>
__global__ void __launch_bounds__(256) inpaint_rows0_kernel(const __grid_constant__ Src src) {
    grid_dep_wait();
    const InpaintImage im = src();
    if (im.st->n_holes == 0) return;
    const int lane = threadIdx.x & 31, y = blockIdx.x * 8 + (threadIdx.x >> 5);
    if (y >= im.ho) return;
    unsigned long long carry = kEmptyKey;
    for (int w0 = 0; w0 < im.words; w0 += 32) {
        const int w = w0 + lane;
        unsigned long long k = kEmptyKey;
        if (w < im.words) {
            const MaskWords m = mask_words(im, y, w);
            const uint32_t ev = events(m);
            if (ev) k = event_key(m, ev, w * 32, y);
        }
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned long long v = __shfl_up_sync(0xffffffffu, k, o);
            if (lane >= o) k = umin64(k, v);
        }
        unsigned long long ex = __shfl_up_sync(0xffffffffu, k, 1);
        if (lane == 0) ex = kEmptyKey;
        if (w < im.words) im.before[(size_t)y * im.words + w] = umin64(ex, carry);
        carry = umin64(carry, __shfl_sync(0xffffffffu, k, 31));
    }
}

// Sweep 0, columns (forward): D0, S0 (p) = lexmin over q.y <= p.y of
// (R(q).d + p.y - q.y, src), at the holes.  Grid (strips, groups, images),
// 256 threads.  PRE: only the group's column minima are stored (and those of
// sweep 1 that its non-holes give); otherwise the group is scanned from the
// minima of the groups above it.
template <class Src, bool PRE>
__global__ void __launch_bounds__(32 * COL_WARPS) inpaint_cols0_kernel(const __grid_constant__ Src src) {
    grid_dep_wait();
    const InpaintImage im = src();
    if (PRE && im.st->n_holes == 0) return;
    __shared__ unsigned long long s_total[COL_WARPS][32], s_carry[COL_WARPS][32];
    const int G = group_count(im.ho), g = blockIdx.y, w = blockIdx.x;
    if (g >= G || w >= im.words) return;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int x = w * 32 + lane, y0 = g * GROUP + warp * WROWS;
    const uint32_t cols = word_columns(im, w);
    const bool in = cols >> lane & 1u;
    uint32_t holes = 0;
#pragma unroll
    for (int r = 0; r < WROWS; ++r)
        if (y0 + r < im.ho) holes |= __ldg(im.holes + (size_t)(y0 + r) * im.words + w) & cols;
    if (!__syncthreads_or(holes != 0u)) {
        if (PRE && warp == 0 && in) {
            const int yl = min(im.ho, g * GROUP + GROUP) - 1, yf = g * GROUP;
            im.sum[(size_t)g * im.wo + x] = non_hole_key(x, yl);
            im.sum[(size_t)(G + g) * im.wo + x] = ((unsigned long long)yf << 16) | (unsigned long long)yf;
            im.sum[(size_t)(2 * G + g) * im.wo + x] = kEmptyKey;
        }
        return;
    }
    MaskWords m[WROWS];
    unsigned long long key[WROWS], total = kEmptyKey, first = kEmptyKey;
#pragma unroll
    for (int r = 0; r < WROWS; ++r) {
        const int y = y0 + r;
        m[r] = MaskWords{0u, 0u, 0u};
        key[r] = kEmptyKey;
        if (y >= im.ho) continue;
        m[r] = mask_words(im, y, w);
        if (m[r].own >> lane & 1u) {
            if (in) key[r] = column_key(m[r], im.before[(size_t)y * im.words + w], w * 32, y, lane);
        } else {
            key[r] = non_hole_key(x, y);
            first = umin64(first, ((unsigned long long)y << 16) | (unsigned long long)y);
        }
        total = umin64(total, key[r]);
    }
    s_total[warp][lane] = total;
    if (PRE) {
        s_carry[warp][lane] = first;
        __syncthreads();
        if (warp > 1 || !in) return;
        unsigned long long t = kEmptyKey;
#pragma unroll
        for (int k = 0; k < COL_WARPS; ++k) t = umin64(t, warp == 0 ? s_total[k][lane] : s_carry[k][lane]);
        im.sum[(size_t)(warp * G + g) * im.wo + x] = t;
        if (warp == 1) im.sum[(size_t)(2 * G + g) * im.wo + x] = kEmptyKey;
        return;
    }
    // What lies above matters only to holes that reach the group's first
    // row; a non-hole there beats it.
    unsigned long long run = kEmptyKey;
    if (in && (__ldg(im.holes + (size_t)g * GROUP * im.words + w) >> lane & 1u))
        for (int h = warp; h < g; h += COL_WARPS) run = umin64(run, im.sum[(size_t)h * im.wo + x]);
    s_carry[warp][lane] = run;
    __syncthreads();
    if (!holes) return;
#pragma unroll
    for (int k = 0; k < COL_WARPS; ++k) {
        run = umin64(run, s_carry[k][lane]);
        if (k < warp) run = umin64(run, s_total[k][lane]);
    }
#pragma unroll
    for (int r = 0; r < WROWS; ++r) {
        const int y = y0 + r;
        run = umin64(run, key[r]);
        if (in && (m[r].own >> lane & 1u))
            im.ds[(size_t)y * im.wo + x] = run == kEmptyKey
                                               ? pack_dxy((uint32_t)(im.wo + im.ho), x, y)
                                               : run + ((unsigned long long)(uint32_t)(y - kScanBias) << 32);
    }
}

constexpr int ROW_WARPS = 8;
constexpr int MAX_WORDS = 32768 / 32;

// Sweep 1, seeds and rows (backward, exclusive), at the holes:
// T(q) = best of stay (D0(q), S0(q)), left (D0 + 1, S0 of left), up (D0 + 1,
// S0 of up) with priority stay > left > up; T'(q) the same without stay.
// RR(x, y) = min over q.x > x of (T(q).d + q.x, q.x).  One CTA per row; its
// warps take the words that hold holes, and the words' minima meet in shared
// memory.  Both terms of a hole's column scan
// go into its group's minima as well.  Grid (max_ho, 1, images).
template <class Src>
__global__ void __launch_bounds__(32 * ROW_WARPS) inpaint_rows1_kernel(const __grid_constant__ Src src) {
    grid_dep_wait();
    const InpaintImage im = src();
    const int y = blockIdx.x;
    if (y >= im.ho) return;
    __shared__ unsigned long long s_min[MAX_WORDS + 1];
    __shared__ uint32_t s_own[MAX_WORDS + 1], s_up[MAX_WORDS];  // s_own[0]: left of the row
    __shared__ uint16_t s_list[MAX_WORDS];
    __shared__ int s_n;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, tid = threadIdx.x;
    if (tid == 0) {
        s_n = 0;
        s_own[0] = 0u;
        s_min[im.words] = kEmptyKey;
    }
    __syncthreads();
    for (int w = tid; w < im.words; w += 32 * ROW_WARPS) {
        const uint32_t own = __ldg(im.holes + (size_t)y * im.words + w);
        s_own[w + 1] = own;
        s_up[w] = y > 0 ? __ldg(im.holes + (size_t)(y - 1) * im.words + w) : 0u;
        // Without holes the word's first pixel is its minimum.
        s_min[w] = ((unsigned long long)(w * 32) << 16) | (unsigned long long)(w * 32);
        if (own & word_columns(im, w)) s_list[atomicAdd(&s_n, 1)] = (uint16_t)w;
    }
    __syncthreads();
    const int n = s_n;
    if (n == 0) return;
    for (int k = warp; k < n; k += ROW_WARPS) {
        const int w = s_list[k], x = w * 32 + lane;
        const uint32_t own = s_own[w + 1];
        unsigned long long key = kEmptyKey;
        if (x < im.wo) {
            uint32_t d = 0;
            if (own >> lane & 1u) {
                const size_t o = (size_t)y * im.wo + x;
                uint64_t best = im.ds[o];
                // (D0, S0) of a non-hole: 0, itself.
                uint64_t left = pack_dxy(0, x - 1, y), up = pack_dxy(0, x, y - 1);
                if ((lane ? own >> (lane - 1) : s_own[w] >> 31) & 1u) left = im.ds[o - 1];
                if (s_up[w] >> lane & 1u) up = im.ds[o - im.wo];
                uint64_t bp = ~0ull;
                if (x > 0) {
                    const uint64_t c = left + (1ull << 32);
                    if ((c >> 32) < (best >> 32)) best = c;
                    bp = c;
                }
                if (y > 0) {
                    const uint64_t c = up + (1ull << 32);
                    if ((c >> 32) < (best >> 32)) best = c;
                    if (bp == ~0ull || (c >> 32) < (bp >> 32)) bp = c;
                }
                im.tq[o] = best;
                im.tp[o] = bp;
                d = (uint32_t)(best >> 32);
            }
            key = ((unsigned long long)(d + (uint32_t)x) << 16) | (unsigned long long)x;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) key = umin64(key, __shfl_xor_sync(0xffffffffu, key, o));
        if (lane == 0) s_min[w] = key;
    }
    __syncthreads();
    // Suffix minima over the words, by warp 0 in runs of consecutive words.
    if (warp == 0) {
        const int per = (im.words + 31) / 32, b = min(im.words, lane * per), e = min(im.words, b + per);
        unsigned long long m = kEmptyKey;
        for (int w = e - 1; w >= b; --w) s_min[w] = m = umin64(m, s_min[w]);
        unsigned long long suf = m;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned long long v = __shfl_down_sync(0xffffffffu, suf, o);
            if (lane + o < 32) suf = umin64(suf, v);
        }
        const unsigned long long after = __shfl_down_sync(0xffffffffu, suf, 1);
        if (lane < 31)
            for (int w = b; w < e; ++w) s_min[w] = umin64(s_min[w], after);
    }
    __syncthreads();
    const int G = group_count(im.ho), g = y / GROUP;
    unsigned long long* sum = reinterpret_cast<unsigned long long*>(im.sum);
    for (int k = warp; k < n; k += ROW_WARPS) {
        const int w = s_list[k], x = w * 32 + lane;
        const bool in = x < im.wo, hole = in && (s_own[w + 1] >> lane & 1u);
        const size_t o = (size_t)y * im.wo + x;
        const uint32_t d = hole ? (uint32_t)(im.tq[o] >> 32) : 0u;
        unsigned long long key = in ? ((unsigned long long)(d + (uint32_t)x) << 16) | (unsigned long long)x : kEmptyKey;
#pragma unroll
        for (int s = 1; s < 32; s <<= 1) {
            const unsigned long long v = __shfl_down_sync(0xffffffffu, key, s);
            if (lane + s < 32) key = umin64(key, v);
        }
        unsigned long long ex = __shfl_down_sync(0xffffffffu, key, 1);
        if (lane == 31) ex = kEmptyKey;
        ex = umin64(ex, s_min[w + 1]);
        if (!hole) continue;
        im.rr[o] = ex;
        atomicMin(sum + (size_t)(G + g) * im.wo + x,
                  ((unsigned long long)(d + (uint32_t)y) << 16) | (unsigned long long)y);
        if (ex != kEmptyKey)
            atomicMin(sum + (size_t)(2 * G + g) * im.wo + x, (((ex >> 16) - (uint64_t)x + (uint64_t)y) << 32) |
                                                                 ((uint64_t)(0xffff - y) << 16) | (ex & 0xffff));
    }
}

// Sweep 1, columns (backward): for each hole p its sweep-1 choice, from the
// column part (T.d + y) << 16 | y (minimum y on ties) of the rows below and
// the off-column part (RR.d - x + y) << 32 | (0xffff - y) << 16 | qx (largest
// y, then smallest x on ties) of its own and the rows below.  A non-hole
// below outdoes both from there on: its column term is at least as good as
// anything further down, and better than any off-column term from its row on.
//
// Then the fill of inpaint_color (inpainting.cpp:191-198) for the 2x2 blocks
// of the group that hold at least one hole, a block per thread: each hole
// follows its choice to its source and takes the source's codes (written back
// for the passes that read them later: the auxiliary outputs, the source
// list); then, unless the resize writes the output, the block's Y/U/V samples
// are written.  Sources are never holes (without any, a hole is its own), so
// the codes read here are never the ones another thread writes.
//
// Grid (strips, groups, images), 256 threads.
template <class Src>
__global__ void __launch_bounds__(32 * COL_WARPS) inpaint_cols1_kernel(const __grid_constant__ Src src) {
    grid_dep_wait();
    const InpaintImage im = src();
    __shared__ unsigned long long s_c[COL_WARPS][32], s_o[COL_WARPS][32], s_cc[COL_WARPS][32], s_co[COL_WARPS][32];
    __shared__ uint64_t s_choice[GROUP][32];
    __shared__ uint32_t s_own[GROUP];
    const int G = group_count(im.ho), g = blockIdx.y, w = blockIdx.x;
    if (g >= G || w >= im.words) return;
    const int wo = im.wo, ho = im.ho;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int x = w * 32 + lane, y0 = g * GROUP + warp * WROWS;
    const uint32_t cols = word_columns(im, w);
    const bool in = cols >> lane & 1u;
    uint32_t own[WROWS], holes = 0;
#pragma unroll
    for (int r = 0; r < WROWS; ++r) {
        own[r] = y0 + r < ho ? __ldg(im.holes + (size_t)(y0 + r) * im.words + w) & cols : 0u;
        holes |= own[r];
    }
    if (!__syncthreads_or(holes != 0u)) return;
    uint64_t t[WROWS], rr[WROWS], tp[WROWS], ds[WROWS];
#pragma unroll
    for (int r = 0; r < WROWS; ++r) {
        if (lane == 0) s_own[warp * WROWS + r] = own[r];
        if (own[r] >> lane & 1u) {
            const size_t o = (size_t)(y0 + r) * wo + x;
            t[r] = im.tq[o];
            rr[r] = im.rr[o];
            tp[r] = im.tp[o];
            ds[r] = im.ds[o];
        }
    }
    // What lies below matters only to holes that reach the group's last row.
    unsigned long long run_c = kEmptyKey, run_o = kEmptyKey;
    const int yl = min(ho, g * GROUP + GROUP) - 1;
    if (in && (__ldg(im.holes + (size_t)yl * im.words + w) >> lane & 1u))
        for (int h = g + 1 + warp; h < G; h += COL_WARPS) {
            run_c = umin64(run_c, im.sum[(size_t)(G + h) * wo + x]);
            run_o = umin64(run_o, im.sum[(size_t)(2 * G + h) * wo + x]);
        }
    s_cc[warp][lane] = run_c;
    s_co[warp][lane] = run_o;
    unsigned long long ck[WROWS], ok[WROWS], tc = kEmptyKey, to = kEmptyKey;
#pragma unroll
    for (int r = 0; r < WROWS; ++r) {
        const int y = y0 + r;
        ck[r] = ok[r] = kEmptyKey;
        if (y >= ho) continue;
        const bool hole = own[r] >> lane & 1u;
        ck[r] = ((unsigned long long)((hole ? t[r] >> 32 : 0ull) + (uint64_t)y) << 16) | (unsigned long long)y;
        if (hole && rr[r] != kEmptyKey)
            ok[r] = (((rr[r] >> 16) - (uint64_t)x + (uint64_t)y) << 32) | ((uint64_t)(0xffff - y) << 16) |
                    (rr[r] & 0xffff);
        tc = umin64(tc, ck[r]);
        to = umin64(to, ok[r]);
    }
    s_c[warp][lane] = tc;
    s_o[warp][lane] = to;
    __syncthreads();
    if (holes) {
#pragma unroll
        for (int k = 0; k < COL_WARPS; ++k) {
            run_c = umin64(run_c, s_cc[k][lane]);
            run_o = umin64(run_o, s_co[k][lane]);
            if (k > warp) {
                run_c = umin64(run_c, s_c[k][lane]);
                run_o = umin64(run_o, s_o[k][lane]);
            }
        }
#pragma unroll
        for (int r = WROWS - 1; r >= 0; --r) {
            const int y = y0 + r;
            // run_c holds the exclusive (rows below) column minimum here.
            run_o = umin64(run_o, ok[r]);
            if (own[r] >> lane & 1u) {
                uint64_t c_cost = tp[r] == ~0ull ? (uint64_t)1 << 40 : (tp[r] >> 32);
                int c_y = y;
                if (run_c != kEmptyKey) {
                    const uint64_t cost = (run_c >> 16) - (uint64_t)y;
                    if (cost < c_cost) {
                        c_cost = cost;
                        c_y = (int)(run_c & 0xffff);
                    }
                }
                uint64_t o_cost = (uint64_t)1 << 40;
                int o_x = 0, o_y = 0;
                if (run_o != kEmptyKey) {
                    o_cost = (run_o >> 32) - (uint64_t)y;
                    o_y = 0xffff - (int)((run_o >> 16) & 0xffff);
                    o_x = (int)(run_o & 0xffff);
                }
                const uint64_t d0 = ds[r] >> 32;
                // The choice: the source itself (stay: S0; own seed T'), or
                // the seed T(q) of the column or off-column minimum.
                uint64_t choice = ds[r] & 0xffffffffull;
                if (c_cost <= o_cost) {
                    if (c_cost < d0)
                        choice = (c_y == y) ? (tp[r] & 0xffffffffull)
                                            : kSeedRef | ((uint64_t)x << 16) | (uint64_t)c_y;
                } else {
                    if (o_cost < d0) choice = kSeedRef | ((uint64_t)o_x << 16) | (uint64_t)o_y;
                }
                s_choice[warp * WROWS + r][lane] = choice;
            }
            run_c = umin64(run_c, ck[r]);
        }
    }
    __syncthreads();
    const int bx = 2 * (threadIdx.x & 15), by = 2 * (threadIdx.x >> 4);
    const int px = w * 32 + bx, py = g * GROUP + by;
    const uint32_t top = s_own[by] >> bx & 3u, bottom = s_own[by + 1] >> bx & 3u;
    if (!(top | bottom)) return;
    // A raster of odd width or height (Precision != 1) ends in partial
    // blocks: their missing pixels are neither filled nor written.
    const bool has_r = px + 1 < wo, has_b = py + 1 < ho;
    uint64_t* __restrict__ codes = im.codes;
    const size_t o = (size_t)py * wo + px;
    auto fill = [&](size_t q, bool hole, uint64_t c) -> uint64_t {
        if (!hole) return codes ? codes[q] : 0ull;
        int sx = (int)((c >> 16) & 0xffff), sy = (int)(c & 0xffff);
        // T of a non-hole is the pixel itself.
        if ((c & kSeedRef) && (__ldg(im.holes + (size_t)sy * im.words + (sx >> 5)) >> (sx & 31) & 1u)) {
            const uint64_t s = im.tq[(size_t)sy * wo + sx];
            sx = (int)((s >> 16) & 0xffff);
            sy = (int)(s & 0xffff);
        }
        uint64_t v = 0;
        if (codes) {
            v = (codes[(size_t)sy * wo + sx] & kCodeMask) | kHoleBit;
            codes[q] = v;
        }
        if (im.sources) {
            im.sources[q * 2 + 0] = sx;
            im.sources[q * 2 + 1] = sy;
        }
        return v;
    };
    const uint64_t c00 = fill(o, top & 1u, s_choice[by][bx]),
                   c01 = has_r ? fill(o + 1, top & 2u, s_choice[by][bx + 1]) : 0ull,
                   c10 = has_b ? fill(o + wo, bottom & 1u, s_choice[by + 1][bx]) : 0ull,
                   c11 = has_r && has_b ? fill(o + wo + 1, bottom & 2u, s_choice[by + 1][bx + 1]) : 0ull;
    if (im.no_write) return;
    im.out_y[o] = (uint16_t)(c00 & 0xffff);
    im.out_y[o + 1] = (uint16_t)(c01 & 0xffff);
    im.out_y[o + wo] = (uint16_t)(c10 & 0xffff);
    im.out_y[o + wo + 1] = (uint16_t)(c11 & 0xffff);
    const size_t co = (size_t)(py / 2) * (wo / 2) + px / 2;
    const uint32_t su = (uint32_t)((c00 >> 16) & 0xffff) + ((c01 >> 16) & 0xffff) + ((c10 >> 16) & 0xffff) +
                        ((c11 >> 16) & 0xffff);
    const uint32_t sv = (uint32_t)((c00 >> 32) & 0xffff) + ((c01 >> 32) & 0xffff) + ((c10 >> 32) & 0xffff) +
                        ((c11 >> 32) & 0xffff);
    im.out_u[co] = quarter_round(su, im.ties_up);
    im.out_v[co] = quarter_round(sv, im.ties_up);
}

// The passes of `src` (grid z = images), sized for max_w x max_h.
template <class Src>
int launch_passes(const Src& src, int max_w, int max_h, int images, cudaStream_t s) {
    const dim3 tiles((max_w + 31) / 32, group_count(max_h), images);
    launch_dependent(inpaint_rows0_kernel<Src>, dim3((max_h + 7) / 8, 1, images), dim3(256), 0, s, src);
    launch_dependent(inpaint_cols0_kernel<Src, true>, tiles, dim3(32 * COL_WARPS), 0, s, src);
    launch_dependent(inpaint_cols0_kernel<Src, false>, tiles, dim3(32 * COL_WARPS), 0, s, src);
    launch_dependent(inpaint_rows1_kernel<Src>, dim3(max_h, 1, images), dim3(32 * ROW_WARPS), 0, s, src);
    launch_dependent(inpaint_cols1_kernel<Src>, tiles, dim3(32 * COL_WARPS), 0, s, src);
    return 5;
}

}  // namespace

size_t inpaint_sum_words(int wo, int ho) { return (size_t)3 * group_count(ho) * wo; }

template <class Tabs>
int launch_inpaint(const Tabs& tabs, const BatchShape& sh, cudaStream_t s) {
    return launch_passes(FromTables<Tabs>{tabs}, sh.max_wo, sh.max_ho, sh.slots, s);
}

template int launch_inpaint<TableParam>(const TableParam&, const BatchShape&, cudaStream_t);
template int launch_inpaint<TablePtr>(const TablePtr&, const BatchShape&, cudaStream_t);

void launch_inpaint_sources(const DevStatus* st, const uint32_t* holes, uint64_t* const scan[4], uint64_t* sum, int w,
                            int h, int32_t* sources, cudaStream_t s) {
    Direct src;
    src.im.wo = w;
    src.im.ho = h;
    src.im.words = (w + 31) / 32;
    src.im.st = st;
    src.im.holes = holes;
    src.im.codes = nullptr;
    src.im.rr = src.im.before = scan[0];
    src.im.ds = scan[1];
    src.im.tq = scan[2];
    src.im.tp = scan[3];
    src.im.sum = sum;
    src.im.sources = sources;
    src.im.out_y = src.im.out_u = src.im.out_v = nullptr;
    src.im.ties_up = 0;
    src.im.no_write = 1;
    launch_passes(src, w, h, 1, s);
}

}  // namespace rvsb
