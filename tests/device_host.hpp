// The device intrinsics the tested kernels' helpers use, for the host: the
// same arithmetic, rounded as the device rounds it.  The approximate
// reciprocals and roots are the correctly rounded values moved by up to
// `g_ulp` ulp; a warp is 32 threads that meet in its collective operations.
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <barrier>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <limits>
#include <thread>
#include <vector>

#define __noinline__ __attribute__((noinline))

using std::max;
using std::min;
using std::isfinite;
using std::isinf;
using std::isnan;

inline float __fadd_rn(float a, float b) { return a + b; }
inline float __fsub_rn(float a, float b) { return a - b; }
inline float __fmul_rn(float a, float b) { return a * b; }
inline float __fdiv_rn(float a, float b) { return a / b; }
inline float __frcp_rn(float a) { return 1.f / a; }
inline float __fsqrt_rn(float a) { return std::sqrt(a); }
inline float __fmaf_rn(float a, float b, float c) { return std::fma(a, b, c); }
inline double __dadd_rn(double a, double b) { return a + b; }
inline double __dsub_rn(double a, double b) { return a - b; }
inline double __dmul_rn(double a, double b) { return a * b; }
inline double __ddiv_rn(double a, double b) { return a / b; }
inline double __dsqrt_rn(double a) { return std::sqrt(a); }
inline double __fma_rn(double a, double b, double c) { return std::fma(a, b, c); }
inline float __double2float_rn(double a) { return (float)a; }

template <class To, class From>
inline To bits_as(From f) {
    To t;
    static_assert(sizeof(t) == sizeof(f));
    std::memcpy(&t, &f, sizeof(t));
    return t;
}
inline float __int_as_float(int a) { return bits_as<float>(a); }
inline float __uint_as_float(unsigned a) { return bits_as<float>(a); }
inline int __float_as_int(float a) { return bits_as<int>(a); }
inline unsigned __float_as_uint(float a) { return bits_as<unsigned>(a); }
inline int __double2loint(double a) { return (int)(unsigned)bits_as<uint64_t>(a); }
inline int __float2int_rz(float a) { return (int)a; }
inline unsigned __float2uint_rz(float a) { return !(a > 0.f) ? 0u : a >= 4294967296.f ? ~0u : (unsigned)a; }
inline unsigned __funnelshift_r(unsigned lo, unsigned hi, unsigned s) {
    return (unsigned)((((uint64_t)hi << 32) | lo) >> (s & 31));
}
inline int __popc(unsigned a) { return __builtin_popcount(a); }

// Approximations: off by a number of ulp drawn from -g_ulp .. g_ulp.
inline int g_ulp = 0;
inline thread_local unsigned t_draw = 1;
inline float off_by(float v) {
    if (g_ulp == 0 || !std::isfinite(v) || v == 0.f) return v;
    t_draw = t_draw * 1664525u + 1013904223u;
    return bits_as<float>(bits_as<int>(v) + (int)((t_draw >> 8) % (2 * g_ulp + 1)) - g_ulp);
}
inline float flushed(float v) { return std::fabs(v) < std::numeric_limits<float>::min() ? std::copysign(0.f, v) : v; }
inline float ptx_rcp(float x) { return off_by((float)(1.0 / (double)x)); }
inline float ptx_rcp_ftz(float x) { return flushed(ptx_rcp(flushed(x))); }
inline float ptx_rsqrt_ftz(float x) { return off_by((float)(1.0 / std::sqrt((double)flushed(x)))); }
inline float __fdividef(float a, float b) { return std::fabs(b) > 0x1p126f ? 0.f : off_by((float)((double)a / (double)b)); }

// Loads: one outside the table set here is noted and gives 0.
inline const void* g_table = nullptr;
inline size_t g_table_bytes = 0;
inline int g_bad_loads = 0;
template <class T>
inline T __ldg(const T* p) {
    const uintptr_t a = (uintptr_t)p, b = (uintptr_t)g_table;
    if (g_table && (a < b || a + sizeof(T) > b + g_table_bytes)) {
        ++g_bad_loads;
        return T{};
    }
    return *p;
}

// A warp of 32 threads.
struct Warp {
    std::barrier<> meet{32};
    uint32_t word[32];
};
inline thread_local Warp* t_warp = nullptr;
inline thread_local int t_lane = 0;
inline void __syncwarp() { t_warp->meet.arrive_and_wait(); }
inline unsigned __ballot_sync(unsigned, bool v) {
    t_warp->word[t_lane] = v;
    __syncwarp();
    unsigned m = 0;
    for (int k = 0; k < 32; ++k) m |= t_warp->word[k] << k;
    __syncwarp();
    return m;
}
inline int __shfl_sync(unsigned, int v, int from) {
    t_warp->word[t_lane] = (uint32_t)v;
    __syncwarp();
    const int r = (int)t_warp->word[from & 31];
    __syncwarp();
    return r;
}
inline int atomicAdd(int* p, int v) { return __atomic_fetch_add(p, v, __ATOMIC_RELAXED); }
template <class F>
void run_warp(F&& f) {
    Warp w;
    std::vector<std::thread> t;
    for (int k = 0; k < 32; ++k)
        t.emplace_back([&, k] {
            t_warp = &w;
            t_lane = k;
            f(k);
        });
    for (auto& x : t) x.join();
}
