// CUDA's names on the CPU, as far as the device headers under test need them: the 32 lanes of a
// warp are fibers that change only at warp-wide operations.  Between two of them a lane runs
// alone, which is the order that shows a missing barrier; warp_run takes the lanes in either
// direction.  A lane that ends while others wait at a warp-wide operation ends the program.
#pragma once
#include <ucontext.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <memory>
#include <vector>

#define __device__
#define __host__
#define __global__
#define __forceinline__ inline
#define __restrict__
#define __align__(n) __attribute__((aligned(n)))

struct float2 { float x, y; };
struct float4 { float x, y, z, w; };
struct int2 { int x, y; };
struct longlong2 { long long x, y; };
struct ulonglong2 { unsigned long long x, y; };
inline float2 make_float2(float x, float y) { return {x, y}; }
inline float4 make_float4(float x, float y, float z, float w) { return {x, y, z, w}; }
inline int2 make_int2(int x, int y) { return {x, y}; }
inline ulonglong2 make_ulonglong2(unsigned long long x, unsigned long long y) { return {x, y}; }
struct Dim3 { unsigned x, y, z; };
inline Dim3 threadIdx{0, 0, 0}, blockIdx{0, 0, 0}, blockDim{32, 1, 1}, gridDim{1, 1, 1};
using std::max;
using std::min;

namespace lanes {
struct Warp {
    ucontext_t home, ctx[32];
    std::unique_ptr<char[]> stack[32];
    std::function<void()> fn;
    bool done[32];
    int lane = -1;
    unsigned value[32];  // what each lane brings to the warp-wide operation
};
inline Warp *now = nullptr;
inline void entry() {
    now->fn();
    now->done[now->lane] = true;
    swapcontext(&now->ctx[now->lane], &now->home);
}
// Waits for the warp; every lane's `bring` is then in now->value.
inline void meet(unsigned bring = 0) {
    now->value[now->lane] = bring;
    swapcontext(&now->ctx[now->lane], &now->home);
}
// One warp whose lane l has threadIdx.x = first + l, lanes in ascending or descending order.
inline void warp_run(int first, bool descending, std::function<void()> fn) {
    Warp w;
    now = &w;
    w.fn = std::move(fn);
    for (int l = 0; l < 32; ++l) {
        w.stack[l].reset(new char[1 << 18]);
        w.done[l] = false;
        getcontext(&w.ctx[l]);
        w.ctx[l].uc_stack.ss_sp = w.stack[l].get();
        w.ctx[l].uc_stack.ss_size = 1 << 18;
        w.ctx[l].uc_link = nullptr;
        makecontext(&w.ctx[l], entry, 0);
    }
    for (int ended = 0; ended < 32;) {
        if (ended) {
            fprintf(stderr, "%d lanes left while the others wait\n", ended);
            exit(3);
        }
        for (int i = 0; i < 32; ++i) {
            const int l = descending ? 31 - i : i;
            w.lane = l;
            threadIdx.x = (unsigned)(first + l);
            swapcontext(&w.home, &w.ctx[l]);
        }
        for (int l = 0; l < 32; ++l) ended += w.done[l];
    }
    now = nullptr;
}
}  // namespace lanes

// warp-wide operations: one meeting to bring the values, one to keep them until all have read
inline void __syncwarp(unsigned = 0xffffffffu) { lanes::meet(); }
inline unsigned lane_read(unsigned bring, int from) {
    lanes::meet(bring);
    const unsigned v = lanes::now->value[from];
    lanes::meet();
    return v;
}
template <class T>
inline T shfl(T v, int from) {
    static_assert(sizeof(T) == 4, "");
    unsigned u;
    memcpy(&u, &v, 4);
    u = lane_read(u, from);
    memcpy(&v, &u, 4);
    return v;
}
template <class T>
inline T __shfl_sync(unsigned, T v, int from) { return shfl(v, from & 31); }
template <class T>
inline T __shfl_xor_sync(unsigned, T v, int m, int = 32) { return shfl(v, lanes::now->lane ^ m); }
template <class T>
inline T __shfl_down_sync(unsigned, T v, int d) { return shfl(v, std::min(lanes::now->lane + d, 31)); }
inline unsigned __ballot_sync(unsigned, int p) {
    lanes::meet(p != 0);
    unsigned v = 0;
    for (int l = 0; l < 32; ++l) v |= lanes::now->value[l] << l;
    lanes::meet();
    return v;
}
inline int __all_sync(unsigned m, int p) { return __ballot_sync(m, p) == 0xffffffffu; }
inline int __any_sync(unsigned m, int p) { return __ballot_sync(m, p) != 0; }

template <class T>
inline T __ldg(const T *p) { return *p; }
inline unsigned long long atomicAdd(unsigned long long *p, unsigned long long v) {
    const unsigned long long old = *p;
    *p += v;
    return old;
}
inline unsigned __cvta_generic_to_shared(const void *) { return 0; }
inline float __fmul_rn(float a, float b) { return a * b; }
inline float __fadd_rn(float a, float b) { return a + b; }
inline float __fmaf_rn(float a, float b, float c) { return std::fma(a, b, c); }
inline float2 __fadd2_rn(float2 a, float2 b) { return {a.x + b.x, a.y + b.y}; }
inline float2 __fmul2_rn(float2 a, float2 b) { return {a.x * b.x, a.y * b.y}; }
inline float2 __ffma2_rn(float2 a, float2 b, float2 c) { return {std::fma(a.x, b.x, c.x), std::fma(a.y, b.y, c.y)}; }
inline long long __float2ll_rn(float v) {  // cvt.rni.s64.f32: saturates, NaN to the lowest value
    if (std::isnan(v) || v < -9.2233720368547758e18f) return INT64_MIN;
    return v >= 9.2233720368547758e18f ? INT64_MAX : (long long)std::nearbyint(v);
}
