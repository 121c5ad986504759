// Collaborative filter, finish and batch kernels.
//
// Compiled for sm_100a with -use_fast_math, the same floating-point mode as the
// reference kernel (vszipcu src/bm3d.zig:20-24): flush-to-zero, approximate
// division / square root, FMA contraction.  The transforms and the shrinkage follow
// the reference's operation order.
//
// Design (B200):
//  * Filtering: 8 lanes per group, packed FP32x2 transforms (zb3d_filter.cuh).
//  * Aggregation: signed 64-bit fixed point (2^32 = 1.0) with integer atomics,
//    which is exact and order independent; the weight sum is accumulated once
//    per patch at its origin and expanded by an 8x8 box sum in the finish pass.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "zb3d_args.h"
#include "zb3d_filter.cuh"
#include "zb3d_match.cuh"
#include "zb3d_match_scan.cuh"
#include "zb3d_transforms.cuh"

namespace zb {

// The DCT in both dimensions: 2 warps of 4 groups per CTA (filter8_groups).
template <bool FINAL>
__global__ void __launch_bounds__(kFilter8Warps * 32) zb_filter8(FilterArgs a) {
    __shared__ __align__(16) float sbuf[kFilterGroups * kGroupStride];
    __shared__ __align__(16) float cbuf[FINAL ? kFilterGroups * kGroupStride : 4];  // Wiener coefficients
    __shared__ long long offs[kFilterGroups * kOffStride];
    filter8_groups<FINAL>(a, (long long)blockIdx.x * kFilterGroups, sbuf, cbuf, offs);
}

// ---------------------------------------------------------------------------
// Collaborative filtering (vszipcu src/bm3d.cu:392-546) and aggregation into
// signed 64-bit fixed point.
// ---------------------------------------------------------------------------
static constexpr int kFilterWarps = 4;

// ---------------------------------------------------------------------------
// Collaborative filtering with 16 lanes per group.  Lane (j, h), j = 0..7,
// h = 0..1, holds 32 of the group's 512 values, half of what a lane of an
// 8-lane group holds, so twice as many groups are resident per SM.  Every 1-D
// transform still runs on 8 values inside one lane, in the reference's order;
// between transforms the values move through shared memory.  The layouts
// (q, t = 0..3; the half h takes the interleaved indices 2q + h, 2t + h):
//   A  column x = j of patches 2q + h, all rows          gather, vertical forward
//   B  row fy = j of patches 2q + h, all columns         horizontal forward
//   C  column fx = j, rows fy = 2t + h, all patches      across patches (Wiener coefficients)
//   D  column fx = j of spectra 2q + h, all rows         shrinkage, vertical inverse
//   E  row y = j of spectra 2q + h, all columns          horizontal inverse
//   F  column x = j, rows y = 2t + h, all patches        inverse across patches, aggregation
// Registers: A, B, D, E as d[q * 8 + i]; C, F as d[p * 4 + t].  The strides of the
// three kinds of move (A->B and D->E, B->C and E->F, C->D) were chosen so that the
// 32 lanes of a warp (two groups) touch 32 distinct banks on every store and load.
// The shrinkage runs in layout D with the vertical inverse directly after it in
// registers, the same code shape as the reference (src/bm3d.cu:445, 457-478): its
// transforms write a * b + c and leave the fusing into FMAs to the compiler, and
// the compiler fuses this stage the reference's way only in that shape.
// ---------------------------------------------------------------------------
static constexpr int kGroupBuf = 592;    // floats per group in the move buffer
static constexpr int kCoeffBuf = 592;    // floats per group in the Wiener coefficient buffer

// A -> B and D -> E: 8x8 transpose of each of the lane's four patches
__device__ __forceinline__ void move_tr(float (&d)[32], float *gb, int h, int j, unsigned gm) {
    __syncwarp(gm);
#pragma unroll
    for (int q = 0; q < 4; ++q)
#pragma unroll
        for (int i = 0; i < 8; ++i) gb[(2 * q + h) * 72 + i + 9 * j] = d[q * 8 + i];
    __syncwarp(gm);
#pragma unroll
    for (int q = 0; q < 4; ++q)
#pragma unroll
        for (int i = 0; i < 8; ++i) d[q * 8 + i] = gb[(2 * q + h) * 72 + j + 9 * i];
}

// B -> C and E -> F: (patch 2q + h, row j, column i) -> (patch p, row 2t + h, column j)
__device__ __forceinline__ void move_bc(float (&d)[32], float *gb, int h, int j, unsigned gm) {
    __syncwarp(gm);
#pragma unroll
    for (int q = 0; q < 4; ++q)
#pragma unroll
        for (int i = 0; i < 8; ++i) gb[(2 * q + h) * 72 + 9 * j + 2 * i] = d[q * 8 + i];
    __syncwarp(gm);
#pragma unroll
    for (int p = 0; p < 8; ++p)
#pragma unroll
        for (int t = 0; t < 4; ++t) d[p * 4 + t] = gb[p * 72 + 9 * (2 * t + h) + 2 * j];
}

// C -> D: (spectrum p, row 2t + h, column j) -> (spectrum 2q + h, row i, column j)
__device__ __forceinline__ void move_cd(float (&d)[32], float *gb, int h, int j, unsigned gm) {
    __syncwarp(gm);
#pragma unroll
    for (int p = 0; p < 8; ++p)
#pragma unroll
        for (int t = 0; t < 4; ++t) gb[p * 72 + 8 * (2 * t + h) + j] = d[p * 4 + t];
    __syncwarp(gm);
#pragma unroll
    for (int q = 0; q < 4; ++q)
#pragma unroll
        for (int i = 0; i < 8; ++i) d[q * 8 + i] = gb[(2 * q + h) * 72 + 8 * i + j];
}

// layout A -> layout C through the forward 3D transform
template <class T2, class T1>
__device__ __forceinline__ void forward3_16(float (&d)[32], float *gb, int h, int j, unsigned gm) {
#pragma unroll
    for (int q = 0; q < 4; ++q) T2::fwd(&d[q * 8]);
    move_tr(d, gb, h, j, gm);
#pragma unroll
    for (int q = 0; q < 4; ++q) T2::fwd(&d[q * 8]);
    move_bc(d, gb, h, j, gm);
#pragma unroll
    for (int t = 0; t < 4; ++t) {
        float v[8];
#pragma unroll
        for (int p = 0; p < 8; ++p) v[p] = d[p * 4 + t];
        T1::fwd(v);
#pragma unroll
        for (int p = 0; p < 8; ++p) d[p * 4 + t] = v[p];
    }
}

// layout D (after the shrinkage) -> layout F through the rest of the inverse 3D
// transform: vertical, horizontal, then across patches
template <class T2, class T1>
__device__ __forceinline__ void inverse3_16(float (&d)[32], float *gb, int h, int j, unsigned gm) {
#pragma unroll
    for (int q = 0; q < 4; ++q) T2::inv(&d[q * 8]);
    move_tr(d, gb, h, j, gm);
#pragma unroll
    for (int q = 0; q < 4; ++q) T2::inv(&d[q * 8]);
    move_bc(d, gb, h, j, gm);
#pragma unroll
    for (int t = 0; t < 4; ++t) {
        float v[8];
#pragma unroll
        for (int p = 0; p < 8; ++p) v[p] = d[p * 4 + t];
        T1::inv(v);
#pragma unroll
        for (int p = 0; p < 8; ++p) d[p * 4 + t] = v[p];
    }
}

// the lane's four patches 2q + h, column j, into layout A
__device__ __forceinline__ void gather16(float (&d)[32], const float *plane, const FilterArgs &a, long long grp,
                                         int h, int j) {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const int2 v = a.list[grp * 8 + 2 * q + h];
        const float *s = plane + ((unsigned)v.y >> 24) * a.frame_stride + (long long)(v.y & 0xffffff) * a.pitch + v.x + j;
#pragma unroll
        for (int i = 0; i < 8; ++i) d[q * 8 + i] = __ldg(s + i * a.pitch);
    }
}

// Groups g0 + threadIdx.x / 16 (16 lanes each) of one entry; tbuf: kFilterWarps * 2 *
// kGroupBuf floats, cbuf (Wiener): (blockDim.x / 16) * kCoeffBuf floats.
template <bool FINAL, int T2D, int T1D>
__device__ __forceinline__ void filter16_groups(const FilterArgs &a, long long g0, float *tbuf, float *cbuf) {
    using T2 = typename TransformOf<T2D>::type;
    using T1 = typename TransformOf<T1D>::type;
    const int lane = threadIdx.x & 31;
    const int j = lane & 7, h = (lane >> 3) & 1, gw = lane >> 4;
    const unsigned gm = 0xffffu << (lane & 16);
    const long long grp = g0 + (threadIdx.x >> 4);
    if (grp >= a.nblocks) return;
    float *gb = tbuf + ((threadIdx.x >> 5) * 2 + gw) * kGroupBuf;
    float *cb = cbuf + (threadIdx.x >> 4) * kCoeffBuf;
    const float E = a.extractor;

    for (int pl = 0; pl < a.nplanes; ++pl) {
        const float sigma = pl == 0 ? a.sigma[0] : (pl == 1 ? a.sigma[1] : a.sigma[2]);
        if (a.chroma && sigma < ZB_FLT_EPS) continue;
        float d[32];
        float k = 0.0f;
        if constexpr (FINAL) {
            // Wiener coefficients r^2 / (r^2 + sigma^2) of the basic estimate's spectrum (the
            // reference rounds r^2 once and adds sigma^2 without FMA); the weight's sum of
            // squared coefficients (after the shrinkage below) is accumulated by FMA over
            // spectrum and row for column j in the reference's order: every lane runs the full
            // chain of its column.  The basic estimate and the noisy patches share one copy of
            // the forward transform's code.
            const float s2 = sigma * sigma;
#pragma unroll 1
            for (int pass = 0; pass < 2; ++pass) {
                gather16(d, a.src + (pass ? a.clip_stride : 0) + pl * a.plane_stride, a, grp, h, j);
                forward3_16<T2, T1>(d, gb, h, j, gm);
                if (pass) break;
#pragma unroll
                for (int p = 0; p < 8; ++p)
#pragma unroll
                    for (int t = 0; t < 4; ++t) {
                        const float rv = d[p * 4 + t];
                        const float r2 = __fmul_rn(rv, rv);
                        float coeff = r2 / __fadd_rn(r2, s2);
                        if (p == 0 && t == 0 && h == 0 && j == 0) coeff = 1.0f;
                        cb[p * 72 + (2 * t + h) * 8 + j] = coeff;
                    }
                __syncwarp(gm);
            }
        } else {
            gather16(d, a.src + pl * a.plane_stride, a, grp, h, j);
            forward3_16<T2, T1>(d, gb, h, j, gm);
        }
        // shrinkage in layout D, right before the vertical inverse: d[q * 8 + i] is
        // spectrum 2q + h, row i, column j
        move_cd(d, gb, h, j, gm);
        if constexpr (!FINAL) {
#pragma unroll
            for (int q = 0; q < 4; ++q)
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const float val = d[q * 8 + i];
                    const float thr = (q == 0 && i == 0 && h == 0 && j == 0) ? 0.0f : sigma;
                    const float flag = fabsf(val) >= thr;
                    k += flag;
                    d[q * 8 + i] = flag ? (val * (1.0f / 4096.0f)) : 0.0f;
                }
            // kept-coefficient count: integer-valued, exact in any order
            k += __shfl_xor_sync(gm, k, 1, 16);
            k += __shfl_xor_sync(gm, k, 2, 16);
            k += __shfl_xor_sync(gm, k, 4, 16);
            k += __shfl_xor_sync(gm, k, 8, 16);
        } else {
#pragma unroll
            for (int q = 0; q < 4; ++q)
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    float val = d[q * 8 + i];
                    val *= cb[(2 * q + h) * 72 + i * 8 + j];
                    d[q * 8 + i] = val * (1.0f / 4096.0f);
                }
            // the weight's chain, here so that it can overlap the vertical inverse transforms
            // (it only reads the coefficient buffer)
#pragma unroll 8
            for (int p = 0; p < 8; ++p)
#pragma unroll
                for (int r = 0; r < 8; ++r) {
                    const float c = cb[p * 72 + r * 8 + j];
                    k = __fmaf_rn(c, c, k);
                }
            k += __shfl_xor_sync(gm, k, 1, 8);
            k += __shfl_xor_sync(gm, k, 2, 8);
            k += __shfl_xor_sync(gm, k, 4, 8);
        }
        const float w = 1.0f / k;
        inverse3_16<T2, T1>(d, gb, h, j, gm);

        unsigned long long *num = a.num + pl * a.acc_plane_stride;
#pragma unroll
        for (int p = 0; p < 8; ++p) {
            const int2 v = a.list[grp * 8 + p];
            unsigned long long *q = num + ((unsigned)v.y >> 24) * a.acc_frame_stride +
                                    (long long)(v.y & 0xffffff) * a.pitch + v.x + j;
#pragma unroll
            for (int t = 0; t < 4; ++t) {
                const float val = __fmaf_rn(w, d[p * 4 + t], E) - E;
                atomicAdd(q + (2 * t + h) * a.pitch, to_fix(val * kFixScale));
            }
        }
        if (h == 0) {
            // lane j books the weight of patch j once, at its origin
            const float wq = (w + E) - E;
            const int2 v = a.list[grp * 8 + j];
            atomicAdd(a.den + pl * a.acc_plane_stride + ((unsigned)v.y >> 24) * a.acc_frame_stride +
                          (long long)(v.y & 0xffffff) * a.pitch + v.x,
                      to_fix(wq * kFixScale));
        }
        __syncwarp(gm);  // the coefficient buffer is rewritten by the next plane
    }
}

template <bool FINAL, int T2D, int T1D>
__global__ void __launch_bounds__(kFilterWarps * 32) zb_filter16(FilterArgs a) {
    __shared__ float tbuf[kFilterWarps * 2 * kGroupBuf];
    // Wiener: the group's 512 coefficients at [spectrum * 72 + row * 8 + column]
    extern __shared__ float cbuf[];
    filter16_groups<FINAL, T2D, T1D>(a, (long long)blockIdx.x * (blockDim.x >> 4), tbuf, cbuf);
}

// ---------------------------------------------------------------------------
// Finish: fixed point -> float.  The weight at a pixel is the 8x8 box sum of the
// origin weights whose patch covers it.  mode 0 writes num/den (radius 0,
// src/bm3d.cu:898-922, IEEE division); mode 1 writes the stacked accumulator
// planes [plane][t][2][h][pitch] of the temporal path (src/bm3d.zig:1224-1231).
// ---------------------------------------------------------------------------
struct FinishArgs {
    const unsigned long long *num, *den;
    long long acc_plane_stride, acc_frame_stride;
    int w, h, pitch;
    int tw;
    unsigned proc_mask;       // planes written (bit p)
    float *dst;               // mode 0: [planes][h][dst_pitch]; mode 1: stacked
    int dst_pitch;
    long long dst_plane_stride;
    int mode;
};

// One warp per strip of 56 output columns and `rows` output rows (a multiple of 8).  A lane
// owns two neighbouring columns (16-byte loads; 8 columns to the left of the strip are read for
// their weights only) and walks down them in chunks of 8 rows, all of whose loads are in
// flight together: the 8-row sum of origin weights of a column slides in registers, and the
// 8-column sum over it comes from three exchanges between lanes.  The sums are int64, exact in
// any order.  No shared memory and no barrier: the kernel moves 16 B + 4 or 8 B per pixel and
// is bound by that.  (A 39 x 39 tile of weights in shared memory summed per pixel, the form
// before, took 71 us for
// the five 1080p slots of a radius 2 window and 24 us for three 720p planes; this one 46 and 17.)
constexpr int kFinishCols = 56;
constexpr int kFinishWarps = 4;

__device__ __forceinline__ longlong2 finish_load(const unsigned long long *row, int x, int w, bool vec) {
    longlong2 v = make_longlong2(0, 0);
    if (x < 0 || x >= w) return v;
    if (vec && x + 1 < w) return *reinterpret_cast<const longlong2 *>(row + x);
    v.x = (long long)row[x];
    if (x + 1 < w) v.y = (long long)row[x + 1];
    return v;
}

// vec: rows of the accumulators start on 16 bytes (an even pitch); vec_out: pairs of output
// pixels on 8 bytes.
__global__ void __launch_bounds__(kFinishWarps * 32) zb_finish(FinishArgs a, int rows, bool vec, bool vec_out) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int plane = blockIdx.z / a.tw, slot = blockIdx.z - plane * a.tw;
    if (!((a.proc_mask >> plane) & 1)) return;
    const int xs = (blockIdx.x * kFinishWarps + warp) * kFinishCols;
    if (xs >= a.w) return;
    const int x = xs - 8 + 2 * lane, y0 = blockIdx.y * rows;
    const long long base = plane * a.acc_plane_stride + slot * a.acc_frame_stride;
    const unsigned long long *num = a.num + base, *den = a.den + base;
    const bool out = lane >= 4 && x < a.w;
    float *o = a.dst + plane * a.dst_plane_stride + (a.mode ? (long long)slot * 2 * a.h * a.dst_pitch : 0);
    const long long second = (long long)a.h * a.dst_pitch;  // mode 1: the weights' plane
    longlong2 prev[8];
    long long sa = 0, sb = 0;  // 8-row sums of the two columns
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        const int y = y0 - 8 + k;
        prev[k] = y >= 0 ? finish_load(den + (long long)y * a.pitch, x, a.w, vec) : make_longlong2(0, 0);
    }
    longlong2 cur[8], n[8];
    auto load = [&](int yc) {  // weights and numerators of 8 rows
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const int y = min(yc + k, a.h - 1);
            cur[k] = finish_load(den + (long long)y * a.pitch, x, a.w, vec);
            n[k] = out ? finish_load(num + (long long)y * a.pitch, x, a.w, vec) : make_longlong2(0, 0);
        }
    };
    load(y0);  // before the sums below wait for their loads
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        sa += prev[k].x;
        sb += prev[k].y;
    }
    const int yend = min(y0 + rows, a.h);
    for (int yc = y0;;) {
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const int y = yc + k;
            sa += cur[k].x - prev[k].x;
            sb += cur[k].y - prev[k].y;
            prev[k] = cur[k];
            // columns x - 6 .. x + 1, and x - 7 .. x
            long long wb = sa + sb;
            wb += __shfl_up_sync(0xffffffffu, wb, 1);
            wb += __shfl_up_sync(0xffffffffu, wb, 2);
            const long long wa = wb - sb + __shfl_up_sync(0xffffffffu, sb, 4);
            if (!out || y >= yend) continue;
            const float na = __ll2float_rn(n[k].x) * kFixInv, nb = __ll2float_rn(n[k].y) * kFixInv;
            const float da = __ll2float_rn(wa) * kFixInv, db = __ll2float_rn(wb) * kFixInv;
            float *row = o + (long long)y * a.dst_pitch + x;
            if (a.mode == 0) {
                const float2 v = make_float2(__fdiv_rn(na, da), __fdiv_rn(nb, db));
                if (vec_out && x + 1 < a.w) {
                    *reinterpret_cast<float2 *>(row) = v;
                } else {
                    row[0] = v.x;
                    if (x + 1 < a.w) row[1] = v.y;
                }
            } else if (vec_out && x + 1 < a.w) {
                *reinterpret_cast<float2 *>(row) = make_float2(na, nb);
                *reinterpret_cast<float2 *>(row + second) = make_float2(da, db);
            } else {
                row[0] = na;
                row[second] = da;
                if (x + 1 < a.w) {
                    row[1] = nb;
                    row[second + 1] = db;
                }
            }
        }
        if ((yc += 8) >= yend) break;
        load(yc);
    }
}

// ---------------------------------------------------------------------------
// Batch: two launches over a work list of several plane entries (of any sizes) that share the
// filter kind, one CTA per item: the match tiles of every entry, then the filter chunks of
// every entry.  A filter chunk checks, bounded, that all of its entry's match tiles are done
// (the launches are stream-ordered, so they are; on timeout the chunk is skipped and the
// status word set, and the chunks after it do not wait).  Lists are written and read with
// ordinary loads and a fence on both sides of the counter.
// Items go to CTAs in order, so those in flight are neighbours in a plane and share its
// lines, and the CTAs of a higher-priority stream get their turn between them.  (Persistent
// CTAs taking chunks of 128 groups from a counter kept the entries outside the list waiting for
// whole phases, and spread the chunks in flight over a third of a 4K
// plane.  Four clips from 720x480 to 3840x2160 in one call: filter phase 1948 -> 1396 us with the
// 8-lane filter, the call 4.9 -> 3.9 ms.)
// ---------------------------------------------------------------------------
__device__ __forceinline__ int batch_entry_of(const BatchArgs &b, long long item, bool filter) {
    int lo = 0, hi = b.nentries - 1;  // last entry whose first item <= item
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        const long long f = filter ? b.entries[mid].first_filter : b.entries[mid].first_match;
        if (f <= item) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// PHASE 1: a match tile (8 warps); PHASE 2: a filter chunk (2 warps).
template <bool FINAL, int PHASE>
__global__ void __launch_bounds__(PHASE == 1 ? kScanWarps * 32 : kFilter8Warps * 32) zb_batch(const __grid_constant__ BatchArgs b) {
    extern __shared__ __align__(16) float dyn[];  // matching tile
    __shared__ __align__(16) float sbuf[PHASE == 1 ? 4 : kFilterGroups * kGroupStride];
    __shared__ __align__(16) float cbuf[PHASE == 1 || !FINAL ? 4 : kFilterGroups * kGroupStride];
    __shared__ long long offs[PHASE == 1 ? 1 : kFilterGroups * kOffStride];
    __shared__ int s_ok;
    static_assert(PHASE == 1 || PHASE == 2, "match phase or filter phase");
    const long long item = (PHASE == 2 ? b.match_total : 0) + blockIdx.x;
    if constexpr (PHASE == 1) {
        const int e = batch_entry_of(b, item, false);
        const BatchEntry &E = b.entries[e];
        const MatchArgs &m = E.m;
        const int local = (int)(item - E.first_match);
        const int bx = local % E.tiles_x, by = local / E.tiles_x;
        zero_slice(E.zero, local, E.match_items);
        if (bx == m.tiles_x) {  // the clamped last block column
            const int warp = threadIdx.x >> 5, cy = by * E.rows + warp;
            if (warp < E.rows && cy < m.nby) warp_block<M_SSD>(m, m.nbx - 1, cy);
        } else if (E.direct) {
            if (m.bs == 4) scan_tile<M_SSD, true, 4, false>(m, bx, by, kScanWarps, dyn);
            else scan_tile<M_SSD, false, 8, false>(m, bx, by, kScanWarps, dyn);
        } else {
            if (m.bs == 4) scan_tile<M_SSD, true, 4, true>(m, bx, by, E.rows, dyn);
            else scan_tile<M_SSD, false, 8, true>(m, bx, by, E.rows, dyn);
        }
        __threadfence();  // each thread's list stores before the tile's count
        __syncthreads();
        if (threadIdx.x == 0) atomicAdd(&b.match_done[e], 1u);
    } else {
        const int e = batch_entry_of(b, item, true);
        const BatchEntry &E = b.entries[e];
        if (threadIdx.x == 0) {
            const unsigned need = (unsigned)E.match_items + ((b.unsatisfiable && e == 0) ? 1u : 0u);
            volatile unsigned *done = b.match_done + e;
            int ok = 0;
            for (unsigned i = 0; i < b.wait_polls && *(volatile int *)b.status == 0; ++i) {
                if (*done >= need) {
                    ok = 1;
                    break;
                }
                __nanosleep(100);
            }
            if (!ok) atomicCAS(b.status, 0, 1);
            s_ok = ok;
        }
        __syncthreads();
        if (!s_ok) return;  // this chunk is left out; the status tells the host
        __threadfence();      // the count before the lists, for every reading thread
        const FilterArgs &f = E.f;
        const long long g0 = (item - E.first_filter) * kBatchGroups;
#pragma unroll 1
        for (int g = 0; g < kBatchGroups && g0 + g < f.nblocks; g += kFilterGroups)
            filter8_groups<FINAL>(f, g0 + g, sbuf, cbuf, offs);
    }
}

// ---------------------------------------------------------------------------
// Host-side launchers.
// ---------------------------------------------------------------------------
template <bool FINAL, int T2D, int T1D>
static cudaError_t launch_filter_t(const FilterArgs &a, cudaStream_t st) {
    if constexpr (T2D == T_DCT && T1D == T_DCT) {
        const unsigned grid = (unsigned)(((long long)a.nblocks + kFilterGroups - 1) / kFilterGroups);
        zb_filter8<FINAL><<<grid, kFilter8Warps * 32, 0, st>>>(a);
        return cudaGetLastError();
    } else {
        const long long threads = (long long)a.nblocks * 16;
        const int tpb = kFilterWarps * 32;
        const int dyn = FINAL ? (tpb / 16) * kCoeffBuf * (int)sizeof(float) : 0;  // Wiener coefficient buffer
        auto k = zb_filter16<FINAL, T2D, T1D>;
        if (FINAL) {
            cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, dyn);
            if (e != cudaSuccess) return e;
        }
        k<<<(unsigned)((threads + tpb - 1) / tpb), tpb, dyn, st>>>(a);
        return cudaGetLastError();
    }
}

template <bool FINAL, int T2D>
static cudaError_t launch_filter_f2(const FilterArgs &a, int t1d, cudaStream_t st) {
    switch (t1d) {
    case T_DCT: return launch_filter_t<FINAL, T2D, T_DCT>(a, st);
    case T_HAAR: return launch_filter_t<FINAL, T2D, T_HAAR>(a, st);
    case T_WHT: return launch_filter_t<FINAL, T2D, T_WHT>(a, st);
    default: return launch_filter_t<FINAL, T2D, T_BIOR15>(a, st);
    }
}

template <bool FINAL>
static cudaError_t launch_filter_f(const FilterArgs &a, int t2d, int t1d, cudaStream_t st) {
    switch (t2d) {
    case T_DCT: return launch_filter_f2<FINAL, T_DCT>(a, t1d, st);
    case T_HAAR: return launch_filter_f2<FINAL, T_HAAR>(a, t1d, st);
    case T_WHT: return launch_filter_f2<FINAL, T_WHT>(a, t1d, st);
    default: return launch_filter_f2<FINAL, T_BIOR15>(a, t1d, st);
    }
}

cudaError_t launch_filter(const FilterArgs &a, bool final_, int t2d, int t1d, cudaStream_t st) {
    return final_ ? launch_filter_f<true>(a, t2d, t1d, st) : launch_filter_f<false>(a, t2d, t1d, st);
}

cudaError_t launch_finish(const unsigned long long *num, const unsigned long long *den, long long acc_plane_stride,
                          long long acc_frame_stride, int w, int h, int pitch, int nplanes, int tw,
                          unsigned proc_mask, float *dst, int dst_pitch, long long dst_plane_stride, int mode,
                          cudaStream_t st) {
    FinishArgs a;
    a.num = num;
    a.den = den;
    a.acc_plane_stride = acc_plane_stride;
    a.acc_frame_stride = acc_frame_stride;
    a.w = w;
    a.h = h;
    a.pitch = pitch;
    a.tw = mode == 0 ? 1 : tw;
    a.proc_mask = proc_mask;
    a.dst = dst;
    a.dst_pitch = dst_pitch;
    a.dst_plane_stride = dst_plane_stride;
    a.mode = mode;
    const int strips = (w + kFinishCols - 1) / kFinishCols, planes = nplanes * a.tw;
    // 32 rows read 25% more weights than pixels, 8 rows 100%: fewer rows only where 32 would
    // leave warps missing (16 fit an SM)
    const int rows = (long long)strips * ((h + 31) / 32) * planes >= 148 * 16 ? 32 : 8;
    const bool vec = pitch % 2 == 0 && acc_plane_stride % 2 == 0 && acc_frame_stride % 2 == 0 &&
                     reinterpret_cast<uintptr_t>(num) % 16 == 0 && reinterpret_cast<uintptr_t>(den) % 16 == 0;
    const bool vec_out = dst_pitch % 2 == 0 && dst_plane_stride % 2 == 0 && reinterpret_cast<uintptr_t>(dst) % 8 == 0;
    dim3 grid((strips + kFinishWarps - 1) / kFinishWarps, (h + rows - 1) / rows, planes);
    zb_finish<<<grid, kFinishWarps * 32, 0, st>>>(a, rows, vec, vec_out);
    return cudaGetLastError();
}

// The batch kernels for the filter kind (final, t2d, t1d); only the DCT in both dimensions
// is built in (other kinds run entry by entry).  match_smem: dynamic shared memory of the
// match items.
cudaError_t launch_batch(const BatchArgs &b, bool final_, int t2d, int t1d, size_t match_smem, cudaStream_t st) {
    if (t2d != T_DCT || t1d != T_DCT) return cudaErrorNotSupported;
    if (b.match_total <= 0) return cudaSuccess;
    auto match = zb_batch<false, 1>;  // the same for both filter kinds
    // the same limit at every launch (see launch_scan_t)
    cudaError_t e = cudaFuncSetAttribute(match, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemOptIn);
    if (e != cudaSuccess) return e;
    match<<<(unsigned)b.match_total, kScanWarps * 32, match_smem, st>>>(b);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    auto filter = final_ ? zb_batch<true, 2> : zb_batch<false, 2>;
    filter<<<(unsigned)(b.items_total - b.match_total), kFilter8Warps * 32, 0, st>>>(b);
    return cudaGetLastError();
}

}  // namespace zb
