// Match lists, patch distances and candidate scans shared by the matching kernels
// (zb3d_match.cu, zb3d_match_scan.cuh, zb3d_match_tc.cu).
#pragma once
#include <cuda_runtime.h>

#include "zb3d_args.h"

namespace zb {

#define ZB_FLT_MAX 3.402823466e+38f
#define ZB_FLT_EPS 1.192092896e-07f

// ---------------------------------------------------------------------------
// Top-8 list: sorted by distance; a candidate enters before the first strictly
// larger entry (vszipcu src/bm3d.cu:641-653), so ties keep scan order.
// ---------------------------------------------------------------------------
__device__ __forceinline__ void top8_insert(float (&e)[8], int (&q)[8], float err, int pos) {
#pragma unroll
    for (int i = 7; i > 0; --i) {
        const bool ci = err < e[i];
        const bool cp = err < e[i - 1];
        e[i] = cp ? e[i - 1] : (ci ? err : e[i]);
        q[i] = cp ? q[i - 1] : (ci ? pos : q[i]);
    }
    if (err < e[0]) {
        e[0] = err;
        q[0] = pos;
    }
}

// The same strict-less insertion into a list of K entries.  Its entries are the first K
// of the 8-entry list that the same candidates would build (stable in scan order).
template <int K>
__device__ __forceinline__ void topk_insert(float (&e)[K], int (&q)[K], float err, int pos) {
#pragma unroll
    for (int i = K - 1; i > 0; --i) {
        const bool ci = err < e[i];
        const bool cp = err < e[i - 1];
        e[i] = cp ? e[i - 1] : (ci ? err : e[i]);
        q[i] = cp ? q[i - 1] : (ci ? pos : q[i]);
    }
    if (err < e[0]) {
        e[0] = err;
        q[0] = pos;
    }
}

__device__ __forceinline__ void top8_insert_z(float (&e)[8], int (&q)[8], int (&z)[8], float err, int pos, int zz) {
#pragma unroll
    for (int i = 7; i > 0; --i) {
        const bool ci = err < e[i];
        const bool cp = err < e[i - 1];
        e[i] = cp ? e[i - 1] : (ci ? err : e[i]);
        q[i] = cp ? q[i - 1] : (ci ? pos : q[i]);
        z[i] = cp ? z[i - 1] : (ci ? zz : z[i]);
    }
    if (err < e[0]) {
        e[0] = err;
        q[0] = pos;
        z[0] = zz;
    }
}

__device__ __forceinline__ int pack_pos(int x, int y) { return x | (y << 16); }
__device__ __forceinline__ int pos_x(int p) { return p & 0xffff; }
__device__ __forceinline__ int pos_y(int p) { return (int)((unsigned)p >> 16); }

// Writes a finished list (with self inclusion at radius 0) and its distances.
__device__ __forceinline__ void store_list(const MatchArgs &a, long long bi, int xb, int y, float (&e)[8],
                                           int (&q)[8]) {
    const int self = pack_pos(xb, y);
    if (a.self_incl) {
        bool found = false;
#pragma unroll
        for (int i = 0; i < 8; ++i) found |= (q[i] == self);
        if (!found) {
#pragma unroll
            for (int i = 7; i > 0; --i) {
                e[i] = e[i - 1];
                q[i] = q[i - 1];
            }
            e[0] = 0.0f;
            q[0] = self;
        }
    }
    int2 *out = a.list + bi * 8;
    const int zr = a.radius << 24;
#pragma unroll
    for (int i = 0; i < 8; ++i) out[i] = make_int2(pos_x(q[i]), pos_y(q[i]) | zr);
    if (a.errs) {
#pragma unroll
        for (int i = 0; i < 8; ++i) a.errs[bi * 8 + i] = e[i];
    }
}

constexpr unsigned kFull = 0xffffffffu;

// ---------------------------------------------------------------------------
// Global -> shared staging with cp.async: no register round trip, every copy of
// the CTA in flight at once, one wait.  Columns outside [0, w) are zero-filled
// (src-size 0; the source address then stays a valid in-plane address).
// ---------------------------------------------------------------------------
__device__ __forceinline__ void cp_async_f32(float *sdst, const float *gsrc, bool valid) {
    const unsigned saddr = (unsigned)__cvta_generic_to_shared(sdst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(saddr), "l"(gsrc), "r"(valid ? 4 : 0)
                 : "memory");
}

__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

// rows [0, nrows) x cols [0, ncols) of the plane window at (gx0, gy0) -> smem rows of pitch sp
__device__ __forceinline__ void stage_window(float *smem, int sp, const float *plane, long long pitch, int gx0,
                                             int gy0, int nrows, int ncols, int w) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    for (int r = warp; r < nrows; r += nw) {
        const float *srow = plane + (long long)(gy0 + r) * pitch;
        float *drow = smem + r * sp;
        for (int c = lane; c < ncols; c += 32) {
            const int gx = gx0 + c;
            const bool ok = gx >= 0 && gx < w;
            cp_async_f32(drow + c, srow + (ok ? gx : 0), ok);
        }
    }
}

// ---------------------------------------------------------------------------
// Patch distances, per half block (4 columns x 8 rows), vszipcu src/bm3d.cu:282-390.
// Column j: even rows and odd rows accumulate separately, column = e0 + e1; the
// 8 columns join as ((s0+s1)+(s2+s3)) + ((s4+s5)+(s6+s7)): each half returns its
// bracket, the caller adds the two halves.  `st` is the reference patch's
// statistic (mean for zssd/zsad, norm for ssd/norm); `pm` the lane-pair mask.
// ---------------------------------------------------------------------------
__device__ __forceinline__ float colsum8(const float (&n)[8][4], int j) {
    return ((n[0][j] + n[1][j]) + (n[2][j] + n[3][j])) + ((n[4][j] + n[5][j]) + (n[6][j] + n[7][j]));
}

template <int M>
__device__ __forceinline__ float half_distance(const float (&c)[8][4], const float (&n)[8][4], float st, unsigned pm) {
    float s[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    if constexpr (M == M_SSD) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            float d[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) d[i] = c[i][j] - n[i][j];
            float e0 = __fmul_rn(d[0], d[0]);
            float e1 = __fmul_rn(d[1], d[1]);
            e0 = __fmaf_rn(d[2], d[2], e0);
            e1 = __fmaf_rn(d[3], d[3], e1);
            e0 = __fmaf_rn(d[4], d[4], e0);
            e1 = __fmaf_rn(d[5], d[5], e1);
            e0 = __fmaf_rn(d[6], d[6], e0);
            e1 = __fmaf_rn(d[7], d[7], e1);
            s[j] = e0 + e1;
        }
    } else if constexpr (M == M_SAD) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            float e0 = 0.0f, e1 = 0.0f;
#pragma unroll
            for (int i = 0; i < 8; i += 2) {
                e0 += fabsf(c[i][j] - n[i][j]);
                e1 += fabsf(c[i + 1][j] - n[i + 1][j]);
            }
            s[j] = e0 + e1;
        }
    } else if constexpr (M == M_ZSSD || M == M_ZSAD) {
        float hsum = (colsum8(n, 0) + colsum8(n, 1)) + (colsum8(n, 2) + colsum8(n, 3));
        float tot = hsum + __shfl_xor_sync(pm, hsum, 1);
        const float dm = st - tot * (1.0f / 64.f);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            float v[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) v[i] = (c[i][j] - n[i][j]) - dm;
            if constexpr (M == M_ZSSD) {
                float e0 = __fmul_rn(v[0], v[0]);
                float e1 = __fmul_rn(v[1], v[1]);
                e0 = __fmaf_rn(v[2], v[2], e0);
                e1 = __fmaf_rn(v[3], v[3], e1);
                e0 = __fmaf_rn(v[4], v[4], e0);
                e1 = __fmaf_rn(v[5], v[5], e1);
                e0 = __fmaf_rn(v[6], v[6], e0);
                e1 = __fmaf_rn(v[7], v[7], e1);
                s[j] = e0 + e1;
            } else {
                float e0 = 0.0f, e1 = 0.0f;
#pragma unroll
                for (int i = 0; i < 8; i += 2) {
                    e0 += fabsf(v[i]);
                    e1 += fabsf(v[i + 1]);
                }
                s[j] = e0 + e1;
            }
        }
    } else {  // M_SSD_NORM: 2 - 2 <a,b> / (|a| |b| + eps)
        float q[4], x[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            float e0 = __fmul_rn(n[0][j], n[0][j]);
            float e1 = __fmul_rn(n[1][j], n[1][j]);
            float f0 = __fmul_rn(c[0][j], n[0][j]);
            float f1 = __fmul_rn(c[1][j], n[1][j]);
#pragma unroll
            for (int i = 2; i < 8; i += 2) {
                e0 = __fmaf_rn(n[i][j], n[i][j], e0);
                e1 = __fmaf_rn(n[i + 1][j], n[i + 1][j], e1);
                f0 = __fmaf_rn(c[i][j], n[i][j], f0);
                f1 = __fmaf_rn(c[i + 1][j], n[i + 1][j], f1);
            }
            q[j] = e0 + e1;
            x[j] = f0 + f1;
        }
        float hq = (q[0] + q[1]) + (q[2] + q[3]);
        float hx = (x[0] + x[1]) + (x[2] + x[3]);
        float nn = sqrtf(hq + __shfl_xor_sync(pm, hq, 1));
        float dot = hx + __shfl_xor_sync(pm, hx, 1);
        // full distance; the caller's half join is skipped for this metric.  The
        // reference's 2 - 2 dot / (|a| |b| + eps) under fast math is the approximate
        // reciprocal of the denominator with the subtraction fused into it; written out
        // so that no kernel's instruction selection can round it differently
        float r;
        asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(__fmaf_rn(st, nn, ZB_FLT_EPS)));
        return __fmaf_rn(-2.0f * dot, r, 2.0f);
    }
    return (s[0] + s[1]) + (s[2] + s[3]);
}

// Joins the two half distances (pair lanes) into the block distance.
template <int M>
__device__ __forceinline__ float join_pair(float hd, unsigned pm) {
    if constexpr (M == M_SSD_NORM) return hd;
    return hd + __shfl_xor_sync(pm, hd, 1);
}

// Statistic of the reference patch needed by the mean- or norm-based metrics.
template <int M>
__device__ __forceinline__ float ref_stat(const float (&c)[8][4], unsigned pm) {
    if constexpr (M == M_ZSSD || M == M_ZSAD) {
        float h = (colsum8(c, 0) + colsum8(c, 1)) + (colsum8(c, 2) + colsum8(c, 3));
        return (h + __shfl_xor_sync(pm, h, 1)) * (1.0f / 64.f);
    } else if constexpr (M == M_SSD_NORM) {
        float q[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            float e0 = __fmul_rn(c[0][j], c[0][j]);
            float e1 = __fmul_rn(c[1][j], c[1][j]);
#pragma unroll
            for (int i = 2; i < 8; i += 2) {
                e0 = __fmaf_rn(c[i][j], c[i][j], e0);
                e1 = __fmaf_rn(c[i + 1][j], c[i + 1][j], e1);
            }
            q[j] = e0 + e1;
        }
        float h = (q[0] + q[1]) + (q[2] + q[3]);
        return sqrtf(h + __shfl_xor_sync(pm, h, 1));
    }
    return 0.0f;
}

// metrics whose column terms can be shared between neighbouring blocks
template <int M> struct Shareable { static constexpr bool value = (M == M_SSD || M == M_SAD); };

__device__ __forceinline__ float f4c(const float4 &v, int k) {
    return k == 0 ? v.x : k == 1 ? v.y : k == 2 ? v.z : v.w;
}

// ---------------------------------------------------------------------------
// Scan of one rectangular candidate window from global memory by a lane pair
// (row-major, the reference's order).  `plane` is already offset by this
// lane's half (4*hh columns).  A 4-column ring holds the sliding window.
// ---------------------------------------------------------------------------
template <int M, int K = 8>
__device__ __forceinline__ void scan_window(const float *__restrict__ plane, int pitch, int left, int right, int top,
                                            int bottom, const float (&c)[8][4], float st, unsigned pm,
                                            float (&e)[K], int (&q)[K]) {
    for (int row = top; row <= bottom; ++row) {
        const float *rp = plane + (long long)row * pitch;
        float w[8][4];
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) w[i][j] = __ldg(rp + i * pitch + left + j);
        for (int col = left; col <= right; col += 4) {
#pragma unroll
            for (int s = 0; s < 4; ++s) {
                const int cc = col + s;
                if (cc > right) break;
                float n[8][4];
#pragma unroll
                for (int i = 0; i < 8; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j) n[i][j] = w[i][(s + j) & 3];
                const float hd = half_distance<M>(c, n, st, pm);
                const float err = join_pair<M>(hd, pm);
                if (err < e[K - 1]) topk_insert<K>(e, q, err, pack_pos(cc, row));
                if (cc + 1 <= right) {
#pragma unroll
                    for (int i = 0; i < 8; ++i) w[i][s] = __ldg(rp + i * pitch + cc + 4);
                }
            }
        }
    }
}

// The same scan for SSD on packed FP32x2 arithmetic: the ring holds rows (2k, 2k+1) of
// each of its 4 columns as a float2, nc the negated reference half in the same pairs, and
// one __ffma2_rn advances the even-row and the odd-row chain of a column together (each
// with its own rounding), so every distance is half_distance<M_SSD>'s; n + (-c) is
// exactly -(c - n), so the squares are the same.
template <int K = 8>
__device__ __forceinline__ void scan_window_ssd2(const float *__restrict__ plane, int pitch, int left, int right,
                                                 int top, int bottom, const float2 (&nc)[4][4], unsigned pm,
                                                 float (&e)[K], int (&q)[K]) {
    for (int row = top; row <= bottom; ++row) {
        const float *rp = plane + (long long)row * pitch;
        float2 w[4][4];
#pragma unroll
        for (int k = 0; k < 4; ++k)
#pragma unroll
            for (int j = 0; j < 4; ++j)
                w[k][j] = make_float2(__ldg(rp + 2 * k * pitch + left + j), __ldg(rp + (2 * k + 1) * pitch + left + j));
        for (int col = left; col <= right; col += 4) {
#pragma unroll
            for (int s = 0; s < 4; ++s) {
                const int cc = col + s;
                if (cc > right) break;
                float sj[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    float2 d = __fadd2_rn(w[0][(s + j) & 3], nc[0][j]);
                    float2 acc = __fmul2_rn(d, d);
#pragma unroll
                    for (int k = 1; k < 4; ++k) {
                        d = __fadd2_rn(w[k][(s + j) & 3], nc[k][j]);
                        acc = __ffma2_rn(d, d, acc);
                    }
                    sj[j] = acc.x + acc.y;
                }
                const float hd = (sj[0] + sj[1]) + (sj[2] + sj[3]);
                const float err = hd + __shfl_xor_sync(pm, hd, 1);
                if (err < e[K - 1]) topk_insert<K>(e, q, err, pack_pos(cc, row));
                if (cc + 1 <= right) {
#pragma unroll
                    for (int k = 0; k < 4; ++k)
                        w[k][s] = make_float2(__ldg(rp + 2 * k * pitch + cc + 4), __ldg(rp + (2 * k + 1) * pitch + cc + 4));
                }
            }
        }
    }
}

// The negated reference half as row pairs (2k, 2k+1) of each of its 4 columns.
__device__ __forceinline__ void neg_pairs(const float (&c)[8][4], float2 (&nc)[4][4]) {
#pragma unroll
    for (int k = 0; k < 4; ++k)
#pragma unroll
        for (int j = 0; j < 4; ++j) nc[k][j] = make_float2(-c[2 * k][j], -c[2 * k + 1][j]);
}

// One block by a whole warp: the clamped last block column (x = W - 8) that the tiled kernels
// leave out, and every block of small planes at the other block steps.  Its candidate rows are split into 16 consecutive ranges in order, one per lane
// pair, each scanned in the reference's order into a list of its own; the lists are then
// merged in row order, a later range's entries inserted (strict less) after the earlier
// ranges', which is the list of one scan over all the rows.
template <int M>
__device__ __forceinline__ void warp_block(const MatchArgs &a, int kx, int by) {
    const int lane = threadIdx.x & 31;
    const int hh = lane & 1, pr = lane >> 1;
    const int W = a.w, H = a.h, R = a.range;
    const int x = min(a.bs * kx, W - 8), y = min(a.bs * by, H - 8);
    const unsigned pm = 3u << (lane & 30);
    const float *plane = a.frames + (long long)a.radius * a.fstride + 4 * hh;

    float c[8][4];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) c[i][j] = __ldg(plane + (long long)(y + i) * a.pitch + x + j);
    const float st = ref_stat<M>(c, pm);
    float e[8];
    int q[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        e[i] = ZB_FLT_MAX;
        q[i] = 0;
    }
    const int top = max(y - R, 0), bottom = min(y + R, H - 8);
    const int per = (bottom - top + 16) / 16;
    const int r0 = top + pr * per, r1 = min(r0 + per - 1, bottom);
    if (r0 <= r1) {
        if constexpr (M == M_SSD) {
            float2 nc[4][4];
            neg_pairs(c, nc);
            scan_window_ssd2(plane, a.pitch, max(x - R, 0), min(x + R, W - 8), r0, r1, nc, pm, e, q);
        } else {
            scan_window<M>(plane, a.pitch, max(x - R, 0), min(x + R, W - 8), r0, r1, c, st, pm, e, q);
        }
    }
#pragma unroll
    for (int k = 1; k < 16; k <<= 1) {
        float oe[8];
        int oq[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            oe[i] = __shfl_down_sync(kFull, e[i], 2 * k);
            oq[i] = __shfl_down_sync(kFull, q[i], 2 * k);
        }
        if ((pr & (2 * k - 1)) == 0) {
#pragma unroll
            for (int i = 0; i < 8; ++i)
                if (oe[i] < e[7]) top8_insert(e, q, oe[i], oq[i]);
        }
    }
    if (lane != 0) return;
    store_list(a, (long long)by * a.nbx + kx, x, y, e, q);
}

}  // namespace zb
