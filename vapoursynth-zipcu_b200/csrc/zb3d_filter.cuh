// Collaborative filtering with the DCT in both dimensions (vszipcu src/bm3d.cu:392-546) and
// aggregation into signed 64-bit fixed point, 8 lanes per group: device code of zb_filter8
// and of the batch kernel.
//
// A group's 512 values are 64 per lane, and a warp holds 4 groups.  Two layouts, each with
// 32 packed FP32x2 pairs per lane:
//   X  lane x = column x of all 8 patches, all rows: gather and aggregation (8 lanes on
//      consecutive pixels), the vertical transforms, the transform across patches, the
//      shrinkage
//   P  lane p = patch (or spectrum) p, all 8x8 positions: the horizontal transforms
// so the values change lanes four times (X -> P -> X -> P -> X), through shared memory in
// 16-byte accesses and in place: a lane stores where it loaded.  Each instruction of a
// transform does two lines (sm_100 FADD2 / FMUL2 / FFMA2): the vertical transforms pair
// neighbouring patches, the others neighbouring rows.  The last operation of the vertical
// transforms, and the shrinkage, run on the halves one by one and put them into the other
// pairing, which costs no instruction of its own.
//
// What bounds it: the load-store unit's data path (86% of cycles in the Wiener pass): per warp
// 512 wavefronts for the four changes of layout, 256 for the gather (each 8-pixel row of a
// patch is a line of its own), about 190 for the 64-bit reductions; behind it the reductions'
// 32-byte sectors to L2 (69% of that path in the hard threshold).  1920x1080 Y at
// block_step 4, 128,851 groups: hard threshold 176 -> 144 us, 135 -> 69 M instructions;
// Wiener 274 -> 222 us, 188 -> 97 M.  The form before had 16 lanes per group, scalar
// transforms and five changes of layout in 4-byte accesses.
//
// Exactness.  The reference writes a * b + c and leaves the fusing to its compiler.  Here each
// operation is stated, in the form that equals the compiler's on the reference's code shape,
// found by comparing every form on random lines: the forward transform fuses everywhere; the
// inverse joins its two even products (coefficients 0 and 4) in three ways, by what feeds it
// (DctIn).  The 1/4096 of the unnormalised 3D pair is applied with the weight: a power of two
// commutes with the roundings before it.  The 2^32 of the fixed point comes after the extractor,
// whose 2^e may be any float.
#pragma once
#include "zb3d_args.h"
#include "zb3d_match.cuh"

namespace zb {

constexpr int kFilter8Warps = 2;               // warps per CTA: warps do not meet, so CTAs are small
constexpr int kFilterGroups = kFilter8Warps * 4;
constexpr int kPatchStride = 68;               // floats per patch: 17 16-byte units, odd, so that the 8
                                               // lanes of a quarter warp (patches) are on 8 bank quads
constexpr int kOffStride = 18;                 // patch offsets per group (16 used): the 4 groups of a
                                               // warp read theirs on different banks
constexpr int kGroupStride = 8 * kPatchStride + 8;  // = 8 mod 32: the 4 groups' 8-lane rows on 32 banks

// v already scaled by 2^32
__device__ __forceinline__ unsigned long long to_fix(float v) {
    return (unsigned long long)__float2ll_rn(v);
}

// ---------------------------------------------------------------------------
// Packed 8-point DCT pair (gain 4 per axis), two lines at a time.
// ---------------------------------------------------------------------------
__device__ __forceinline__ float2 pk(float v) { return make_float2(v, v); }
__device__ __forceinline__ float2 padd(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 psub(float2 a, float2 b) { return __ffma2_rn(b, pk(-1.0f), a); }  // a - b, one rounding
__device__ __forceinline__ float2 pmul(float k, float2 a) { return __fmul2_rn(pk(k), a); }
__device__ __forceinline__ float2 pfma(float k, float2 a, float2 c) { return __ffma2_rn(pk(k), a, c); }

struct DctK {
    static constexpr float k414 = (float)0.414213562373095048801688724209698078569671875;
    static constexpr float k1847 = (float)1.847759065022573512256366378793576573644833252;
    static constexpr float k198 = (float)0.198912367379658006911597622644676228597850501;
    static constexpr float k1961 = (float)1.961570560806460898252364472268478073947867462;
    static constexpr float k1414 = (float)1.414213562373095048801688724209698078569671875;
    static constexpr float k668 = (float)0.668178637919298919997757686523080761552472251;
    static constexpr float k1662 = (float)1.662939224605090474157576755235811513477121624;
    static constexpr float k707 = (float)0.707106781186547524400844362104849039284835938;
};

// Forward up to the output factors: v[i] becomes output i divided by fwd_factor(i).
__device__ __forceinline__ void dct_fwd_core(float2 (&v)[8]) {
    using K = DctK;
    const float2 d07 = psub(v[0], v[7]), s07 = padd(v[0], v[7]);
    const float2 d43 = psub(v[4], v[3]), s43 = padd(v[4], v[3]);
    const float2 d25 = psub(v[2], v[5]), s25 = padd(v[2], v[5]);
    const float2 d16 = psub(v[1], v[6]), s16 = padd(v[1], v[6]);
    const float2 a = padd(d25, d16), b = psub(d25, d16);
    const float2 p = pfma(-K::k707, a, d07), q = pfma(-K::k707, b, d43);
    const float2 g = pfma(K::k707, a, d07), h = pfma(K::k707, b, d43);
    const float2 e = padd(s07, s43), f = padd(s25, s16);
    const float2 m = psub(s07, s43), n = psub(s25, s16);
    v[0] = padd(e, f);
    v[4] = psub(e, f);
    v[3] = pfma(K::k668, q, p);
    v[5] = pfma(-K::k668, p, q);
    v[1] = pfma(-K::k198, h, g);
    v[7] = pfma(K::k198, g, h);
    v[2] = pfma(-K::k414, n, m);
    v[6] = pfma(K::k414, m, n);
}

__device__ __forceinline__ constexpr float fwd_factor(int i) {
    return i == 0 || i == 4 ? DctK::k1414
           : i == 3         ? DctK::k1662
           : i == 5         ? -DctK::k1662
           : i == 1 || i == 7 ? DctK::k1961
                              : DctK::k1847;
}

// What feeds an inverse transform, which decides how the reference's compiler fuses it.
enum DctIn {
    IN_MOVED,   // values from another lane
    IN_HARD,    // the hard threshold in the same registers
    IN_WIENER,  // the Wiener product in the same registers
};

// Inverse up to its last additions: output i = fma(inv_factor(i), b[i], a[i]).
template <int IN>
__device__ __forceinline__ void dct_inv_core(const float2 (&v)[8], float2 (&a)[4], float2 (&b)[4]) {
    using K = DctK;
    const float2 pc = pmul(K::k1414, v[4]);
    float2 e0, e1;
    if constexpr (IN == IN_HARD) {
        const float2 dc = pmul(K::k1414, v[0]);
        e0 = padd(dc, pc);
        e1 = psub(dc, pc);
    } else {
        e0 = pfma(K::k1414, v[0], pc);
        e1 = __ffma2_rn(pk(K::k1414), v[0], make_float2(-pc.x, -pc.y));
    }
    const float2 o0 = pfma(K::k414, v[6], v[2]);
    const float2 o1 = __ffma2_rn(pk(K::k414), v[2], make_float2(-v[6].x, -v[6].y));
    const float2 s53 = padd(v[5], v[3]), d35 = psub(v[3], v[5]);
    float2 u, t, r, w;
    if constexpr (IN == IN_WIENER) {
        const float2 m1 = pmul(K::k707, s53), m2 = pmul(K::k707, d35);
        u = padd(m1, v[1]);
        t = psub(v[7], m2);
        r = padd(m2, v[7]);
        w = psub(v[1], m1);
    } else {
        u = pfma(K::k707, s53, v[1]);
        t = pfma(-K::k707, d35, v[7]);
        r = pfma(K::k707, d35, v[7]);
        w = pfma(-K::k707, s53, v[1]);
    }
    a[0] = pfma(K::k1847, o0, e0);
    b[0] = pfma(K::k198, r, u);
    a[1] = pfma(-K::k1847, o1, e1);
    b[1] = pfma(K::k668, w, t);
    a[2] = pfma(-K::k1847, o0, e0);
    b[2] = pfma(-K::k198, u, r);
    a[3] = pfma(K::k1847, o1, e1);
    b[3] = pfma(-K::k668, t, w);
}

__device__ __forceinline__ constexpr int inv_pair(int i) {  // which (a, b) output i takes
    return i == 0 || i == 7 ? 0 : i == 2 || i == 5 ? 1 : i == 3 || i == 4 ? 2 : 3;
}

__device__ __forceinline__ constexpr float inv_factor(int i) {
    return i == 0 || i == 4 ? DctK::k1961 : i == 7 || i == 3 ? -DctK::k1961 : i == 2 || i == 1 ? DctK::k1662 : -DctK::k1662;
}

// Transforms of a pair of lines, the result as a pair or as two separate lines.
__device__ __forceinline__ void dct_fwd(float2 (&v)[8]) {
    dct_fwd_core(v);
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = pmul(fwd_factor(i), v[i]);
}

__device__ __forceinline__ void dct_fwd_split(float2 (&v)[8], float (&x)[8], float (&y)[8]) {
    dct_fwd_core(v);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        x[i] = __fmul_rn(fwd_factor(i), v[i].x);
        y[i] = __fmul_rn(fwd_factor(i), v[i].y);
    }
}

__device__ __forceinline__ void dct_inv(float2 (&v)[8]) {
    float2 a[4], b[4];
    dct_inv_core<IN_MOVED>(v, a, b);
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = pfma(inv_factor(i), b[inv_pair(i)], a[inv_pair(i)]);
}

template <int IN>
__device__ __forceinline__ void dct_inv_split(const float2 (&v)[8], float (&x)[8], float (&y)[8]) {
    float2 a[4], b[4];
    dct_inv_core<IN>(v, a, b);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        x[i] = __fmaf_rn(inv_factor(i), b[inv_pair(i)].x, a[inv_pair(i)].x);
        y[i] = __fmaf_rn(inv_factor(i), b[inv_pair(i)].y, a[inv_pair(i)].y);
    }
}

// ---------------------------------------------------------------------------
// Shared-memory positions (floats) of the group's buffer: [patch][column][row], the two
// 16-byte halves of a column swapped for columns 4..7, so that the 8 lanes of a quarter warp
// are on 8 bank quads both as patches and as columns.
// ---------------------------------------------------------------------------
__device__ __forceinline__ float4 lds4(const float *p) { return *reinterpret_cast<const float4 *>(p); }
__device__ __forceinline__ void sts4(float *p, float a, float b, float c, float d) {
    *reinterpret_cast<float4 *>(p) = make_float4(a, b, c, d);
}

// [column][row half] of a patch buffer
__device__ __forceinline__ constexpr int col_off(int x, int half) { return x * 8 + ((half ^ (x >> 2)) << 2); }

// One column of a patch, from layout X.
__device__ __forceinline__ void store_column(float *xb, float *xs, int p, const float (&v)[8]) {
    sts4(xb + p * kPatchStride, v[0], v[1], v[2], v[3]);
    sts4(xs + p * kPatchStride, v[4], v[5], v[6], v[7]);
}

// Layout X, pairs of rows: d[r][p] = rows (2r, 2r + 1) of the lane's column of patch p.
__device__ __forceinline__ void load_x(const float *xb, const float *xs, float2 (&d)[4][8]) {
#pragma unroll
    for (int p = 0; p < 8; ++p) {
        const float4 lo = lds4(xb + p * kPatchStride), hi = lds4(xs + p * kPatchStride);
        d[0][p] = make_float2(lo.x, lo.y);
        d[1][p] = make_float2(lo.z, lo.w);
        d[2][p] = make_float2(hi.x, hi.y);
        d[3][p] = make_float2(hi.z, hi.w);
    }
}

// The horizontal transform in layout P, in place.
template <bool INV>
__device__ __forceinline__ void horizontal(float *patch) {
    float2 h[4][8];  // [row pair][column]
#pragma unroll
    for (int x = 0; x < 8; ++x) {
        const float4 lo = lds4(patch + col_off(x, 0)), hi = lds4(patch + col_off(x, 1));
        h[0][x] = make_float2(lo.x, lo.y);
        h[1][x] = make_float2(lo.z, lo.w);
        h[2][x] = make_float2(hi.x, hi.y);
        h[3][x] = make_float2(hi.z, hi.w);
    }
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        if constexpr (INV) dct_inv(h[r]);
        else dct_fwd(h[r]);
    }
#pragma unroll
    for (int x = 0; x < 8; ++x) {
        sts4(patch + col_off(x, 0), h[0][x].x, h[0][x].y, h[1][x].x, h[1][x].y);
        sts4(patch + col_off(x, 1), h[2][x].x, h[2][x].y, h[3][x].x, h[3][x].y);
    }
}

// Gather of the group's 8 patches of one plane (8 lanes read 8 consecutive pixels; off: the
// patches' offsets) and their 3D transform into d.
__device__ __forceinline__ void forward8(const float *plane, const long long *off, int pitch, float *xb, float *xs,
                                         float *patch, float2 (&d)[4][8]) {
#pragma unroll
    for (int pp = 0; pp < 4; ++pp) {
        const float *s0 = plane + off[2 * pp], *s1 = plane + off[2 * pp + 1];
#pragma unroll
        for (int y = 0; y < 8; ++y) {
            // d is free until the transform across patches: it holds the gathered pixels
            d[pp][y] = make_float2(__ldg(s0 + (long long)y * pitch), __ldg(s1 + (long long)y * pitch));
        }
    }
#pragma unroll
    for (int pp = 0; pp < 4; ++pp) {
        float a[8], b[8];
        dct_fwd_split(d[pp], a, b);
        store_column(xb, xs, 2 * pp, a);
        store_column(xb, xs, 2 * pp + 1, b);
    }
    __syncwarp();
    horizontal<false>(patch);
    __syncwarp();
    load_x(xb, xs, d);
#pragma unroll
    for (int r = 0; r < 4; ++r) dct_fwd(d[r]);
}

// Groups g0 + threadIdx.x / 8 of one entry.  sbuf: kFilterGroups * kGroupStride floats, cbuf
// (Wiener): the same again, offs: kFilterGroups * kOffStride.
template <bool FINAL>
__device__ __forceinline__ void filter8_groups(const FilterArgs &a, long long g0, float *sbuf, float *cbuf,
                                               long long *offs) {
    const int l8 = threadIdx.x & 7;
    const int gi = threadIdx.x >> 3;
    const bool live = g0 + gi < a.nblocks;
    const long long grp = live ? g0 + gi : a.nblocks - 1;  // the warp stays whole
    float *gb = sbuf + gi * kGroupStride;
    float *patch = gb + l8 * kPatchStride;                       // layout P
    float *xb = gb + col_off(l8, 0), *xs = gb + col_off(l8, 1);  // layout X, the two row halves
    long long *off = offs + gi * kOffStride;
    const float E = a.extractor;
    __syncwarp();  // a caller's previous groups: their offsets have been read
    {
        const int2 v = a.list[grp * 8 + l8];
        const long long z = (unsigned)v.y >> 24, yx = (long long)(v.y & 0xffffff) * a.pitch + v.x;
        off[l8] = z * a.frame_stride + yx;
        off[8 + l8] = z * a.acc_frame_stride + yx;
    }
    __syncwarp();

    for (int pl = 0; pl < a.nplanes; ++pl) {
        const float sigma = pl == 0 ? a.sigma[0] : (pl == 1 ? a.sigma[1] : a.sigma[2]);
        if (a.chroma && sigma < ZB_FLT_EPS) continue;
        float k = 0.0f;
        float2 d[4][8];
        float *cx = cbuf + gi * kGroupStride + col_off(l8, 0), *cs = cbuf + gi * kGroupStride + col_off(l8, 1);
        if constexpr (FINAL) {
            // Wiener coefficients r^2 / (r^2 + sigma^2) of the basic estimate's spectrum (the
            // reference rounds r^2 once and adds sigma^2 without FMA), and the weight's sum of
            // their squares by FMA over spectrum and row of the lane's column, in the
            // reference's order
            forward8(a.src + pl * a.plane_stride + l8, off, a.pitch, xb, xs, patch, d);
            const float s2 = sigma * sigma;
#pragma unroll
            for (int p = 0; p < 8; ++p) {
                float c[8];
#pragma unroll
                for (int r = 0; r < 4; ++r) {
                    const float2 r2 = __fmul2_rn(d[r][p], d[r][p]);
                    c[2 * r] = r2.x / __fadd_rn(r2.x, s2);
                    c[2 * r + 1] = r2.y / __fadd_rn(r2.y, s2);
                    if (p == 0 && r == 0 && l8 == 0) c[0] = 1.0f;
                    k = __fmaf_rn(c[2 * r], c[2 * r], k);
                    k = __fmaf_rn(c[2 * r + 1], c[2 * r + 1], k);
                }
                store_column(cx, cs, p, c);  // read back by this lane alone
            }
        }
        forward8(a.src + (FINAL ? a.clip_stride : 0) + pl * a.plane_stride + l8, off, a.pitch, xb, xs, patch, d);
        // the shrinkage, from pairs of rows into pairs of patches, and the vertical inverse
        int kept = 0;
#pragma unroll
        for (int pp = 0; pp < 4; ++pp) {
            float2 v[8];
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                const float2 p0 = d[2 * half][2 * pp], p1 = d[2 * half + 1][2 * pp];
                const float2 q0 = d[2 * half][2 * pp + 1], q1 = d[2 * half + 1][2 * pp + 1];
                const float s0[4] = {p0.x, p0.y, p1.x, p1.y}, s1[4] = {q0.x, q0.y, q1.x, q1.y};
                if constexpr (FINAL) {
                    const float4 c0 = lds4((half ? cs : cx) + 2 * pp * kPatchStride);
                    const float4 c1 = lds4((half ? cs : cx) + (2 * pp + 1) * kPatchStride);
                    v[4 * half + 0] = make_float2(s0[0] * c0.x, s1[0] * c1.x);
                    v[4 * half + 1] = make_float2(s0[1] * c0.y, s1[1] * c1.y);
                    v[4 * half + 2] = make_float2(s0[2] * c0.z, s1[2] * c1.z);
                    v[4 * half + 3] = make_float2(s0[3] * c0.w, s1[3] * c1.w);
                } else {
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const float thr = (pp == 0 && half == 0 && i == 0 && l8 == 0) ? 0.0f : sigma;
                        const bool k0 = fabsf(s0[i]) >= thr, k1 = fabsf(s1[i]) >= sigma;
                        kept += k0;
                        kept += k1;
                        v[4 * half + i] = make_float2(k0 ? s0[i] : 0.0f, k1 ? s1[i] : 0.0f);
                    }
                }
            }
            float x[8], y[8];
            dct_inv_split<FINAL ? IN_WIENER : IN_HARD>(v, x, y);
            store_column(xb, xs, 2 * pp, x);
            store_column(xb, xs, 2 * pp + 1, y);
        }
        if constexpr (!FINAL) k = (float)kept;  // at most 512 in all: exact in any order
        k += __shfl_xor_sync(kFull, k, 1);
        k += __shfl_xor_sync(kFull, k, 2);
        k += __shfl_xor_sync(kFull, k, 4);
        const float w = 1.0f / k;
        const float ws = w * (1.0f / 4096.0f);
        __syncwarp();
        horizontal<true>(patch);
        __syncwarp();
        load_x(xb, xs, d);
#pragma unroll
        for (int r = 0; r < 4; ++r) dct_inv(d[r]);
        if (!live) continue;

        unsigned long long *num = a.num + pl * a.acc_plane_stride + l8;
#pragma unroll
        for (int p = 0; p < 8; ++p) {
            unsigned long long *q = num + off[8 + p];
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const float2 v = pmul(kFixScale, __fadd2_rn(__ffma2_rn(pk(ws), d[r][p], pk(E)), pk(-E)));
                atomicAdd(q, to_fix(v.x));
                q += a.pitch;
                atomicAdd(q, to_fix(v.y));
                q += a.pitch;
            }
        }
        // lane p books the weight of patch p once, at its origin
        const float wq = (w + E) - E;
        atomicAdd(a.den + pl * a.acc_plane_stride + off[8 + l8], to_fix(wq * kFixScale));
    }
}

}  // namespace zb
