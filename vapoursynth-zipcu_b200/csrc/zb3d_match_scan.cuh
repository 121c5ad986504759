// Spatial SSD / SAD matching of one shared-memory tile, used by the per-plane kernel
// (zb3d_match.cu) and by the batch kernel (zb3d_kernels.cu).
//
// A CTA has a warp per block row (candidates inserted into the lists at once), or kScanWarps
// warps: rows_per_cta block rows times `split` ranges of candidate rows (candidates queued).  A
// warp covers one row of reference blocks and one of the ranges; lane k's half
// block starts at tile column 4k (SHARED, block_step 4: block k = lanes k, k+1) or, in
// pair mode (block_step 8), block b = lanes 2b, 2b+1.
//
// The tile is stored twice with candidate rows interleaved in pairs, once with pairs
// starting at even tile rows and once at odd ones; a float2 then holds rows (2k, 2k+1) of
// one column of a window, exactly the operands of the even- and odd-row partial sums,
// which advance together on packed FP32x2 (sm_100 FADD2 / FMUL2 / FFMA2):
// acc = fma2(d, d, acc) computes the reference's e0 and e1 chains in one instruction and
// acc.x + acc.y is their join.  d = n + (-c) = -(c - n) exactly, so d*d is the reference's
// square.  A pair row holds the tile's columns as 16-byte chunks of two columns
// each, in two half-planes of g chunks: columns 4u, 4u+1 form chunk u of the first,
// columns 4u+2, 4u+3 chunk u of the second.  A lane's block half starts at a column
// that is a multiple of 4, so at every step the lanes of a quarter warp read eight
// consecutive chunks of one half-plane (float4 loads free of bank conflicts), and a
// lane's address advances by one chunk per step.  With g fixed at compile time (kTile2G,
// bm_range <= 15) every other offset is an immediate.
//
// What bounds it: the FMA pipe, 72 cycles of it per warp and candidate (16 subtractions and 16
// multiply-adds of two cycles each, and the joins); with queues 73% of active cycles at 1920x1080,
// block_step 4, bm_range 12, whose 544 CTAs are 1.84 waves.  The queues' 32 KB decide how many
// CTAs share an SM, so where that costs more than they save candidates are inserted at once:
// 1080p us at block_step 4 / 8, inserted at once and queued (8 rows, ssd, a noisy plane of
// gradients): bm_range 9 174 / 97 and 185 / 119, bm_range 12 275 / 149 and 284 / 175, bm_range 24
// 1184 / 601 and 1049 / 544; 326 before the column stream (block_step 4, bm_range 12, textured
// plane; 291 now, queued).  Small planes take queues for their ranges of candidate rows: 320x240
// at block_step 4, bm_range 12: 92 at once, 40 with 8 ranges.  scan_shape (zb3d_match.cu) has the
// rule, and the autotuner times both.
#pragma once
#include "zb3d_match.cuh"

namespace zb {

constexpr int kScanWarps = 8;  // 2 CTAs of 8 warps fit the register file at 128 registers
constexpr int kTile2G = 40;    // half-plane chunks of the fixed layout (tile pitch <= 160)

__host__ __device__ constexpr int tile2_g(int tile_pitch, bool fixed) {  // chunks per half-plane
    return fixed ? kTile2G : tile_pitch / 4;
}

__host__ __device__ constexpr bool tile2_fixed(int chunks) { return chunks <= (4 * kTile2G - 128) / 4; }

// float offset of column `col` in a pair row of half-plane size g
__device__ __forceinline__ int split_off(int col, int g) { return ((col >> 1) & 1) * 4 * g + 4 * (col >> 2) + 2 * (col & 1); }

__device__ __forceinline__ float2 f4lo(const float4 &v) { return make_float2(v.x, v.y); }
__device__ __forceinline__ float2 f4hi(const float4 &v) { return make_float2(v.z, v.w); }

// ---------------------------------------------------------------------------
// Pending candidates (QUEUE).  A candidate below the list's last error is not inserted at once:
// the lane appends it to its own queue in shared memory, and the warp drains all its queues
// together when one of them could overflow, and at the end.  With immediate insertion a
// warp ran the 38-instruction insertion at about 380 of the 625 candidates of bm_range 12,
// because one of its 31 blocks wanted it; drained in bulk it runs about 110 times.  A
// queue keeps scan order and the insertion still tests each entry against the list
// (strict less), so the list is the one of immediate insertion.  Slot i of lane l is at
// 256 i + 8 l bytes: whatever slots the lanes are at, a half warp touches 32 banks.
// ---------------------------------------------------------------------------
constexpr int kPend = 16;                       // slots per lane
constexpr int kPendBytes = kPend * 32 * 8;      // per warp
constexpr int kPendFull = (kPend - 8) * 256;    // two steps append at most 8

__device__ __forceinline__ void pend_store(unsigned at, float err, int pos) {
    asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(at), "f"(err), "r"(pos) : "memory");
}

__device__ __forceinline__ void pend_load(unsigned at, float &err, int &pos) {
    asm volatile("ld.shared.v2.b32 {%0, %1}, [%2];" : "=f"(err), "=r"(pos) : "r"(at) : "memory");
}

// Strict-less insertion without a branch: an error that is not below e[7] changes nothing.
__device__ __forceinline__ void top8_insert_always(float (&e)[8], int (&q)[8], float err, int pos) {
#pragma unroll
    for (int i = 7; i > 0; --i) {
        const bool ci = err < e[i];
        const bool cp = err < e[i - 1];
        q[i] = cp ? q[i - 1] : (ci ? pos : q[i]);
        e[i] = fminf(e[i], fmaxf(e[i - 1], err));
    }
    q[0] = err < e[0] ? pos : q[0];
    e[0] = fminf(e[0], err);
}

// Inserts every lane's entries in [base, end) and empties the queues.
__device__ __forceinline__ void pend_drain(unsigned base, unsigned &end, float (&e)[8], int (&q)[8]) {
    unsigned at = base;
    while (__any_sync(kFull, at < end)) {
        float err = ZB_FLT_MAX;  // not below any list entry
        int pos = 0;
        if (at < end) pend_load(at, err, pos);
        at += 256;
        top8_insert_always(e, q, err, pos);
    }
    end = base;
}

// ---------------------------------------------------------------------------
// One step of a candidate row: tile columns 4m .. 4m + 3 of the lane (pc points at the
// first).  Every column is loaded once, as rows (2k, 2k+1) pairs, and feeds the four chains
// (displacement s = col - j, column j of the half block); a chain runs over its pair rows
// in order, so every sum is the reference's.  Displacement 4m + c - 3 is complete after
// column 4m + c: err[c] = (s0 + s1) + (s2 + s3).  st carries the unfinished sums of the
// next three displacements.  FIRST: no displacement below 0; SMAX: the largest
// displacement of the row relative to 4m (3: all), chains beyond it are left out.
// Against chunks of 4 displacements that reload the columns they share this halves the
// shared-memory reads, and the row's ends no longer compute displacements outside
// [-R, R] (28 for 25 at bm_range 12).
// ---------------------------------------------------------------------------
template <int M, int GF, bool FIRST, int SMAX>
__device__ __forceinline__ void scan_step(const float *pc, int pp_rt, int g_rt, const float2 (&nc)[4][4],
                                          float (&st)[4], float (&err)[4]) {
    const int pp = GF ? 8 * GF : pp_rt, g = GF ? GF : g_rt;
    float s0[7], s01[7], s2[7];  // by displacement - 4m + 3
    if constexpr (!FIRST) {
        s01[0] = st[0];
        s2[0] = st[1];
        s01[1] = st[2];
        s0[2] = st[3];
    }
#pragma unroll
    for (int p = 0; p < 2; ++p) {
        if (2 * p - 3 > SMAX) continue;
        float4 v[4];  // columns (2p, 2p + 1) of pair rows k: (row 2k, row 2k + 1) of each
#pragma unroll
        for (int k = 0; k < 4; ++k) v[k] = *reinterpret_cast<const float4 *>(pc + k * pp + p * 4 * g);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int col = 2 * p + h;
#pragma unroll
            for (int j = 3; j >= 0; --j) {
                const int r = col - j;
                if ((FIRST && r < 0) || r > SMAX) continue;
                float2 d = __fadd2_rn(h ? f4hi(v[0]) : f4lo(v[0]), nc[0][j]);
                float s;
                if constexpr (M == M_SSD) {
                    float2 acc = __fmul2_rn(d, d);
#pragma unroll
                    for (int k = 1; k < 4; ++k) {
                        d = __fadd2_rn(h ? f4hi(v[k]) : f4lo(v[k]), nc[k][j]);
                        acc = __ffma2_rn(d, d, acc);
                    }
                    s = acc.x + acc.y;
                } else {  // SAD
                    float e0 = fabsf(d.x), e1 = fabsf(d.y);
#pragma unroll
                    for (int k = 1; k < 4; ++k) {
                        d = __fadd2_rn(h ? f4hi(v[k]) : f4lo(v[k]), nc[k][j]);
                        e0 += fabsf(d.x);
                        e1 += fabsf(d.y);
                    }
                    s = e0 + e1;
                }
                if (j == 0) s0[r + 3] = s;
                if (j == 1) s01[r + 3] = s0[r + 3] + s;
                if (j == 2) s2[r + 3] = s;
                if (j == 3) err[col] = s01[r + 3] + (s2[r + 3] + s);
            }
        }
    }
    if constexpr (SMAX == 3) {
        st[0] = s01[4];
        st[1] = s2[4];
        st[2] = s01[5];
        st[3] = s0[6];
    }
}

// Displacement at `pos` of the joined error err: queued, or inserted at once, where it is below
// the list's last error.
template <bool QUEUE>
__device__ __forceinline__ void scan_take(float err, int pos, unsigned &end, float (&e)[8], int (&q)[8]) {
    if (err < e[7]) {
        if constexpr (QUEUE) {
            pend_store(end, err, pos);
            end += 256;
        } else {
            top8_insert(e, q, err, pos);
        }
    }
}

template <bool QUEUE>
__device__ __forceinline__ void scan_vote(unsigned base, unsigned &end, float (&e)[8], int (&q)[8]) {
    if constexpr (QUEUE)
        if (__any_sync(kFull, end > base + kPendFull)) pend_drain(base, end, e, q);
}

// The step, then its finished displacements C0 .. C1 - 1 joined with the other half block
// and taken.  pos: packed position of displacement 4m - 3.
template <int M, bool SHARED, int GF, bool QUEUE, bool FIRST, int SMAX, int C0, int C1>
__device__ __forceinline__ void scan_step_append(const float *pc, int pp, int g, const float2 (&nc)[4][4],
                                                 float (&st)[4], int pos, unsigned base, unsigned &end, float (&e)[8],
                                                 int (&q)[8]) {
    float err[4];
    scan_step<M, GF, FIRST, SMAX>(pc, pp, g, nc, st, err);
#pragma unroll
    for (int c = C0; c < C1; ++c)
        err[c] += SHARED ? __shfl_down_sync(kFull, err[c], 1) : __shfl_xor_sync(kFull, err[c], 1);
#pragma unroll
    for (int c = C0; c < C1; ++c) scan_take<QUEUE>(err[c], pos + c, end, e, q);
    scan_vote<QUEUE>(base, end, e, q);
}

// Two whole steps with one vote.
template <int M, bool SHARED, int GF, bool QUEUE>
__device__ __forceinline__ void scan_two_steps(const float *pc, int pp, int g, const float2 (&nc)[4][4],
                                               float (&st)[4], int pos, unsigned base, unsigned &end, float (&e)[8],
                                               int (&q)[8]) {
    float err[2][4];
    scan_step<M, GF, false, 3>(pc, pp, g, nc, st, err[0]);
    scan_step<M, GF, false, 3>(pc + 4, pp, g, nc, st, err[1]);
#pragma unroll
    for (int c = 0; c < 8; ++c)
        err[c >> 2][c & 3] += SHARED ? __shfl_down_sync(kFull, err[c >> 2][c & 3], 1) : __shfl_xor_sync(kFull, err[c >> 2][c & 3], 1);
#pragma unroll
    for (int c = 0; c < 8; ++c) scan_take<QUEUE>(err[c >> 2][c & 3], pos + c, end, e, q);
    scan_vote<QUEUE>(base, end, e, q);
}

// Bytes of dynamic shared memory: the two copies of the tile, then the queues (none where
// candidates are inserted at once).
inline size_t scan_tile_bytes(const MatchArgs &a, int rows_per_cta) {
    return (size_t)((rows_per_cta - 1) * a.bs + 2 * a.range + 8) * 8 * tile2_g(a.tile_pitch, tile2_fixed(a.chunks)) *
           sizeof(float);
}

inline size_t scan_smem_bytes(const MatchJob &a, int rows_per_cta) {
    return scan_tile_bytes(a, rows_per_cta) + (a.direct ? 0 : (size_t)kScanWarps * kPendBytes);
}

// CTA `part` of `parts` clears its share of the accumulators (16-byte stores; the arrays start
// on 16 bytes).
__device__ __forceinline__ void zero_slice(const ZeroArgs &zero, int part, int parts) {
    if (!zero.acc[0]) return;
    const long long pairs = zero.count / 2, per = (pairs + parts - 1) / parts;
    const long long first = per * part, last = min(first + per, pairs);
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        ulonglong2 *z = reinterpret_cast<ulonglong2 *>(zero.acc[k]);
        for (long long i = first + threadIdx.x; i < last; i += blockDim.x) z[i] = make_ulonglong2(0, 0);
        if (part == 0 && threadIdx.x == 0 && (zero.count & 1)) zero.acc[k][zero.count - 1] = 0;
    }
}

// Tiles per row of an entry: 31 (SHARED) or 16 unclamped block columns each.
inline int scan_tiles_x(const MatchArgs &a) {
    const int nbw = a.bs == 4 ? 31 : 16;
    return (a.nbx_al + nbw - 1) / nbw;
}

// One tile: block columns [31 bx, 31 bx + 31) (SHARED) or [16 bx, ...), block rows
// [rows by, rows by + rows); `tile` is the dynamic shared memory (scan_smem_bytes).
// QUEUE: kScanWarps warps, split = kScanWarps / rows ranges of candidate rows per block row:
// with fewer rows per CTA a plane gives more CTAs, which is what fills the GPU for small planes.
// The ranges' lists are merged in row order at the end, a later range's entries inserted
// (strict less) after the earlier ranges', which is the list of one scan.  Else: a warp per block
// row, no queues and no ranges.
template <int M, bool SHARED, int BS, bool FIXED, bool QUEUE>
__device__ __forceinline__ void scan_tile_g(const MatchArgs &a, int bx, int by_cta, int rows, float *tile) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    constexpr int NBW = SHARED ? 31 : 16;
    constexpr int GF = FIXED ? kTile2G : 0;
    const int warps = QUEUE ? kScanWarps : rows, split = QUEUE ? kScanWarps / rows : 1;
    const int R = a.range, W = a.w, H = a.h, tp = a.tile_pitch;
    const int g = tile2_g(tp, FIXED), pp = 8 * g;
    const int kx0 = bx * NBW;
    const int x0 = kx0 * BS;
    const int by0 = by_cta * rows;
    const int by_last = min(by0 + rows - 1, a.nby - 1);
    const int y_first = min(BS * by0, H - 8);
    const int y_last = min(BS * by_last, H - 8);
    const int r0 = max(y_first - R, 0);
    const int nrows = min(y_last + R, H - 8) + 8 - r0;
    const int npe = (nrows + 1) >> 1;  // even-start pair rows
    float *tE = tile;
    float *tO = tile + npe * pp;
    const float *plane = a.frames + (long long)a.radius * a.fstride;
    {
        // columns outside the image are +inf: every candidate that touches one has an
        // infinite (or NaN) distance and never enters a list, so the scan needs no bounds tests
        const int gx0 = x0 - R;
        for (int t = warp; t < nrows; t += warps) {
            const float *srow = plane + (long long)(r0 + t) * a.pitch;
            float *de = tE + (t >> 1) * pp + (t & 1);
            float *dq = t > 0 ? tO + ((t - 1) >> 1) * pp + ((t - 1) & 1) : nullptr;
            for (int c = lane; c < tp; c += 32) {
                const int gx = gx0 + c;
                const int so = split_off(c, g);
                if (gx >= 0 && gx < W) {
                    cp_async_f32(de + so, srow + gx, true);
                    if (dq) cp_async_f32(dq + so, srow + gx, true);
                } else {
                    de[so] = __int_as_float(0x7f800000);
                    if (dq) dq[so] = __int_as_float(0x7f800000);
                }
            }
        }
    }
    cp_async_wait_all();
    __syncthreads();

    const int sp = warp / rows;                       // range of candidate rows
    const int by = by0 + (warp - sp * rows);
    const bool work = by < a.nby;
    const int y = min(BS * min(by, a.nby - 1), H - 8);
    const int b = SHARED ? lane : (lane >> 1);
    const int hh = SHARED ? 0 : (lane & 1);
    const int kx = kx0 + b;
    const int xb = BS * kx;
    const int uo = BS * b + 4 * hh;  // tile column of this half at dx = -R (a multiple of 4)
    const bool blk = (SHARED ? lane < 31 : true) && kx < a.nbx_al;

    float e[8];
    int q[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        e[i] = blk ? ZB_FLT_MAX : -1.0f;  // helper lanes take no candidate
        q[i] = 0;
    }
    const unsigned base = (unsigned)__cvta_generic_to_shared(tile) +
                          (unsigned)(((rows - 1) * BS + 2 * R + 8) * 8 * g * 4 + warp * kPendBytes + lane * 8);
    unsigned end = base;
    if (work) {
        // negated reference half as row pairs (2k, 2k+1) of each of its 4 columns
        float2 nc[4][4];
        {
            const int t0 = y - r0;
            const float *ref = (t0 & 1) ? tO + ((t0 - 1) >> 1) * pp : tE + (t0 >> 1) * pp;
#pragma unroll
            for (int k = 0; k < 4; ++k)
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float2 v = *reinterpret_cast<const float2 *>(ref + k * pp + split_off(uo + R + j, g));
                    nc[k][j] = make_float2(-v.x, -v.y);
                }
        }
        int top = max(y - R, 0), bottom = min(y + R, H - 8);
        const int per = (bottom - top + split) / split;
        top += sp * per;
        bottom = min(bottom, top + per - 1);
        for (int row = top; row <= bottom; ++row) {
            const int t0 = row - r0;
            const float *pc = ((t0 & 1) ? tO + ((t0 - 1) >> 1) * pp : tE + (t0 >> 1) * pp) + uo;
            int pos = pack_pos(0, row) + (xb - R - 3);
            float st[4];
            scan_step_append<M, SHARED, GF, QUEUE, true, 3, 3, 4>(pc, pp, g, nc, st, pos, base, end, e, q);
            int m = 1;
            for (; m + 1 < (R + 1) / 2; m += 2) {
                scan_two_steps<M, SHARED, GF, QUEUE>(pc + 4, pp, g, nc, st, pos + 4, base, end, e, q);
                pc += 8;
                pos += 8;
            }
            if (m < (R + 1) / 2) {
                pc += 4;
                pos += 4;
                scan_step_append<M, SHARED, GF, QUEUE, false, 3, 0, 4>(pc, pp, g, nc, st, pos, base, end, e, q);
            }
            // displacement 2R is the first of its step (R even) or the last of the step before
            if (R & 1)
                scan_step_append<M, SHARED, GF, QUEUE, false, -2, 0, 2>(pc + 4, pp, g, nc, st, pos + 4, base, end, e, q);
            else
                scan_step_append<M, SHARED, GF, QUEUE, false, 0, 0, 4>(pc + 4, pp, g, nc, st, pos + 4, base, end, e, q);
        }
        if constexpr (QUEUE) pend_drain(base, end, e, q);
    }
    // merge of the ranges, in order: range sp takes the list of range sp + k
    for (int k = 1; k < split; k <<= 1) {
        if ((sp & (2 * k - 1)) == k) {
#pragma unroll
            for (int i = 0; i < 8; ++i) pend_store(base + 256 * i, e[i], q[i]);
        }
        __syncthreads();
        if ((sp & (2 * k - 1)) == 0) {
            const unsigned other = base + k * rows * kPendBytes;
#pragma unroll 1
            for (int i = 0; i < 8; ++i) {
                float err;
                int pos;
                pend_load(other + 256 * i, err, pos);
                if (!__any_sync(kFull, err < e[7])) break;  // the rest of that list is no smaller
                top8_insert_always(e, q, err, pos);
            }
        }
    }
    if (!work || sp != 0 || !blk || (!SHARED && hh)) return;
    store_list(a, (long long)by * a.nbx + kx, xb, y, e, q);
}

// The tile with the fixed half-plane size where the displacements allow it.
template <int M, bool SHARED, int BS, bool QUEUE>
__device__ __forceinline__ void scan_tile(const MatchArgs &a, int bx, int by_cta, int rows, float *tile) {
    if (tile2_fixed(a.chunks))
        scan_tile_g<M, SHARED, BS, true, QUEUE>(a, bx, by_cta, rows, tile);
    else
        scan_tile_g<M, SHARED, BS, false, QUEUE>(a, bx, by_cta, rows, tile);
}

}  // namespace zb
