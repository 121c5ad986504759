// Spatial SSD matching of one shared-memory tile, used by the per-plane kernel (zb3d_match.cu)
// and by the batch kernel (zb3d_kernels.cu).
#pragma once
#include "zb3d_match.cuh"

namespace zb {

// ---------------------------------------------------------------------------
// SSD matching with packed FP32x2 arithmetic (sm_100 FADD2 / FMUL2 / FFMA2).
// The tile is stored twice with candidate rows interleaved in pairs, once with
// pairs starting at even tile rows and once at odd ones; a float2 then holds
// rows (2k, 2k+1) of one column of a window, exactly the operands of the even-
// and odd-row partial sums, which advance together: acc = fma2(d, d, acc)
// computes the reference's e0 and e1 chains in one instruction and acc.x + acc.y
// is their join.  d = n + (-c) = -(c - n) exactly, so d*d is the reference's
// square.  A pair row holds the tile's columns as 16-byte chunks of two columns
// each, in two half-planes of g chunks: columns 4u, 4u+1 form chunk u of the first,
// columns 4u+2, 4u+3 chunk u of the second.  A lane's block half starts at a column
// that is a multiple of 4, so at every step the lanes of a quarter warp read eight
// consecutive chunks of one half-plane (float4 loads free of bank conflicts), and a
// lane's address advances by one chunk per displacement chunk.  With g fixed at
// compile time (kTile2G, for up to 8 chunks of displacements: bm_range <= 15) every
// other offset is an immediate.
// ---------------------------------------------------------------------------
constexpr int kTile2G = 40;  // half-plane chunks of the fixed layout (tile pitch <= 160)

__host__ __device__ constexpr int tile2_g(int tile_pitch, bool fixed) {  // chunks per half-plane
    return fixed ? kTile2G : tile_pitch / 4;
}

__host__ __device__ constexpr bool tile2_fixed(int chunks) { return chunks <= (4 * kTile2G - 128) / 4; }

// float offset of column `col` in a pair row of half-plane size g
__device__ __forceinline__ int split_off(int col, int g) { return ((col >> 1) & 1) * 4 * g + 4 * (col >> 2) + 2 * (col & 1); }

__device__ __forceinline__ float2 f4lo(const float4 &v) { return make_float2(v.x, v.y); }
__device__ __forceinline__ float2 f4hi(const float4 &v) { return make_float2(v.z, v.w); }

// One chunk: displacements dx = -R + 4m + s (s = 0..3) of candidate row `row`.  The
// chunk reads window columns c0 .. c0 + 6 (c0 = the lane's tile column at dx = -R, plus
// 4m; a multiple of 4) of the four pair rows; pc points at column c0 of the first pair
// row.  GF: half-plane chunks when fixed at compile time, else 0 (pp_rt and g_rt give
// the pitch and half-plane size).  The columns are loaded one column pair at a time, just
// before the sums that use them: column col feeds the (s, j = col - s) chains, each
// of which runs over its pair rows k = 0..3 in order, so every sum is the reference's.
// Keeping no window in registers holds the kernel at 112-116 registers.  The four distances
// come first (no branch between their FMA chains), then the insertions in scan order;
// a displacement past R is computed from the tile's padding columns and discarded.
template <bool SHARED, int GF>
__device__ __forceinline__ void tiled2_chunk(const float *pc, int pp_rt, int g_rt, int m, int R, int row, int xb,
                                             int lo, int hi, const float2 (&nc)[4][4], float (&e)[8], int (&q)[8]) {
    const int pp = GF ? 8 * GF : pp_rt, g = GF ? GF : g_rt;
    float sj[4][4];
#pragma unroll
    for (int p = 0; p < 4; ++p) {
        float4 v[4];  // columns (2p, 2p + 1) of pair rows k: (row 2k, row 2k + 1) of each
#pragma unroll
        for (int k = 0; k < 4; ++k)
            v[k] = *reinterpret_cast<const float4 *>(pc + k * pp + (p & 1) * 4 * g + 4 * (p >> 1));
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int col = 2 * p + h;
#pragma unroll
            for (int s = 0; s < 4; ++s) {
                const int j = col - s;
                if (j < 0 || j > 3) continue;
                float2 d = __fadd2_rn(h ? f4hi(v[0]) : f4lo(v[0]), nc[0][j]);
                float2 acc = __fmul2_rn(d, d);
#pragma unroll
                for (int k = 1; k < 4; ++k) {
                    d = __fadd2_rn(h ? f4hi(v[k]) : f4lo(v[k]), nc[k][j]);
                    acc = __ffma2_rn(d, d, acc);
                }
                sj[s][j] = acc.x + acc.y;
            }
        }
    }
    float err[4];
#pragma unroll
    for (int s = 0; s < 4; ++s) err[s] = (sj[s][0] + sj[s][1]) + (sj[s][2] + sj[s][3]);
#pragma unroll
    for (int s = 0; s < 4; ++s) {
        if constexpr (SHARED)
            err[s] += __shfl_down_sync(kFull, err[s], 1);
        else
            err[s] += __shfl_xor_sync(kFull, err[s], 1);
    }
#pragma unroll
    for (int s = 0; s < 4; ++s) {
        const int dx = -R + 4 * m + s;
        if (dx <= R && dx >= lo && dx <= hi && err[s] < e[7]) top8_insert(e, q, err[s], pack_pos(xb + dx, row));
    }
}

// One tile of the packed FP32x2 SSD matcher: block columns [31 bx, 31 bx + 31) (SHARED)
// or [16 bx, ...), block rows [nw by, nw by + nw), nw = the CTA's warps; `tile` is the
// dynamic shared-memory tile (match_tile2_bytes).
template <bool SHARED, int BS, bool FIXED>
__device__ __forceinline__ void match_tiled2_tile_g(const MatchArgs &a, int bx, int by_cta, float *tile) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    constexpr int NBW = SHARED ? 31 : 16;
    const int R = a.range, W = a.w, H = a.h, tp = a.tile_pitch;
    const int g = tile2_g(tp, FIXED), pp = 8 * g;
    const int kx0 = bx * NBW;
    const int x0 = kx0 * BS;
    const int by0 = by_cta * nw;
    const int by_last = min(by0 + nw - 1, a.nby - 1);
    const int y_first = min(BS * by0, H - 8);
    const int y_last = min(BS * by_last, H - 8);
    const int r0 = max(y_first - R, 0);
    const int nrows = min(y_last + R, H - 8) + 8 - r0;
    const int npe = (nrows + 1) >> 1;  // even-start pair rows
    float *tE = tile;
    float *tO = tile + npe * pp;
    const float *plane = a.frames + (long long)a.radius * a.fstride;
    {
        const int gx0 = x0 - R;
        for (int t = warp; t < nrows; t += nw) {
            const float *srow = plane + (long long)(r0 + t) * a.pitch;
            float *de = tE + (t >> 1) * pp + (t & 1);
            float *dq = t > 0 ? tO + ((t - 1) >> 1) * pp + ((t - 1) & 1) : nullptr;
            for (int c = lane; c < tp; c += 32) {
                const int gx = gx0 + c;
                const bool ok = gx >= 0 && gx < W;
                const float *gs = srow + (ok ? gx : 0);
                cp_async_f32(de + split_off(c, g), gs, ok);
                if (dq) cp_async_f32(dq + split_off(c, g), gs, ok);
            }
        }
    }
    cp_async_wait_all();
    __syncthreads();

    const int by = by0 + warp;
    if (by >= a.nby) return;
    const int y = min(BS * by, H - 8);
    const int b = SHARED ? lane : (lane >> 1);
    const int hh = SHARED ? 0 : (lane & 1);
    const int kx = kx0 + b;
    const int xb = BS * kx;
    const int uo = BS * b + 4 * hh;  // tile column of this half at dx = -R (a multiple of 4)
    const bool blk = (SHARED ? lane < 31 : true) && kx < a.nbx_al;

    // negated reference half as row pairs (2k, 2k+1) of each of its 4 columns
    float2 nc[4][4];
    {
        const int t0 = y - r0;
        const float *base = (t0 & 1) ? tO + ((t0 - 1) >> 1) * pp : tE + (t0 >> 1) * pp;
#pragma unroll
        for (int k = 0; k < 4; ++k)
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float2 v = *reinterpret_cast<const float2 *>(base + k * pp + split_off(uo + R + j, g));
                nc[k][j] = make_float2(-v.x, -v.y);
            }
    }

    float e[8];
    int q[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        e[i] = ZB_FLT_MAX;
        q[i] = 0;
    }
    const int top = max(y - R, 0), bottom = min(y + R, H - 8);
    const int lo = blk ? -xb : 1, hi = blk ? W - 8 - xb : 0;
    const int chunks = a.chunks;

    for (int row = top; row <= bottom; ++row) {
        const int t0 = row - r0;
        const float *prow = (t0 & 1) ? tO + ((t0 - 1) >> 1) * pp : tE + (t0 >> 1) * pp;
        const float *pc = prow + uo;  // column uo: chunk uo / 4 of the first half-plane
        for (int m = 0; m < chunks; ++m, pc += 4)
            tiled2_chunk<SHARED, FIXED ? kTile2G : 0>(pc, pp, g, m, R, row, xb, lo, hi, nc, e, q);
    }

    if (!blk || (!SHARED && hh)) return;
    store_list(a, (long long)by * a.nbx + kx, xb, y, e, q);
}

// The tile with the fixed half-plane size where the displacements allow it.
template <bool SHARED, int BS>
__device__ __forceinline__ void match_tiled2_tile(const MatchArgs &a, int bx, int by_cta, float *tile) {
    if (tile2_fixed(a.chunks))
        match_tiled2_tile_g<SHARED, BS, true>(a, bx, by_cta, tile);
    else
        match_tiled2_tile_g<SHARED, BS, false>(a, bx, by_cta, tile);
}

// packed FP32x2 SSD kernel: two pair-interleaved copies of the tile
inline size_t match_tile2_bytes(const MatchArgs &a, int rows_per_cta) {
    return (size_t)((rows_per_cta - 1) * a.bs + 2 * a.range + 8) * 8 * tile2_g(a.tile_pitch, tile2_fixed(a.chunks)) *
           sizeof(float);
}

}  // namespace zb
