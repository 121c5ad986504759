// Temporal predictive search (vszipcu src/bm3d.cu:663-756) for ssd with ps_num <= 2: search
// windows staged in shared memory, one lane per candidate row.  Compiled with
// -use_fast_math like the other matching kernels; the lists are theirs bit for bit.
//
// A group of 2P + 1 lanes (P = ps_range) serves one reference block, and a warp holds
// 32 / (2P + 1) groups (3 for P = 4).  For each neighbouring frame and each of the ps_num
// windows the group stages the window's (2P + 8)^2 pixels; lane r then scans candidate row r:
// every column of its 8 rows is loaded once, as row pairs (2k, 2k+1), and feeds the packed
// FP32x2 chains of all displacements that cover it.  Each lane keeps the first two candidates
// of its row; they are merged in row order, then window after window, by strict-less
// insertion, which gives the first two entries of the reference's frame list (the only ones it
// reads for ps_num <= 2).
//
// What bounds it: the FMA pipe (576 packed operations per lane and window; 27 of 32 lanes have
// a row), shared with the load-store unit's 128 column reads and 32 copies per window.  A
// window's place is only known once an earlier one is done, so the two directions take turns
// and the next window is copied (cp.async, a second buffer) while this one is scanned.
// 1920x1080, block_step 8, radius 2 (21.0 M candidates): 355 us for the lane-pair form that this
// replaces (zb_match_temporal, still used for other metrics, ps_num > 2 and other window sizes:
// it reads its windows through L1 with one lane pair per block and waits on those loads), about
// 190 us here; ps_range 2 124 -> 95, 3 218 -> 133, 5 490 -> 340, 6 670 -> 395.  Windows loaded to
// registers ahead of each scan instead of copied under it: the same alone, 2.5% slower a
// window among others, and only for 16-byte aligned planes.
#include <cuda_runtime.h>

#include <cstdint>

#include "zb3d_args.h"
#include "zb3d_match.cuh"

namespace zb {

constexpr int kTempWarps = 4;

template <int P>
struct TempShape {
    static constexpr int G = 2 * P + 1;              // lanes per group, candidate rows and columns of a window
    static constexpr int NG = 32 / G;                // groups per warp
    static constexpr int N = 2 * P + 8;              // window side in pixels
    static constexpr int LN = G < 8 ? G : 8;         // lanes that copy a row
    static constexpr int PITCH = N | 1;              // floats per row: odd
    // floats between the groups' windows; for P = 4 the rows of the three groups (at 0, 10 and 20
    // mod 32, 17 floats apart) are on 27 different banks
    static constexpr int WIN = N * PITCH + 26;
    static constexpr int BUF = NG * WIN;             // floats of a warp's windows; each warp has two sets
};

// Strict-less insertion into a list of two.
__device__ __forceinline__ void top2_insert(float &e0, int &q0, float &e1, int &q1, float err, int pos) {
    const bool c0 = err < e0, c1 = err < e1;
    q1 = c0 ? q0 : (c1 ? pos : q1);
    q0 = c0 ? pos : q0;
    e1 = fminf(e1, fmaxf(e0, err));
    e0 = fminf(e0, err);
}

// Starts the copy of the group's window of frame plane fp around (xx, yy) into win: LN lanes on
// LN consecutive pixels, row after row.  Rows and columns past the plane are only read by
// candidates that do not exist: clamped.
template <int P>
__device__ __forceinline__ void stage_window_group(const MatchArgs &a, const float *__restrict__ fp, int xx, int yy,
                                                   int r, float *win) {
    using S = TempShape<P>;
    constexpr int N = S::N, LN = S::LN, CH = (N + LN - 1) / LN;
    const int left = max(xx - P, 0), top = max(yy - P, 0);
    if (r < LN) {
        const int ymax = a.h - 1 - top;
        const float *src[CH];
#pragma unroll
        for (int c = 0; c < CH; ++c) src[c] = fp + (long long)top * a.pitch + min(left + r + LN * c, a.w - 1);
#pragma unroll
        for (int row = 0; row < N; ++row) {
            const long long o = (long long)min(row, ymax) * a.pitch;
#pragma unroll
            for (int c = 0; c < CH; ++c)
                if (LN * (c + 1) <= N || r + LN * c < N)
                    cp_async_f32(win + row * S::PITCH + r + LN * c, src[c] + o, true);
        }
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
}

// The staged window around (xx, yy): its first two candidates in scan order, on every lane of
// the group.  r: the lane's candidate row (>= G: a lane without one).
template <int P>
__device__ __forceinline__ void scan_window_group(const MatchArgs &a, int xx, int yy, int r, int lane, unsigned gmask,
                                                  const float *win, const float2 (&nc)[4][8], float &e0, int &q0,
                                                  float &e1, int &q1) {
    using S = TempShape<P>;
    constexpr int G = S::G, N = S::N, PITCH = S::PITCH;
    const int W = a.w, H = a.h;
    const int left = max(xx - P, 0), right = min(xx + P, W - 8);
    const int top = max(yy - P, 0), bottom = min(yy + P, H - 8);
    const int dy = min(r, G - 1);
    const bool rowok = r < G && top + dy <= bottom;
    const int nx = rowok ? right - left + 1 : 0;
    const int pos = pack_pos(left, top + dy);
    const float *base = win + dy * PITCH;
    e0 = e1 = ZB_FLT_MAX;
    q0 = q1 = 0;
    float A[G], B[G], C[G], D[G];
#pragma unroll
    for (int c = 0; c < N; ++c) {
        float2 v[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) v[k] = make_float2(base[2 * k * PITCH + c], base[(2 * k + 1) * PITCH + c]);
#pragma unroll
        for (int j = 7; j >= 0; --j) {
            const int s = c - j;
            if (s < 0 || s >= G) continue;
            float2 d = __fadd2_rn(v[0], nc[0][j]);
            float2 acc = __fmul2_rn(d, d);
#pragma unroll
            for (int k = 1; k < 4; ++k) {
                d = __fadd2_rn(v[k], nc[k][j]);
                acc = __ffma2_rn(d, d, acc);
            }
            const float t = acc.x + acc.y;
            // ((s0 + s1) + (s2 + s3)) + ((s4 + s5) + (s6 + s7))
            if (j == 0) A[s] = t;
            if (j == 1) A[s] += t;
            if (j == 2) B[s] = t;
            if (j == 3) A[s] += B[s] + t;
            if (j == 4) C[s] = t;
            if (j == 5) C[s] += t;
            if (j == 6) D[s] = t;
            if (j == 7) {
                float err = A[s] + (C[s] + (D[s] + t));
                err = s < nx && err < ZB_FLT_MAX ? err : ZB_FLT_MAX;  // NaN too: never below an entry
                top2_insert(e0, q0, e1, q1, err, pos + s);
            }
        }
    }
    // The first two of the group in row order, on every lane: the smallest head of the rows'
    // lists, of the first row that has it (errors are not negative: ordered as integers).
    float m[2];
    int w[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const unsigned head = __float_as_uint(e0);
        const unsigned least = __reduce_min_sync(gmask, head);
        const int first = __ffs(__ballot_sync(kFull, head == least) & gmask) - 1;
        m[i] = __uint_as_float(least);
        w[i] = __shfl_sync(kFull, q0, first);
        if (first == lane) {
            e0 = e1;
            q0 = q1;
            e1 = ZB_FLT_MAX;
            q1 = 0;
        }
    }
    e0 = m[0];
    q0 = w[0];
    e1 = m[1];
    q1 = w[1];
}

template <int P>
__global__ void __launch_bounds__(kTempWarps * 32, 4) zb_match_temporal_rows(MatchJob a) {
    using S = TempShape<P>;
    constexpr int G = S::G, NG = S::NG;
    __shared__ float wins[kTempWarps * 2 * S::BUF];
    extern __shared__ int2 found[];  // [group][direction][t][2]: the frame lists (error, position)
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const bool member = lane < NG * G;
    const int g = member ? lane / G : 0, r = member ? lane - g * G : G;
    const unsigned gmask = member ? ((1u << G) - 1u) << (g * G) : ~0u << (NG * G);
    const long long nb = (long long)a.nby * a.nbx;
    const long long slot = ((long long)blockIdx.x * kTempWarps + warp) * NG + g;
    const long long bi = min(slot, nb - 1);  // the warp stays whole
    const int by = (int)(bi / a.nbx), kx = (int)(bi - (long long)by * a.nbx);
    const int W = a.w, H = a.h, R = a.radius;
    const int x = min(a.bs * kx, W - 8), y = min(a.bs * by, H - 8);
    float *win = wins + warp * 2 * S::BUF + g * S::WIN;
    int2 *mine = found + (size_t)(warp * NG + g) * 4 * R;

    // the negated reference patch as row pairs (2k, 2k + 1) of its 8 columns
    float2 nc[4][8];
    {
        const float *c = a.frames + (long long)R * a.fstride + (long long)y * a.pitch + x;
#pragma unroll
        for (int k = 0; k < 4; ++k)
#pragma unroll
            for (int j = 0; j < 8; ++j)
                nc[k][j] = make_float2(-__ldg(c + 2 * k * a.pitch + j), -__ldg(c + (2 * k + 1) * a.pitch + j));
    }
    const int2 l0 = a.list[bi * 8], l1 = a.list[bi * 8 + 1];
    // Windows in the order t = 1..r, direction, i: the window after the current one is then
    // always known (its centre comes from the same direction's frame t - 1), so it is copied
    // while the current one is scanned.  Each direction starts from the spatial list.
    const int s0 = pack_pos(l0.x, l0.y & 0xffffff), s1 = pack_pos(l1.x, l1.y & 0xffffff);
    int p0 = s0, p1 = s1, o0 = s0, o1 = s1;  // centres: this direction's, the other's
    float e0 = ZB_FLT_MAX, e1 = ZB_FLT_MAX, w0 = 0.0f, w1 = 0.0f;
    int q0 = 0, q1 = 0, u0 = 0, u1 = 0;
    const int per_frame = a.ps_num, items = 2 * R * per_frame;
    auto frame_of = [&](int k) {  // plane of item k
        const int f = k / per_frame, t = f / 2 + 1;
        return a.frames + (long long)((f & 1) ? R + t : R - t) * a.fstride;
    };
    stage_window_group<P>(a, frame_of(0), pos_x(p0), pos_y(p0), r, win);
#pragma unroll 1
    for (int k = 0; k < items; ++k) {
        const int i = k - k / per_frame * per_frame;
        const bool last = i == per_frame - 1;  // of its frame: the next item is the other direction's
        float *cur = win + (k & 1) * S::BUF, *nxt = win + ((k + 1) & 1) * S::BUF;
        if (k + 1 < items) {
            const int c = last ? o0 : p1;
            __syncwarp();  // the buffer's window has been read
            stage_window_group<P>(a, frame_of(k + 1), pos_x(c), pos_y(c), r, nxt);
            asm volatile("cp.async.wait_group 1;\n" ::: "memory");
        } else {
            asm volatile("cp.async.wait_group 0;\n" ::: "memory");
        }
        __syncwarp();
        const int p = i ? p1 : p0;
        // a second window at the same place has the same candidates
        if (i == 0 || !__all_sync(kFull, p1 == p0))
            scan_window_group<P>(a, pos_x(p), pos_y(p), r, lane, gmask, cur, nc, w0, u0, w1, u1);
        top2_insert(e0, q0, e1, q1, w0, u0);
        top2_insert(e0, q0, e1, q1, w1, u1);
        if (last) {
            const int f = k / per_frame;
            if (r == 0) {
                int2 *o = mine + ((f & 1) * R + f / 2) * 2;
                o[0] = make_int2(__float_as_int(e0), q0);
                o[1] = make_int2(__float_as_int(e1), q1);
            }
            // the other direction next; this one goes on from the frame's list
            p0 = o0;
            p1 = o1;
            o0 = q0;
            o1 = q1;
            e0 = e1 = ZB_FLT_MAX;
            q0 = q1 = 0;
        }
    }
    if (r != 0 || slot >= nb) return;
    // the block's list: the spatial one, then every frame's first ps_num entries in order
    float ge[8];
    int gq[8], gz[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int2 v = a.list[bi * 8 + i];
        ge[i] = a.errs[bi * 8 + i];
        gq[i] = pack_pos(v.x, v.y & 0xffffff);
        gz[i] = R;
    }
#pragma unroll 1
    for (int k = 0; k < 2 * R; ++k) {
        const int zt = k < R ? R - 1 - k : k + 1;
#pragma unroll 1
        for (int i = 0; i < a.ps_num; ++i) {
            const int2 f = mine[2 * k + i];
            const float fe = __int_as_float(f.x);
            if (fe < ge[7]) top8_insert_z(ge, gq, gz, fe, f.y, zt);
        }
    }
    const int self = pack_pos(x, y);
    bool have = false;
#pragma unroll
    for (int i = 0; i < 8; ++i) have |= (gq[i] == self && gz[i] == R);
    if (!have) {
#pragma unroll
        for (int i = 7; i > 0; --i) {
            gq[i] = gq[i - 1];
            gz[i] = gz[i - 1];
        }
        gq[0] = self;
        gz[0] = R;
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) a.list[bi * 8 + i] = make_int2(pos_x(gq[i]), pos_y(gq[i]) | (gz[i] << 24));
}

template <int P>
static cudaError_t launch_rows_t(const MatchJob &a, cudaStream_t st) {
    const long long nb = (long long)a.nby * a.nbx;
    const int per = kTempWarps * TempShape<P>::NG;
    zb_match_temporal_rows<P><<<(unsigned)((nb + per - 1) / per), kTempWarps * 32,
                                (size_t)per * 4 * a.radius * sizeof(int2), st>>>(a);
    return cudaGetLastError();
}

// Whether the row kernel takes this search: window rows that fill a warp well, in a plane of more
// than 4 candidate positions (it scans whole windows: 8x8, 1 position, radius 3, ps_range 4: 37 us a
// search, 14.5 with a lane pair per block, which scans the positions that exist; 10x10, 9
// positions: equal).
bool temporal_rows_eligible(const MatchArgs &a, int metric) {
    return metric == M_SSD && a.ps_num >= 1 && a.ps_num <= 2 && a.ps_range >= 2 && a.ps_range <= 6 &&
           (long long)(a.w - 7) * (a.h - 7) > 4;
}

cudaError_t launch_temporal_rows(const MatchJob &a, cudaStream_t st) {
    switch (a.ps_range) {
    case 2: return launch_rows_t<2>(a, st);
    case 3: return launch_rows_t<3>(a, st);
    case 4: return launch_rows_t<4>(a, st);
    case 5: return launch_rows_t<5>(a, st);
    default: return launch_rows_t<6>(a, st);
    }
}

}  // namespace zb
