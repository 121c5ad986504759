// Block matching kernels and their launchers.
//
// Compiled for sm_100a with -use_fast_math, the same floating-point mode as the
// reference kernel (vszipcu src/bm3d.zig:20-24).  The distance chains are written with
// explicit __fmul_rn/__fmaf_rn in the reference's order, so every match list is
// bit-identical to the reference's.
//
// Design (B200): one lane owns 4 columns ("half block") of a reference block and
// slides a 4x8 candidate window along each candidate row.  With block_step 4,
// lane k's half is the first half of block k and the second half of block
// k-1, so every column distance is computed once for two blocks.  Candidate
// rows of a whole warp-row of blocks are staged in a shared-memory tile and
// read as float4 (bank-conflict free, no shuffles in the inner loop except one
// to join the two halves).  The top-8 list lives in registers and follows the
// reference's insertion rule in scan order, so the lists are bit-identical.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "zb3d_args.h"
#include "zb3d_match.cuh"
#include "zb3d_match_scan.cuh"

namespace zb {

// ---------------------------------------------------------------------------
// Spatial matching, block_step 4 or 8, from a shared-memory tile.
// A warp covers one row of reference blocks; lane k's half starts at column
// x0 + 4k (SHARED: block k = lanes k, k+1) or, in PAIR mode, block b = lanes
// 2b, 2b+1.  The CTA's warps take consecutive block rows and share the tile,
// which is staged with cp.async.  Each candidate row is scanned in chunks of 4
// displacements; the two float4 window halves alternate roles between chunks so
// the sliding window never moves between registers.
// ---------------------------------------------------------------------------
template <int M, bool SHARED>
__device__ __forceinline__ void tiled_chunk(const float4 (&X)[8], const float4 (&Y)[8], int m, int R, int row, int xb,
                                            int lo, int hi, const float (&c)[8][4], float st, float (&e)[8],
                                            int (&q)[8]) {
#pragma unroll
    for (int s = 0; s < 4; ++s) {
        const int dx = -R + 4 * m + s;
        if (dx > R) break;
        float n[8][4];
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) n[i][j] = (j + s < 4) ? f4c(X[i], j + s) : f4c(Y[i], j + s - 4);
        const float hd = half_distance<M>(c, n, st, kFull);
        float err;
        if constexpr (SHARED)
            err = hd + __shfl_down_sync(kFull, hd, 1);
        else
            err = join_pair<M>(hd, kFull);
        if (dx >= lo && dx <= hi && err < e[7]) top8_insert(e, q, err, pack_pos(xb + dx, row));
    }
}

template <int M, bool SHARED, int BS>
__global__ void __launch_bounds__(128) zb_match_tiled(MatchArgs a) {
    extern __shared__ __align__(16) float tile[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    constexpr int NBW = SHARED ? 31 : 16;
    const int R = a.range, W = a.w, H = a.h, tp = a.tile_pitch;
    const int kx0 = blockIdx.x * NBW;
    const int x0 = kx0 * BS;
    const int by0 = blockIdx.y * nw;
    const int by_last = min(by0 + nw - 1, a.nby - 1);
    const int y_first = min(BS * by0, H - 8);
    const int y_last = min(BS * by_last, H - 8);
    const int r0 = max(y_first - R, 0);
    const int nrows = min(y_last + R, H - 8) + 8 - r0;
    const float *plane = a.frames + (long long)a.radius * a.fstride;
    stage_window(tile, tp, plane, a.pitch, x0 - R, r0, nrows, tp, W);
    cp_async_wait_all();
    __syncthreads();

    const int by = by0 + warp;
    if (by >= a.nby) return;
    const int y = min(BS * by, H - 8);
    const int b = SHARED ? lane : (lane >> 1);
    const int hh = SHARED ? 0 : (lane & 1);
    const int kx = kx0 + b;
    const int xb = BS * kx;
    const int uo = BS * b + 4 * hh;  // tile column of this half at dx = -R
    const bool blk = (SHARED ? lane < 31 : true) && kx < a.nbx_al;

    float c[8][4];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) c[i][j] = tile[(y - r0 + i) * tp + uo + R + j];
    const float st = ref_stat<M>(c, kFull);

    float e[8];
    int q[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        e[i] = ZB_FLT_MAX;
        q[i] = 0;
    }
    const int top = max(y - R, 0), bottom = min(y + R, H - 8);
    // valid displacements of this block: 0 <= xb + dx <= W - 8 (none for helper lanes)
    const int lo = blk ? -xb : 1, hi = blk ? W - 8 - xb : 0;
    const int chunks = a.chunks;

    for (int row = top; row <= bottom; ++row) {
        const float *tr = tile + (row - r0) * tp + uo;
        float4 A[8], B[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) A[i] = *reinterpret_cast<const float4 *>(tr + i * tp);
        for (int m = 0; m < chunks; m += 2) {
#pragma unroll
            for (int i = 0; i < 8; ++i) B[i] = *reinterpret_cast<const float4 *>(tr + i * tp + 4 * (m + 1));
            tiled_chunk<M, SHARED>(A, B, m, R, row, xb, lo, hi, c, st, e, q);
            if (m + 1 < chunks) {
#pragma unroll
                for (int i = 0; i < 8; ++i) A[i] = *reinterpret_cast<const float4 *>(tr + i * tp + 4 * (m + 2));
                tiled_chunk<M, SHARED>(B, A, m + 1, R, row, xb, lo, hi, c, st, e, q);
            }
        }
    }

    if (!blk || (!SHARED && hh)) return;
    store_list(a, (long long)by * a.nbx + kx, xb, y, e, q);
}

// The column on its own, beside the tiled kernels of the metrics that zb_match_scan does not take.
template <int M>
__global__ void __launch_bounds__(128) zb_match_column(MatchArgs a) {
    const int by = blockIdx.x * 4 + (threadIdx.x >> 5);
    if (by < a.nby) warp_block<M>(a, a.nbx - 1, by);  // whole warps
}

// Spatial SSD / SAD matching at block_step 4 and 8 (scan_tile), `rows` block rows per CTA of 8
// warps (QUEUE) or `rows` warps.  Where the plane's width leaves a clamped last block column, one more column of CTAs
// scans it, a warp per block, instead of a launch of its own (11 to 17 us, most of it the
// latency of one warp per block).
template <int M, bool SHARED, int BS, bool QUEUE>
__global__ void __launch_bounds__(kScanWarps * 32, 2) zb_match_scan(MatchArgs a, ZeroArgs zero, int rows) {
    extern __shared__ __align__(16) float tile[];
    zero_slice(zero, blockIdx.y * gridDim.x + blockIdx.x, gridDim.x * gridDim.y);
    if ((int)blockIdx.x == a.tiles_x) {
        const int warp = threadIdx.x >> 5, by = blockIdx.y * rows + warp;
        if (warp < rows && by < a.nby) warp_block<M>(a, a.nbx - 1, by);
        return;
    }
    scan_tile<M, SHARED, BS, QUEUE>(a, blockIdx.x, blockIdx.y, rows, tile);
}

// Spatial matching for block steps the tiled kernels do not take (and the blocks the
// tensor-core form lists), reading candidates through the L1/L2 path.  Lane pair per block.
template <int M>
__global__ void __launch_bounds__(128) zb_match_global(MatchArgs a) {
    const int lane = threadIdx.x & 31;
    const long long pair = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 1;
    const int hh = lane & 1;
    const long long nb = a.gen_mode == 2 ? (long long)a.tc_ws[0] : (long long)a.nby * a.nbx;
    if (pair >= nb) return;
    int kx, by;
    if (a.gen_mode == 2) {
        const int bi = a.tc_ws[kTcWsList + pair];
        by = bi / a.nbx;
        kx = bi - by * a.nbx;
    } else {
        by = (int)(pair / a.nbx);
        kx = (int)(pair - (long long)by * a.nbx);
    }
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
    if constexpr (M == M_SSD) {
        float2 nc[4][4];
        neg_pairs(c, nc);
        scan_window_ssd2(plane, a.pitch, max(x - R, 0), min(x + R, W - 8), max(y - R, 0), min(y + R, H - 8), nc, pm,
                         e, q);
    } else {
        scan_window<M>(plane, a.pitch, max(x - R, 0), min(x + R, W - 8), max(y - R, 0), min(y + R, H - 8), c, st, pm,
                       e, q);
    }
    if (hh) return;
    store_list(a, (long long)by * a.nbx + kx, x, y, e, q);
}

// ---------------------------------------------------------------------------
// Temporal predictive search (vszipcu src/bm3d.cu:663-756) and self inclusion
// (:758-788).  Starts from the spatial list; for direction -1 then +1 and
// t = 1..r a per-frame list is built from ps_range windows around the first
// ps_num entries of the previous list (t = 1: the spatial list), and its first
// ps_num entries are merged into the block's list.  Only those first ps_num entries of a
// per-frame list are ever read, so the per-frame list holds K >= ps_num entries: the
// first K of the reference's 8-entry list (K = 2 covers the default ps_num).  For SSD the
// kernel is held at 128 registers, 4 CTAs per SM, so that a 1080p plane at block_step 8
// (507 CTAs) runs in one wave; the other metrics keep their 3 CTAs per SM.
// ---------------------------------------------------------------------------
template <int M, int K>
__global__ void __launch_bounds__(128, M == M_SSD ? 4 : 3) zb_match_temporal(MatchArgs a) {
    const int lane = threadIdx.x & 31;
    const long long pair = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 1;
    const int hh = lane & 1;
    const long long nb = (long long)a.nby * a.nbx;
    if (pair >= nb) return;
    const int by = (int)(pair / a.nbx), kx = (int)(pair - (long long)by * a.nbx);
    const int W = a.w, H = a.h, r = a.radius, P = a.ps_range;
    const int x = min(a.bs * kx, W - 8), y = min(a.bs * by, H - 8);
    const unsigned pm = 3u << (lane & 30);
    const float *centre = a.frames + (long long)r * a.fstride + 4 * hh;

    float c[8][4];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) c[i][j] = __ldg(centre + (long long)(y + i) * a.pitch + x + j);
    const float st = ref_stat<M>(c, pm);
    float2 nc[4][4];
    if constexpr (M == M_SSD) neg_pairs(c, nc);

    float ge[8];
    int gq[8], gz[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int2 v = a.list[pair * 8 + i];
        ge[i] = a.errs[pair * 8 + i];
        gq[i] = pack_pos(v.x, v.y & 0xffffff);
        gz[i] = r;
    }
#pragma unroll 1
    for (int dir = -1; dir <= 1; dir += 2) {
        // each direction starts from the spatial list (still unchanged in memory)
        int lq[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int2 v = a.list[pair * 8 + i];
            lq[i] = pack_pos(v.x, v.y & 0xffffff);
        }
#pragma unroll 1
        for (int t = 1; t <= r; ++t) {
            const int zt = r + dir * t;
            const float *fp = a.frames + (long long)zt * a.fstride + 4 * hh;
            float fe[K];
            int fq[K];
#pragma unroll
            for (int i = 0; i < K; ++i) {
                fe[i] = ZB_FLT_MAX;
                fq[i] = 0;
            }
#pragma unroll
            for (int i = 0; i < K; ++i) {
                if (i < a.ps_num) {
                    const int xx = pos_x(lq[i]), yy = pos_y(lq[i]);
                    if constexpr (M == M_SSD)
                        scan_window_ssd2<K>(fp, a.pitch, max(xx - P, 0), min(xx + P, W - 8), max(yy - P, 0),
                                            min(yy + P, H - 8), nc, pm, fe, fq);
                    else
                        scan_window<M, K>(fp, a.pitch, max(xx - P, 0), min(xx + P, W - 8), max(yy - P, 0),
                                          min(yy + P, H - 8), c, st, pm, fe, fq);
                }
            }
#pragma unroll
            for (int i = 0; i < K; ++i)
                if (i < a.ps_num && fe[i] < ge[7]) top8_insert_z(ge, gq, gz, fe[i], fq[i], zt);
#pragma unroll
            for (int i = 0; i < K; ++i) lq[i] = fq[i];
        }
    }
    if (hh) return;
    const int self = pack_pos(x, y);
    bool found = false;
#pragma unroll
    for (int i = 0; i < 8; ++i) found |= (gq[i] == self && gz[i] == r);
    if (!found) {
#pragma unroll
        for (int i = 7; i > 0; --i) {
            gq[i] = gq[i - 1];
            gz[i] = gz[i - 1];
        }
        gq[0] = self;
        gz[0] = r;
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) a.list[pair * 8 + i] = make_int2(pos_x(gq[i]), pos_y(gq[i]) | (gz[i] << 24));
}

// ---------------------------------------------------------------------------
// Host-side launchers.
// ---------------------------------------------------------------------------
size_t match_tile_bytes(const MatchArgs &a, int rows_per_cta);

template <int M, bool SHARED, int BS>
static cudaError_t launch_tiled_t(const MatchArgs &a, int rows_per_cta, cudaStream_t st) {
    constexpr int NBW = SHARED ? 31 : 16;
    const int gx = (a.nbx_al + NBW - 1) / NBW;
    const int gy = (a.nby + rows_per_cta - 1) / rows_per_cta;
    const size_t smem = match_tile_bytes(a, rows_per_cta);
    auto k = zb_match_tiled<M, SHARED, BS>;
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemOptIn);
    if (e != cudaSuccess) return e;
    k<<<dim3(gx, gy), rows_per_cta * 32, smem, st>>>(a);
    return cudaGetLastError();
}

// Whether the scan kernel takes an entry with this many block rows per CTA: ssd and sad at
// block_step 4 and 8, a tile that fits shared memory.
bool scan_rows_fit(const MatchJob &a, int metric, int rows_per_cta) {
    if ((metric != M_SSD && metric != M_SAD) || (a.bs != 4 && a.bs != 8)) return false;
    return scan_smem_bytes(a, rows_per_cta) <= kSmemOptIn;
}

// Whether two such CTAs share an SM (227 KB, 1 KB of it reserved per CTA).
bool scan_rows_fit2(const MatchJob &a, int metric, int rows_per_cta) {
    return scan_rows_fit(a, metric, rows_per_cta) && scan_smem_bytes(a, rows_per_cta) <= kSmemOptIn / 2;
}

size_t scan_smem(const MatchJob &a, int rows) { return scan_smem_bytes(a, rows); }
size_t scan_tile_smem(const MatchJob &a, int rows) { return scan_tile_bytes(a, rows); }

// The scan's shape without a timing: sets a.direct and returns the block rows per CTA (0: the
// kernel takes no shape of the entry).  full: other planes fill the GPU beside this one.
// 3840x2160 ssd, us (block_step 4 / 8; d8 and d4: inserted at once with 8 and 4 rows, q8 .. q1: queues):
//   bm_range  9:  d8  602 /  293, d4  573 /  308, q8  625 /  370, q4  689 /  339
//   bm_range 16:  d8 1618 /  994, d4 1637 /  931, q8 1890 /  907, q4 1702 /  988, q2 1861 /  918
//   bm_range 24:  d8 4373 / 2064, d4 3879 / 1910, q8 3818 / 1825, q4 3955 / 1932, q1 4087 / 1989
// so with CTAs enough (and no temporal search, see tune_entry): at once while two CTAs of 8 rows
// fit an SM, then queues with the most rows
// (2 at least) that two CTAs fit with, then queues with the most rows.  With fewer CTAs than two
// per SM the split of the candidate rows counts most (640x480 at block_step 8, bm_range 9: d8 61,
// d4 51, q4 47, q2 38, q1 32; 320x240 at 4, bm_range 12: d8 92, d4 75, q4 65, q2 42, q1 40): queues
// with 4 rows, which cost the other streams less than more ranges would.
int scan_shape(MatchJob &a, int metric, bool full) {
    int sms = 148, dev = 0;
    if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    full = full || (long long)scan_tiles_x(a) * ((a.nby + 3) / 4) >= 2LL * sms;
    a.direct = 1;
    if (full && a.radius == 0 && scan_rows_fit2(a, metric, 8)) return 8;
    a.direct = 0;
    for (int r = full ? 8 : 4; r >= (full ? 2 : 1); r >>= 1)
        if (scan_rows_fit2(a, metric, r)) return r;
    for (int r = full ? 8 : 4; r >= 1; r >>= 1)
        if (scan_rows_fit(a, metric, r)) return r;
    return 0;
}

template <int M, bool SHARED, int BS>
static cudaError_t launch_scan_t(const MatchJob &a, int rows, cudaStream_t st) {
    auto k = a.direct ? zb_match_scan<M, SHARED, BS, false> : zb_match_scan<M, SHARED, BS, true>;
    // the same limit at every launch: a limit of this launch's size would race with other
    // threads' launches of the same kernel
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemOptIn);
    if (e != cudaSuccess) return e;
    const int gx = a.tiles_x + (a.nbx_al != a.nbx ? 1 : 0), gy = (a.nby + rows - 1) / rows;
    k<<<dim3(gx, gy), (a.direct ? rows : kScanWarps) * 32, scan_smem_bytes(a, rows), st>>>(a, a.zero, rows);
    return cudaGetLastError();
}

// Block rows per CTA of the scan: the asked power of two, or fewer where its tile does not
// fit; 0 where none does.
static int scan_rows(const MatchJob &a, int metric, int rows) {
    int r = rows >= 8 ? 8 : rows >= 4 ? 4 : rows >= 2 ? 2 : 1;
    while (r > 0 && !scan_rows_fit(a, metric, r)) r >>= 1;
    return r;
}

template <int M>
static cudaError_t launch_tiled_m(MatchJob a, int rows_per_cta, cudaStream_t st) {
    if constexpr (M == M_SSD || M == M_SAD) {
        if (const int rows = scan_rows(a, M, rows_per_cta)) {
            a.tiles_x = scan_tiles_x(a);
            return a.bs == 8 ? launch_scan_t<M, false, 8>(a, rows, st) : launch_scan_t<M, true, 4>(a, rows, st);
        }
    }
    rows_per_cta = std::min(rows_per_cta, 4);
    if (a.bs == 8) return launch_tiled_t<M, false, 8>(a, rows_per_cta, st);
    if constexpr (Shareable<M>::value) return launch_tiled_t<M, true, 4>(a, rows_per_cta, st);
    return launch_tiled_t<M, false, 4>(a, rows_per_cta, st);
}

// Every block of a small plane, a warp per block.
template <int M>
__global__ void __launch_bounds__(128) zb_match_blocks(MatchArgs a) {
    const int bi = blockIdx.x * 4 + (threadIdx.x >> 5);
    if (bi >= a.nby * a.nbx) return;  // whole warps
    const int by = bi / a.nbx;
    warp_block<M>(a, bi - by * a.nbx, by);
}

// Up to this many blocks (one wave of 16 warps per SM) a warp takes a block; a lane pair per
// block (zb_match_global) does a third of the work but leaves a plane of this size on at most
// 148 warps: block_step 5,
// bm_range 9, 320 blocks 105 -> 21 us, 960 blocks 105 -> 27 us.  Above it three streams fill the
// GPU with lane pairs and the work counts.
constexpr long long kWarpBlocks = 148 * 16;

template <int M>
static cudaError_t launch_global_m(const MatchArgs &a, cudaStream_t st) {
    if (a.gen_mode == 0 && (long long)a.nby * a.nbx <= kWarpBlocks) {
        zb_match_blocks<M><<<(unsigned)((a.nby * a.nbx + 3) / 4), 128, 0, st>>>(a);
        return cudaGetLastError();
    }
    // listed blocks (gen_mode 2): the count is on the device, so size for every block
    const long long threads = (long long)a.nby * a.nbx * 2;
    zb_match_global<M><<<(unsigned)((threads + 127) / 128), 128, 0, st>>>(a);
    return cudaGetLastError();
}

template <int M>
static cudaError_t launch_column_m(const MatchArgs &a, cudaStream_t st) {
    zb_match_column<M><<<(unsigned)((a.nby + 3) / 4), 128, 0, st>>>(a);
    return cudaGetLastError();
}

template <int M>
static cudaError_t launch_temporal_m(const MatchArgs &a, cudaStream_t st) {
    const long long threads = (long long)a.nby * a.nbx * 2;
    if (a.ps_num <= 2)
        zb_match_temporal<M, 2><<<(unsigned)((threads + 127) / 128), 128, 0, st>>>(a);
    else
        zb_match_temporal<M, 8><<<(unsigned)((threads + 127) / 128), 128, 0, st>>>(a);
    return cudaGetLastError();
}

// Shared-memory bytes the tiled kernel needs for `rows_per_cta` block rows.
size_t match_tile_bytes(const MatchArgs &a, int rows_per_cta) {
    return (size_t)((rows_per_cta - 1) * a.bs + 2 * a.range + 8) * a.tile_pitch * sizeof(float);
}

bool tc_eligible(const MatchArgs &a);                          // zb3d_match_tc.cu
cudaError_t launch_match_tc(const MatchJob &a, cudaStream_t st);
bool temporal_rows_eligible(const MatchArgs &a, int metric);   // zb3d_match_temporal.cu
cudaError_t launch_temporal_rows(const MatchJob &a, cudaStream_t st);

// The FP32 scan of the blocks the tensor-core kernel listed (SSD, radius 0).
cudaError_t launch_tc_fallback(MatchArgs a, cudaStream_t st) {
    a.self_incl = a.radius == 0;
    a.gen_mode = 2;
    return launch_global_m<M_SSD>(a, st);
}

cudaError_t launch_match(MatchJob a, int metric, int rows_per_cta, bool use_tiled, cudaStream_t st) {
    cudaError_t e = cudaSuccess;
    const bool tiled = use_tiled && (a.bs == 4 || a.bs == 8);
    a.self_incl = a.radius == 0;
    const bool tc = metric == M_SSD && a.tc_ws != nullptr && tc_eligible(a);
    a.chunks = (2 * a.range + 1 + 3) / 4;
    a.tile_pitch = 128 + 4 * a.chunks;
    if (a.zero.acc[0] && (tc || !tiled || !scan_rows(a, metric, rows_per_cta))) {
        for (int k = 0; k < 2; ++k)
            if ((e = cudaMemsetAsync(a.zero.acc[k], 0, (size_t)a.zero.count * 8, st)) != cudaSuccess) return e;
        a.zero.acc[0] = nullptr;
    }
    if (tc) {
        // tensor-core bound + exact re-rank; the blocks it lists get the FP32 scan
        if ((e = launch_match_tc(a, st)) != cudaSuccess) return e;
        a.gen_mode = 2;
        if ((e = launch_global_m<M_SSD>(a, st)) != cudaSuccess) return e;
        goto temporal;
    }
    if (tiled) {
        switch (metric) {
        case M_SSD: e = launch_tiled_m<M_SSD>(a, rows_per_cta, st); break;
        case M_SAD: e = launch_tiled_m<M_SAD>(a, rows_per_cta, st); break;
        case M_ZSSD: e = launch_tiled_m<M_ZSSD>(a, rows_per_cta, st); break;
        case M_ZSAD: e = launch_tiled_m<M_ZSAD>(a, rows_per_cta, st); break;
        default: e = launch_tiled_m<M_SSD_NORM>(a, rows_per_cta, st); break;
        }
        if (e != cudaSuccess) return e;
        if (a.nbx_al == a.nbx || scan_rows(a, metric, rows_per_cta)) goto temporal;
        switch (metric) {  // the clamped last column
        case M_SSD: e = launch_column_m<M_SSD>(a, st); break;
        case M_SAD: e = launch_column_m<M_SAD>(a, st); break;
        case M_ZSSD: e = launch_column_m<M_ZSSD>(a, st); break;
        case M_ZSAD: e = launch_column_m<M_ZSAD>(a, st); break;
        default: e = launch_column_m<M_SSD_NORM>(a, st); break;
        }
        if (e != cudaSuccess) return e;
        goto temporal;
    }
    a.gen_mode = 0;
    switch (metric) {
    case M_SSD: e = launch_global_m<M_SSD>(a, st); break;
    case M_SAD: e = launch_global_m<M_SAD>(a, st); break;
    case M_ZSSD: e = launch_global_m<M_ZSSD>(a, st); break;
    case M_ZSAD: e = launch_global_m<M_ZSAD>(a, st); break;
    default: e = launch_global_m<M_SSD_NORM>(a, st); break;
    }
    if (e != cudaSuccess) return e;
temporal:
    if (a.radius > 0 && temporal_rows_eligible(a, metric)) {
        e = launch_temporal_rows(a, st);
    } else if (a.radius > 0) {
        switch (metric) {
        case M_SSD: e = launch_temporal_m<M_SSD>(a, st); break;
        case M_SAD: e = launch_temporal_m<M_SAD>(a, st); break;
        case M_ZSSD: e = launch_temporal_m<M_ZSSD>(a, st); break;
        case M_ZSAD: e = launch_temporal_m<M_ZSAD>(a, st); break;
        default: e = launch_temporal_m<M_SSD_NORM>(a, st); break;
        }
    }
    return e;
}

}  // namespace zb
