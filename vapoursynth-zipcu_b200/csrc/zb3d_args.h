// Kernel argument blocks shared by the CUDA kernels and the C++ host.
#pragma once
#include <cstdint>

namespace zb {

enum Metric { M_SSD = 0, M_SAD = 1, M_ZSSD = 2, M_ZSAD = 3, M_SSD_NORM = 4 };

// Block matching of one plane entry.  Reference blocks sit at
// x = min(bs*kx, w-8), y = min(bs*ky, h-8) (vszipcu src/bm3d.cu:585-595).
// A kernel argument of at most 128 bytes: with a larger one nvcc compiles every kernel that takes
// it to other registers (sad scan from global memory 126 -> 120, general temporal search of ssd
// with 8 entries 228 -> 464 bytes of spills), and those were up to 18% slower.  What only the
// launchers or one kernel want is in MatchJob.  Two kernels are better with the larger argument
// and take a MatchJob: the temporal rows kernel (1920x1080, radius 2: 2 us) and the tensor-core
// form (no spills; 32 bytes with MatchArgs).
struct MatchArgs {
    const float *frames;   // matching plane of window frame t at frames + t*fstride
    long long fstride;
    int w, h, pitch;
    int bs, range;
    int radius, ps_num, ps_range;
    int nbx, nby;          // reference blocks per row / column
    int nbx_al;            // blocks whose x = bs*kx needs no clamp
    int tile_pitch;        // shared tile row pitch in floats (tiled kernel)
    int chunks;            // ceil((2*range+1)/4)
    int tiles_x;           // scan kernel: tiles per row; one more column of CTAs takes the clamped blocks
    int2 *list;            // [nby*nbx][8]: (x, y | z << 24)
    float *errs;           // [nby*nbx][8]: distances of the spatial list (radius > 0)
    int self_incl;         // 1: insert the block itself here (radius 0)
    int gen_mode;          // generic kernel: 0 = every block, 2 = the blocks listed in tc_ws
                           // (fallbacks of the tensor-core form)
    // Tensor-core form (zb3d_match_tc.cu).  tc_ws: [0] number of listed fallback
    // blocks, [kTcWsList..] their block indices.  tc_stats (optional, accumulated):
    // [0] tiles, [1] blocks, [2] re-ranked candidates, [3] fallback blocks.
    int *tc_ws;
    unsigned long long *tc_stats;
    float *tc_dbg;         // optional: pass-1 distances of tile (0, 0), [128][tiles flat candidates]
    unsigned long long *tc_prof;  // optional: per tile [16]: clock64 phase marks [0..7], mbarrier
                                  // polls of the block and issuer warps [8], [10], TMEM load cycles
                                  // and count [11], [13], pass-1 / pass-2 / done-wait cycles [12], [14], [15]; then for tile (1, 1) a per-job trace
                                  // [job][3] (issued, completion seen, slot freed), at most 64 jobs
};

static_assert(sizeof(MatchArgs) <= 128, "see above");

// Accumulators that start from zero after the matching (null: none): two arrays of `count`
// 64-bit words.  The scan kernel writes the zeros itself, its stores being free beside the
// arithmetic; before the other matchers they are cleared by memset nodes.
struct ZeroArgs {
    unsigned long long *acc[2];
    long long count;
};

// What launch_match takes, and the argument of zb_match_temporal_rows and zb_match_tc.
struct MatchJob : MatchArgs {
    ZeroArgs zero;
    int direct;            // scan kernel: 1 = a warp per block row, candidates inserted at once; 0 = 8 warps, queues
};

constexpr int kTcWsList = 8;

// Collaborative filtering + aggregation of one plane entry.
struct FilterArgs {
    const float *src;                 // [clips][planes][tw][h][pitch]
    long long clip_stride, plane_stride, frame_stride;
    int w, h, pitch;
    int nplanes, chroma;
    const int2 *list;                 // [nblocks][8]
    int nblocks;
    float sigma[3];                   // already scaled (hard or Wiener factor)
    float extractor;                  // 2^extractor_exp, or 0
    unsigned long long *num;          // [planes][tw][h][pitch]  fixed point, 2^32 = 1.0
    unsigned long long *den;          // [planes][tw][h][pitch]  weights at patch origins
    long long acc_plane_stride, acc_frame_stride;
};

// One plane entry of a batch (zb3d_process_batch): its matching and filtering arguments
// (own list and accumulators) and its place in the batch's work list.  Items are numbered
// match tiles first (all entries), then filter chunks (all entries).
struct BatchEntry {
    MatchArgs m;                      // tile_pitch, chunks and self_incl set; bs 4 or 8
    ZeroArgs zero;
    FilterArgs f;
    int tiles_x;                      // match items per tile row: m.tiles_x tiles, and one for the
                                      // clamped last block column where there is one
    int rows, direct;                 // the match tiles' shape: block rows, and MatchJob::direct (8 rows)
    int match_items;                  // match tiles
    int filter_items;                 // filter chunks (kBatchGroups groups each)
    long long first_match, first_filter;  // first item number of each kind
};

// A kernel argument (about 20 KB): fields come from the constant bank, where no store of the
// kernel makes the compiler load them again, and a captured launch carries its own copy.
constexpr int kBatchEntries = 48;     // entries per work list; a larger batch has several

struct BatchArgs {
    BatchEntry entries[kBatchEntries];
    int nentries;
    long long match_total, items_total;   // match items, all items
    unsigned *match_done;             // [nentries] match tiles finished
    int *status;                      // 0, or 1 when a filter chunk gave up waiting for its matching
    unsigned wait_polls;              // polls (about 0.1 us apart) before a wait gives up
    int unsatisfiable;                // testing: entry 0's chunks wait for one tile more than it has
};

// Largest dynamic shared memory of a CTA on sm_100 (227 KB), less 1 KB for static variables.
constexpr unsigned kSmemOptIn = 226 * 1024;

constexpr int kBatchGroups = 32;      // groups per filter chunk

// Fixed-point scale of the accumulators: value * 2^32 held in a signed 64-bit sum.
constexpr float kFixScale = 4294967296.0f;
constexpr float kFixInv = 2.3283064365386962890625e-10f;

}  // namespace zb
