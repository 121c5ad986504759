// zb3d_filter.cuh on the CPU (cuda_runtime.h beside this file stands in for CUDA).
//   filter8 chunk <final> <descending>   one chunk of groups (the last 8 short of 3) in one set of buffers, as the batch
//       kernel runs it, against the same groups 8 at a time in fresh buffers: equal sums or exit 1
//   filter8 sums <final> <extractor exponent>   prints how many numerators and weights are not 0
#include "cuda_runtime.h"
#include "zb3d_filter.cuh"

using namespace zb;

constexpr int W = 48, H = 40, PLANES = 3, GROUPS = 29;

struct Job {
    std::vector<float> src;
    std::vector<int2> list;
    std::vector<unsigned long long> num, den;
    FilterArgs a{};

    Job(int groups, float extractor) : src(2 * PLANES * W * H), list(groups * 8), num(PLANES * W * H), den(PLANES * W * H) {
        unsigned s = 12345;
        auto next = [&] { return (s = s * 1664525u + 1013904223u) >> 8; };
        for (float &v : src) v = next() * (1.0f / 16777216.0f);
        for (int2 &v : list) v = make_int2((int)(next() % (W - 7)), (int)(next() % (H - 7)));
        a.src = src.data();
        a.clip_stride = PLANES * W * H;
        a.plane_stride = a.frame_stride = a.acc_plane_stride = a.acc_frame_stride = W * H;
        a.w = W;
        a.h = H;
        a.pitch = W;
        a.nplanes = PLANES;
        a.list = list.data();
        a.nblocks = groups;
        for (float &v : a.sigma) v = 0.4f;
        a.extractor = extractor;
        a.num = num.data();
        a.den = den.data();
    }
};

struct Buffers {
    alignas(16) float sbuf[kFilterGroups * kGroupStride], cbuf[kFilterGroups * kGroupStride];
    long long offs[kFilterGroups * kOffStride];
};

template <bool FINAL>
void run(const FilterArgs &a, Buffers &b, long long g0, long long g1, bool descending) {
    for (int w = 0; w < kFilter8Warps; ++w)  // the warps of a CTA do not meet
        lanes::warp_run(32 * w, descending, [&] {
            for (long long g = g0; g < g1; g += kFilterGroups)
                filter8_groups<FINAL>(a, g, b.sbuf, b.cbuf, b.offs);
        });
}

template <bool FINAL>
int chunk(bool descending) {
    Job one(GROUPS, 8.0f), eight(GROUPS, 8.0f);
    auto b = std::make_unique<Buffers>();
    run<FINAL>(one.a, *b, 0, GROUPS, descending);
    for (int g = 0; g < GROUPS; g += kFilterGroups) {
        auto fresh = std::make_unique<Buffers>();
        run<FINAL>(eight.a, *fresh, g, g + kFilterGroups, descending);
    }
    return one.num == eight.num && one.den == eight.den ? 0 : 1;
}

template <bool FINAL>
int sums(int exponent) {
    Job j(kFilterGroups, std::ldexp(1.0f, exponent));
    auto b = std::make_unique<Buffers>();
    run<FINAL>(j.a, *b, 0, kFilterGroups, false);
    int n = 0, d = 0;
    for (unsigned long long v : j.num) n += v != 0;
    for (unsigned long long v : j.den) d += v != 0;
    printf("%d %d\n", n, d);
    return 0;
}

int main(int argc, char **argv) {
    if (argc != 4) return 2;
    const int final_ = atoi(argv[2]), v = atoi(argv[3]);
    if (!strcmp(argv[1], "chunk")) return final_ ? chunk<true>(v != 0) : chunk<false>(v != 0);
    return final_ ? sums<true>(v) : sums<false>(v);
}
