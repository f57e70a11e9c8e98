// Few tokens of a SwitchGLU: by (token, slot) pairs or by expert.  Host code without CUDA, so that tests can compile it alone.
//
// By pairs (streamed GEMV) an expert's weights are decoded once per pair; by expert (tables, rotations and two launches of
// the tile kernel) once per expert that gets any.  What the second takes goes by the slowest CTA: its tiles, 128
// columns of an expert each, are dealt to the CTAs by their place in the table, and a tile more or less on one of them
// is a third of a launch.
#pragma once
#include <stdint.h>

#include <algorithm>
#include <cmath>

namespace exl3 {

constexpr int kMoePlanCtas = 147;        // of the tile kernel on 148 SMs

// Tiles of the CTA that has most, for `hit` experts in the first slots of `sets` tables of slots x cols columns.
inline int moe_most_tiles(int64_t hit, int64_t slots, int64_t cols, int sets)
{
    int count[kMoePlanCtas] = {};
    const int64_t blocks = cols / 128, stride = 2 * ((cols + 255) / 256);
    for (int t = 0; t < sets; t++)
        for (int64_t s = 0; s < hit; s++)
            for (int64_t c = 0; c < blocks; c++) count[((t * slots + s) * stride + c) % kMoePlanCtas]++;
    return *std::max_element(count, count + kMoePlanCtas);
}

// us of the two ways with the pairs spread evenly over the experts, fitted to 1080 calls on one B200 (K = 1, 2, 3, 4, 6; 1024 .. 2048 /
// 256 .. 512 dims; 64 .. 256 experts; 6 .. 16 tokens, top-8): within 5 % rms by pairs, 3 % by expert.  By expert has to be 6 % less.  Of
// those calls it then is 2 to 3 % slower for two, and 1.65 times as quick for the best.  us by pairs / by expert, K = 4: 16 tokens of 256, 128
// and 64 experts, 2048 / 512: 132 / 118, 131 / 98, 131 / 82; 1664 / 384, 128 experts, 12 tokens: 68 / 75.
// More than 1024 experts or 2^20 pairs have no tables by expert.
inline bool moe_by_expert(int64_t pairs, int64_t experts, int64_t d, int64_t h, int k)
{
    if (experts < 1 || experts > 1024 || pairs < 1 || pairs > (1 << 20)) return false;
    const double e = (double)experts, hit = experts > 1 ? e * -std::expm1((double)pairs * std::log1p(-1.0 / e)) : 1.0;
    const int64_t used = std::max<int64_t>(1, std::llround(hit)), slots = pairs / 256 + experts;
    const double gate_up = moe_most_tiles(used, slots, h, 2) * ((double)d / 64), dn = moe_most_tiles(used, slots, d, 1), down = dn * ((double)h / 64);
    const double n = (double)pairs, nw = n * (double)d * (double)h * 1e-6;
    const double by_pairs = k <= 3 ? 12.3 + 0.887 * nw + 0.050 * n : 13.9 + 0.908 * nw + 0.044 * n;
    const double by_expert = k <= 3 ? 22.6 + 0.306 * gate_up + 0.438 * down + 1.33 * dn : 23.8 + 0.264 * gate_up + 0.404 * down + 1.44 * dn;
    return 1.06 * by_expert < by_pairs;
}

}  // namespace exl3
