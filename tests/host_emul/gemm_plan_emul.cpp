// Host build of the dense GEMM's launch plan (ponyexl3_b200/csrc/exl3_gemm_plan.h), and the same choice by
// exhaustive search: every CTA count, every CTA, every segment.
#include <stdint.h>

#include "../../ponyexl3_b200/csrc/exl3_gemm_plan.h"

using namespace exl3;

extern "C" int emul_joint_beside(int64_t rows, int64_t tiles_n, int nks, int sms, int tok, int tok_wide, int room_tok, int room, int w_bytes, int most)
{
    return ts_joint(ts_plan(rows, tiles_n, nks, sms, tok, tok_wide, room_tok), tiles_n, nks, sms, TsRings{room, w_bytes}, most);
}
// K = 4
extern "C" int emul_joint(int64_t rows, int64_t tiles_n, int nks, int sms, int tok, int tok_wide, int room_tok, int most)
{
    return emul_joint_beside(rows, tiles_n, nks, sms, tok, tok_wide, room_tok, 162 * 1024, 4096, most);
}

// Every number of CTAs that may be asked for, over 16 .. 256 rows, up to sms / 2 column tiles and 2 .. most_nks k-steps: the fewest
// stages of activations beside eight of packed tiles that a cluster is left with, and clusters seen by size (seen[2 .. 8]).
extern "C" int emul_joint_stages(int most_nks, int sms, int tok, int tok_wide, int room, int w_bytes, int* seen)
{
    int least = 1 << 20;
    for (int rows = 16; rows <= 256; rows += 16)
        for (int tiles_n = 1; tiles_n <= sms / 2; tiles_n++)
            for (int nks = 2; nks <= most_nks; nks += 2) {
                const TsPlan p = ts_plan(rows, tiles_n, nks, sms, tok, tok_wide, tok_wide);
                for (int most = 8; most >= 2; most--) {
                    const int n = ts_joint(p, tiles_n, nks, sms, TsRings{room, w_bytes}, most);
                    if (!n) continue;
                    seen[n]++;
                    least = std::min(least, (room - ts_recv_bytes(p.tok, n) - 8 * w_bytes) / (128 * p.tok));
                }
            }
    return least;
}

// out: tok, tiles_m, grid, split, wide.  Shared tiles have room up to room_tok tokens.
extern "C" void emul_plan(int64_t rows, int64_t tiles_n, int nks, int sms, int tok, int tok_wide, int room_tok, int* out)
{
    const TsPlan p = ts_plan(rows, tiles_n, nks, sms, tok, tok_wide, room_tok);
    out[0] = p.tok; out[1] = p.tiles_m; out[2] = p.grid; out[3] = p.split; out[4] = p.wide;
}

extern "C" int emul_countable(int64_t rows, int64_t tiles_n, int nks, int sms, int tok, int tok_wide, int room_tok)
{
    return ts_countable(ts_plan(rows, tiles_n, nks, sms, tok, tok_wide, room_tok), tiles_n, nks);
}

static int64_t slowest(int64_t units, int nks, int g)
{
    int64_t worst = 0;
    for (int c = 0; c < g; c++) {
        int64_t u = units * c / g;
        const int64_t u1 = units * (c + 1) / g;
        int64_t t = u1 - u;
        while (u < u1) {
            const int64_t end = std::min(u1, (u / nks + 1) * nks);
            t += end - u == nks ? 6 : 10;
            u = end;
        }
        worst = std::max(worst, t);
    }
    return worst;
}

extern "C" int64_t emul_slowest(int64_t units, int nks, int g, int walk)
{
    return walk ? slowest(units, nks, g) : ts_slowest(units, nks, g, INT64_MAX);
}

extern "C" void exhaustive_plan(int64_t rows, int64_t tiles_n, int nks, int sms, int tok, int tok_wide, int room_tok, int* out)
{
    double best = -1;
    const int64_t few = (rows + tok_wide - 1) / tok_wide, many = (rows + tok - 1) / tok;
    for (int64_t n = many; n >= few; n--) {
        if (n < many - 8 && n != few) continue;
        const int t = (int)(((rows + n - 1) / n + 15) / 16 * 16);
        if (t > tok_wide) continue;
        const int tiles_m = (int)((rows + t - 1) / t);
        const int64_t tiles = tiles_m * tiles_n, units = tiles * nks;
        int grid = (int)std::min<int64_t>(tiles, sms), split = 0;
        int64_t cost = ((tiles + grid - 1) / grid) * (nks + 6);
        const int most = (int)std::min<int64_t>(sms, units / 4);
        if (t <= room_tok && tiles < 64 * (int64_t)sms && units >= 4 && units <= INT32_MAX)
            for (int g = most; g >= std::max(1, most / 2); g--) {
                const int64_t w = slowest(units, nks, g);
                if (w < cost) { cost = w; grid = g; split = 1; }
            }
        const double c = std::max(610.0, 340.0 + 2.6 * t) * (double)cost;
        if (best < 0 || c < best) {
            best = c;
            out[0] = t; out[1] = tiles_m; out[2] = grid; out[3] = split; out[4] = t > tok;
        }
    }
}
