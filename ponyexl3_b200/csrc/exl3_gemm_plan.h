// The launch plan of a dense tensor-core GEMM: tokens per output tile, number of CTAs, whether they share tiles.
// Host code without CUDA, so that tests can compile it alone.
//
// A server sees a new row count on nearly every call, so a plan has to cost about as little as a launch: the exhaustive
// search over CTA counts, CTAs and segments took 0.1 ms (16 rows) to 24 ms (8191 rows, 17408 columns).  Bounds
// leave some of the CTA counts, and the segments of a CTA are counted without walking them: 4 to 9 us, with the
// same choice (tests/test_gemm_plan.py).
#pragma once
#include <stdint.h>

#include <algorithm>

namespace exl3 {

struct TsPlan {
    int tok, tiles_m;        // tokens per output tile, tiles of tokens
    int grid, split;         // CTAs; whether they share tiles
    int wide;
};

// Costs are in k-steps of the slowest CTA: its k-steps, and for each of its segments the hand-over and the
// epilogue, which the decode warps do themselves.
constexpr int kTsWholeCost = 6, kTsSharedCost = 10;

// The least that `len` consecutive k-steps can cost, however they lie on tiles of nks.
inline int64_t ts_least(int64_t len, int nks)
{
    return len + kTsWholeCost * (len / nks) + (len % nks ? kTsSharedCost : 0);
}

// The slowest of g CTAs that take [U c/g, U (c+1)/g) of U = tiles x nks k-steps; `enough` ends the search.
inline int64_t ts_slowest(int64_t units, int nks, int g, int64_t enough)
{
    const int64_t q = units / g, q_tiles = q / nks;
    const int r = (int)(units % g), q_rest = (int)(q % nks);
    int at = 0, err = 0;                     // where in its tile a CTA starts; Bresenham's remainder
    int64_t worst = 0;
    for (int c = 0; c < g; c++) {
        err += r;
        const int more = err >= g;           // U (c+1)/g - U c/g is q or q + 1
        if (more) err -= g;
        int end = at + q_rest + more;
        int64_t ends = q_tiles;              // tile ends inside or at the end of the range
        if (end >= nks) { end -= nks; ends++; }
        const int64_t whole = ends - (at != 0 && ends > 0 ? 1 : 0);
        const int shared = ends == 0 ? 1 : (at != 0) + (end != 0);
        worst = std::max(worst, q + more + kTsWholeCost * whole + kTsSharedCost * shared);
        if (worst >= enough) break;
        at = end;
    }
    return worst;
}

// How many CTAs a launch of `tiles` output tiles of nks k-steps gets, and whether they share tiles.  For shared
// tiles a count that lets ranges end on tile boundaries saves a segment per CTA, so counts down to half of the SMs
// are looked at, as far as they can still be the best.  Returns the cost; `enough`: a cost that is of no use.
inline int64_t ts_deal(int64_t tiles, int nks, int sms, bool room, int64_t enough, int* grid, int* split)
{
    const int whole = (int)std::min<int64_t>(tiles, sms);
    *grid = whole;
    *split = 0;
    int64_t best = ((tiles + whole - 1) / whole) * (nks + kTsWholeCost);
    const int64_t units = tiles * nks;
    if (!room || tiles >= 64 * (int64_t)sms || units < 4 || units > INT32_MAX) return best;
    const int most = (int)std::min<int64_t>(sms, units / 4);
    for (int g = most; g >= std::max(1, most / 2); g--) {
        const int64_t least = ts_least((units + g - 1) / g, nks), limit = std::min(best, enough);
        if (least - 3 >= limit) break;       // (ts_least falls by 3 where a range becomes whole tiles, and only there)
        if (least >= limit) continue;
        const int64_t worst = ts_slowest(units, nks, g, limit);
        if (worst < best) { best = worst; *grid = g; *split = 1; }
    }
    return best;
}

// Tokens per tile: from as few tiles as wide ones allow to as few as ordinary ones need, whichever is cheapest at
// 340 + 2.6 x tokens clocks of 1965 MHz a k-step, at least 610.  That is fitted to the times of whole launches, the
// lower clock under the power cap included: a wide k-step takes 790 clocks, but 8192 rows run at 1.28 GHz.  One line
// serves all K: against every other number of tiles (K = 2, 4, 6, 8; 5120 x 5120, 5120 x 17408 and 17408 x 5120;
// 200 to 4096 rows) the choice is within 3 % of the best, but for 5120 x 5120 at 300 to 1000 rows, where
// one tile more would be 4 to 10 % faster.  Of many rows' counts the eight nearest to the ordinary tiles' are looked at, and the
// widest: those between them differ by less than one tile in twenty.  Tiles of up to `room` tokens may be shared.
inline TsPlan ts_plan(int64_t rows, int64_t tiles_n, int nks, int sms, int tok, int tok_wide, int room)
{
    TsPlan best = {};
    double best_cost = 0;
    auto look = [&](int64_t n) {
        TsPlan p = {};
        p.tok = (int)(((rows + n - 1) / n + 15) / 16 * 16);
        p.wide = p.tok > tok;
        if (p.tok > tok_wide) return;
        p.tiles_m = (int)((rows + p.tok - 1) / p.tok);
        const double clocks = std::max(610.0, 340.0 + 2.6 * p.tok);
        const int64_t enough = best.tok ? (int64_t)(best_cost / clocks) + 1 : INT64_MAX;     // (rounded up: the exact test follows)
        const double c = clocks * (double)ts_deal(p.tiles_m * tiles_n, nks, sms, p.tok <= room, enough, &p.grid, &p.split);
        if (best.tok == 0 || c < best_cost) { best = p; best_cost = c; }
    };
    const int64_t few = (rows + tok_wide - 1) / tok_wide, many = (rows + tok - 1) / tok;
    for (int64_t n = many; n >= few && n >= many - 8; n--) look(n);
    if (few < many - 8) look(few);
    return best;
}

// Shared memory for the rings of a dense launch, and what a k-step's packed tiles take of it.
struct TsRings {
    int room, w_bytes;
};
// Bytes into which a CTA of a cluster of n gets the other CTAs' sums: up to ceil(tok / 16 / n) pieces of sixteen tokens
// x 128 columns from each.
inline int ts_recv_bytes(int tok, int n) { return n ? (tok / 16 + n - 1) / n * (n - 1) * 16 * 128 * 4 : 0; }
// Stages of the activation ring beside them and w_stages of packed tiles.
inline int ts_x_stages(const TsRings& r, int recv_bytes, int w_stages, int x_bytes, int most)
{
    return std::min(most, (r.room - recv_bytes - w_stages * r.w_bytes) / x_bytes);
}

// CTAs per tile where a tile's CTAs should be a cluster (two to eight of them, of one tile and at least four k-steps each)
// instead of what the plan says, or 0: up to 128 tokens, and where the longer ranges of k-steps of a whole number of CTAs
// per tile cost less than the hand-over through the workspace.  us at 9, 40, 77, 128 rows, through the workspace / as
// clusters, K = 4: 5120 x 5120 (three) 15.5, 19.3, 17.7, 19.7 / 15.4, 18.5, 15.9, 17.1; 4096 x 1024 (eight) 10.8, 15.6, 16.5, 22.2 /
// 10.6, 11.6, 11.3, 12.1; 2048 x 2048 (eight) 9.4, 12.7, 13.0, 14.0 / 9.3, 10.6, 10.3, 11.4.
// The sums that they exchange take the rings' memory, most of it at 128 tokens and six or seven CTAs (80 and 96 of
// 162 KiB).  As many CTAs are taken as leave three stages of activations beside eight of packed tiles: us with two, three and four
// stages at 128 rows, 2048 -> 2560, K = 5 (seven, six, four CTAs) 12.0, 11.2, 11.2; 4096 -> 2816, K = 6 (six, five, four) 14.6, 13.7,
// 13.8.  Two stages are enough where fewer CTAs would not be worth it: 4096 -> 1024, K = 8 (eight) 12.6, through the workspace 22.3.
constexpr int kTsJointCost = 4, kTsJointMost = 8, kTsJointTok = 128, kTsJointStages = 3, kTsLeastStages = 2;
inline int ts_joint(const TsPlan& p, int64_t tiles_n, int nks, int sms, const TsRings& r, int most = kTsJointMost)
{
    const int64_t tiles = p.tiles_m * tiles_n;
    if (!p.split || p.tok > kTsJointTok || 2 * tiles > sms) return 0;
    most = (int)std::min<int64_t>(std::min<int64_t>(most, sms / tiles), nks / 4);
    if (most < 2) return 0;
    const int64_t shared = ts_slowest(tiles * nks, nks, p.grid, INT64_MAX);
    for (int least = kTsJointStages; least >= kTsLeastStages; least--) {
        int n = most;
        while (n >= 2 && ts_x_stages(r, ts_recv_bytes(p.tok, n), 8, 128 * p.tok, least) < least) n--;
        if (n >= 2 && (nks + n - 1) / n + kTsJointCost <= shared) return n;
    }
    return 0;
}

// The kernel counts tiles, k-steps where tiles are shared, and the k-steps of one CTA in 32 bits.
inline bool ts_countable(const TsPlan& p, int64_t tiles_n, int nks)
{
    const int64_t tiles = p.tiles_m * tiles_n;
    return tiles * (p.split ? nks : 1) <= INT32_MAX && (tiles + p.grid - 1) / p.grid * nks <= INT32_MAX;
}

}  // namespace exl3
