// Host side of the tensor-core GEMM: the launch plan and the dispatch over K; the kernel template (exl3_gemm.cuh) is
// instantiated in exl3_gemm_k12.cu .. exl3_gemm_k78.cu.
#include "exl3_gemm.cuh"

namespace exl3 {

template <int K>
int launch_gemm_k(const GemmArgs& a, int cb, const __half* xh, const uint32_t* trellis, cudaStream_t s);
#define EXL3_DECL(K) \
    extern template int launch_gemm_k<K>(const GemmArgs&, int, const __half*, const uint32_t*, cudaStream_t);
EXL3_DECL(1) EXL3_DECL(2) EXL3_DECL(3) EXL3_DECL(4) EXL3_DECL(5) EXL3_DECL(6) EXL3_DECL(7) EXL3_DECL(8)
#undef EXL3_DECL

// How many CTAs a launch of `tiles` output tiles of nks k-steps gets, and whether they share tiles.  Cost in
// k-steps of the slowest CTA: its k-steps, and for each of its segments the hand-over and the epilogue,
// which the decode warps do themselves.  For shared tiles a count that lets ranges end on tile boundaries
// saves a segment per CTA, so all counts down to half of the SMs are looked at.
static double ts_deal(int64_t tiles, int nks, int sms, bool room, int* grid, int* split)
{
    constexpr double kWhole = 6.0, kShared = 10.0;
    const int whole = (int)std::min<int64_t>(tiles, sms);
    *grid = whole;
    *split = 0;
    double best_cost = (double)((tiles + whole - 1) / whole) * (nks + kWhole);
    const int64_t units = tiles * nks;
    if (!room || tiles >= 64 * sms || units < 4) return best_cost;
    const int most = (int)std::min<int64_t>(sms, units / 4);
    for (int g = most; g >= std::max(1, most / 2); g--) {
        double worst = 0;
        for (int c = 0; c < g; c++) {
            int64_t u = units * c / g;
            const int64_t u1 = units * (c + 1) / g;
            double t = (double)(u1 - u);
            while (u < u1) {
                const int64_t end = std::min(u1, (u / nks + 1) * nks);
                t += end - u == nks ? kWhole : kShared;
                u = end;
            }
            worst = std::max(worst, t);
        }
        if (worst < best_cost - 1e-9) { best_cost = worst; *grid = g; *split = 1; }
    }
    return best_cost;
}

// Tokens per tile: from as few tiles as wide ones allow to as few as ordinary ones need, whichever is
// cheapest at 340 + 2.6 x tokens clocks a k-step, at least 610 (measured; decoding bounds small tiles,
// the activations' way from L2 large ones).  The choice is remembered per shape.
TsPlan ts_plan(int64_t rows, int64_t tiles_n, int nks, int sms, size_t partial_bytes, int tok, int tok_wide)
{
    struct Memo { int64_t rows, tiles_n; int nks, sms, tok; size_t partial_bytes; TsPlan plan; };
    static thread_local Memo memo[32] = {};
    static thread_local int memo_next = 0;
    sms = std::min(sms, kGemvMaxGrid);
    for (const Memo& m : memo)
        if (m.rows == rows && m.tiles_n == tiles_n && m.nks == nks && m.sms == sms && m.tok == tok && m.partial_bytes == partial_bytes)
            return m.plan;
    TsPlan best = {};
    double best_cost = 0;
    const int64_t few = (rows + tok_wide - 1) / tok_wide, many = (rows + tok - 1) / tok;
    for (int64_t n = many; n >= few && n >= many - 8; n--) {
        TsPlan p = {};
        p.tok = (int)(((rows + n - 1) / n + 15) / 16 * 16);
        p.wide = p.tok > tok;
        if (p.tok > (p.wide ? tok_wide : tok)) continue;
        p.tiles_m = (int)((rows + p.tok - 1) / p.tok);
        const bool room = partial_bytes >= gemm_tile_partial_bytes(p.tok, sms);
        const double c = ts_deal(p.tiles_m * tiles_n, nks, sms, room, &p.grid, &p.split) * std::max(610.0, 340.0 + 2.6 * p.tok);
        if (best.tok == 0 || c < best_cost) { best = p; best_cost = c; }
    }
    // (many rows: the loop above looks at a few counts near the ordinary tiles'; also the widest)
    if (few < many - 8) {
        TsPlan p = {};
        p.tok = (int)(((rows + few - 1) / few + 15) / 16 * 16);
        p.wide = 1;
        if (p.tok > tok && p.tok <= tok_wide) {
            p.tiles_m = (int)((rows + p.tok - 1) / p.tok);
            const bool room = partial_bytes >= gemm_tile_partial_bytes(p.tok, sms);
            const double c = ts_deal(p.tiles_m * tiles_n, nks, sms, room, &p.grid, &p.split) * std::max(610.0, 340.0 + 2.6 * p.tok);
            if (c < best_cost) { best = p; best_cost = c; }
        }
    }
    memo[memo_next] = Memo{rows, tiles_n, nks, sms, tok, partial_bytes, best};
    memo_next = (memo_next + 1) % 32;
    return best;
}

size_t gemm_partial_bytes(int64_t rows)
{
    return gemm_tile_partial_bytes((int)std::min<int64_t>(kTsWideTok, (rows + 15) / 16 * 16), std::min(device_sm_count(), kGemvMaxGrid));
}

int launch_gemm(const GemmArgs& a, int k, int cb, const __half* xh, const uint32_t* trellis,
                cudaStream_t s)
{
    switch (k) {
        case 1: return launch_gemm_k<1>(a, cb, xh, trellis, s);
        case 2: return launch_gemm_k<2>(a, cb, xh, trellis, s);
        case 3: return launch_gemm_k<3>(a, cb, xh, trellis, s);
        case 4: return launch_gemm_k<4>(a, cb, xh, trellis, s);
        case 5: return launch_gemm_k<5>(a, cb, xh, trellis, s);
        case 6: return launch_gemm_k<6>(a, cb, xh, trellis, s);
        case 7: return launch_gemm_k<7>(a, cb, xh, trellis, s);
        case 8: return launch_gemm_k<8>(a, cb, xh, trellis, s);
        default: return EXL3_E_K;
    }
}

}  // namespace exl3
