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

// How many CTAs a dense launch of `tiles` output tiles of nks k-steps gets, and whether they share tiles.
// Cost in k-steps of the slowest CTA: its k-steps, and for each of its segments the hand-over and the
// epilogue, which the decode warps do themselves.  For shared tiles a count that lets ranges end on tile
// boundaries saves a segment per CTA, so all counts down to half of the SMs are looked at.  The choice is
// remembered per shape.
int ts_plan(int64_t tiles, int nks, int sms, int64_t rows, size_t partial_bytes, int* split)
{
    constexpr double kWhole = 6.0, kShared = 10.0;
    struct Memo { int64_t tiles; int nks, sms, room, grid, split; };
    static thread_local Memo memo[32] = {};
    static thread_local int memo_next = 0;
    sms = std::min(sms, kGemvMaxGrid);
    const int room = partial_bytes >= gemm_tile_partial_bytes(rows, sms) ? 1 : 0;
    for (const Memo& m : memo)
        if (m.tiles == tiles && m.nks == nks && m.sms == sms && m.room == room) {
            *split = m.split;
            return m.grid;
        }
    const int whole = (int)std::min<int64_t>(tiles, sms);
    int best = whole, best_split = 0;
    double best_cost = (double)((tiles + whole - 1) / whole) * (nks + kWhole);
    const int64_t units = tiles * nks;
    if (room && tiles < 64 * sms && units >= 4) {
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
            if (worst < best_cost - 1e-9) { best_cost = worst; best = g; best_split = 1; }
        }
    }
    memo[memo_next] = Memo{tiles, nks, sms, room, best, best_split};
    memo_next = (memo_next + 1) % 32;
    *split = best_split;
    return best;
}

size_t gemm_partial_bytes(int64_t rows) { return gemm_tile_partial_bytes(rows, std::min(device_sm_count(), kGemvMaxGrid)); }

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
