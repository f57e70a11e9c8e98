// Host side of the tensor-core GEMM: the plans' memory and the dispatch over K; the kernel template
// (exl3_gemm.cuh) is instantiated in exl3_gemm_k12.cu .. exl3_gemm_k78.cu.
#include "exl3_gemm.cuh"

namespace exl3 {

template <int K>
int launch_gemm_k(const GemmArgs& a, int cb, const __half* xh, const uint32_t* trellis, cudaStream_t s);
#define EXL3_DECL(K) \
    extern template int launch_gemm_k<K>(const GemmArgs&, int, const __half*, const uint32_t*, cudaStream_t);
EXL3_DECL(1) EXL3_DECL(2) EXL3_DECL(3) EXL3_DECL(4) EXL3_DECL(5) EXL3_DECL(6) EXL3_DECL(7) EXL3_DECL(8)
#undef EXL3_DECL

// The plan of a shape, remembered per thread: looking it up takes 0.02 us, planning 4 to 9 (as long as a small
// call's host path).  Of two shapes with the same slot the later one stays; 256 slots are a model's layers at some
// tens of batch sizes.
TsPlan gemm_plan(int64_t rows, int64_t tiles_n, int nks, int sms, size_t partial_bytes, int tok, int tok_wide)
{
    struct Slot { int64_t rows, tiles_n; int nks, sms, tok, tok_wide, room; TsPlan plan; };
    static thread_local Slot memo[256] = {};
    sms = std::min(sms, kGemvMaxGrid);
    // tokens of the largest tile whose partial sums fit: what the plan depends on, not the workspace's size
    const int room = (int)std::min<size_t>(tok_wide, partial_bytes / gemm_tile_partial_bytes(1, sms));
    uint64_t h = (uint64_t)rows * 0x9E3779B97F4A7C15u;
    h = (h ^ (uint64_t)tiles_n) * 0x9E3779B97F4A7C15u;
    h = (h ^ (uint64_t)nks ^ ((uint64_t)tok << 32)) * 0x9E3779B97F4A7C15u;
    Slot& m = memo[h >> 56];
    if (m.rows != rows || m.tiles_n != tiles_n || m.nks != nks || m.sms != sms || m.tok != tok || m.tok_wide != tok_wide || m.room != room)
        m = Slot{rows, tiles_n, nks, sms, tok, tok_wide, room, ts_plan(rows, tiles_n, nks, sms, tok, tok_wide, room)};
    return m.plan;
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
