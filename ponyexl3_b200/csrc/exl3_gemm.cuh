// GEMM for more than a handful of rows on the 5th-generation tensor cores, weights in tensor memory:
//   y = had( fp16( xh @ W ) ) * svh + bias,  W decoded on the fly from the packed trellis.
//
// The product is computed transposed, D[outs x tokens] = W^T x^T: the decoded weights are the A operand
// of tcgen05.mma, which may live in tensor memory.  The packed order of a 16x16 tile is the fragment
// order of W^T, and that is the register layout of tcgen05.st.16x128b, so a decoded tile goes from
// registers to tensor memory with one store and no address arithmetic, and shared memory carries only
// the activations (operand B) and the packed words.  Decoding into a swizzled operand tile in shared
// memory instead costs four scattered stores per tile and 96 bytes of operand reads per clock.
//
// Output tile: 128 columns (the width of the output rotation) x up to 256 tokens, 384 in the wide form; k-step 64.
//   warp 0      packed tiles: one 3-D TMA box of 8 x 4 tiles per k-step (ring w, as deep as shared memory allows)
//   warp 1      activations: one or more 128B-swizzled TMA boxes per k-step (ring x)
//   warp 2      issues the MMAs: A from tensor memory (eight 32-column stages; four in the wide form), B from ring x
//   warps 4-19  decode, four sets of four warps (a warp may touch the quarter of the tensor-memory
//               lanes that its index names); the sets take the k-steps in turn
// then the 16 decode warps finish the tile:
//   1. D (fp32, lane = column, register = token) is rounded to fp16 as the reference does and parked in
//      shared memory as Y[token][column] in the MN-major operand layout;
//   2. the output rotation is one more product on the tensor cores, D2[token x column] = Y H with the
//      +-1 Sylvester matrix H (exact in fp16, fp32 sums), into D's own columns;
//   3. D2 (lane = token) is scaled by 1/sqrt(128) svh, biased, and stored as 64-byte row pieces.
//
// Work is dealt in k-steps: CTA c takes the k-steps [U c/G, U (c+1)/G) of the tiles laid end to end, so a
// layer with few tiles still uses every SM.  A tile that several CTAs share is finished by the one that
// ends last: each writes its fp32 sums to its own slot of the workspace and counts itself; the last
// one adds the slots in CTA order, so the result does not depend on who came last.  (A cluster's CTAs exchange
// their sums instead, see JOINT.)  Launches over a tile table have a kernel of their own, exl3_gemm_tiles.cuh.
//
// Every mbarrier wait is bounded; a wait that gives up sets ST_TC_TIMEOUT, the thread stops waiting (so
// named barriers still meet) and the tensor memory is freed at the end.
#pragma once
#include <algorithm>
#include <cmath>

#include "exl3_gemm_plan.h"
#include "exl3_internal.h"
#include "exl3_tc.cuh"
#include "exl3_tma.h"

namespace exl3 {

constexpr int kTsDecodeWarps = 16, kTsFirstDecodeWarp = 4, kTsSets = 4;
constexpr int kTsThreads = 32 * (kTsFirstDecodeWarp + kTsDecodeWarps);
constexpr int kTsOuts = 128, kTsStepTiles = 4;      // k-step: 4 tile rows
constexpr int kTsMaxTok = 256, kTsWideTok = 384;    // tokens of a tile; of a wide one
constexpr int kTsStages = 8;                        // barriers of the k-steps in flight
// Four forms of the kernel.
//   PLAIN  for CTAs with hardly more than one tile.
//   JOINT  PLAIN where the two to eight CTAs of a tile are a thread-block cluster: each adds up a share of the tokens
//          from the others' sums, which they write into its shared memory, and finishes them.
//   AHEAD  decodes k-steps of the next tile before it finishes one.
//   WIDE   AHEAD with up to 384 tokens a tile: the weights are decoded once for all of them, and decoding
//          is what bounds the kernel.
// Tensor memory, 512 columns: PLAIN and AHEAD have two accumulators of up to 128 tokens (a tile's MMAs go on
// while the one before is finished) or one of up to 256, and eight stages of weights; WIDE has one of 384 and
// four stages.  (Four stages with 256 tokens were slower for every shape: a set of decode warps then waits for
// the MMAs of its own k-step before it can decode the next.)
enum : int { TS_PLAIN = 0, TS_AHEAD = 1, TS_WIDE = 2, TS_JOINT = 3 };
template <int MODE> struct TsForm {
    static constexpr bool kAhead = MODE == TS_AHEAD || MODE == TS_WIDE, kWide = MODE == TS_WIDE, kJoint = MODE == TS_JOINT;
    static constexpr int kStages = kWide ? 4 : 8;   // stages of the weights in tensor memory
    static constexpr int kACol0 = kWide ? 384 : 256;
};
constexpr int kTsMaxWStages = 12;
constexpr int kTsCtrlBytes = 1024;
constexpr int kTsHBytes = 128 * 128 * 2, kTsYBytes = 128 * 128 * 2;
constexpr int kTsHOff = kTsCtrlBytes, kTsYOff = kTsHOff + kTsHBytes, kTsWOff = kTsYOff + kTsYBytes;
constexpr int kTsSmemBytes = 227 * 1024;

template <int K> struct TsLayout {
    static constexpr int kTileWords = 8 * K;
    static constexpr int kWBytes = 32 * kTileWords * 4;                 // 8 x 4 packed tiles: K KiB
    static constexpr int kRoom = kTsSmemBytes - kTsWOff;                // of the two rings
    // tokens per tile of a dense launch: at least four stages of activations have to fit, three wide ones (beside a cluster's
    // exchange of sums ts_joint sees to it)
    static constexpr int kTok = std::min(kTsMaxTok, kTsSmemBytes - kTsWOff - 8 * kWBytes >= 512 * kTsMaxTok
                                                        ? kTsMaxTok
                                                        : (kTsSmemBytes - kTsWOff - 8 * kWBytes) / 512 / 16 * 16);
    static constexpr int kTokWide = std::min(kTsWideTok, (kTsSmemBytes - kTsWOff - 4 * kWBytes) / 384 / 16 * 16);
};

// Bounded wait.  It has no result, so that the code behind it stays warp-uniform for the compiler; a
// wait that gives up raises the CTA's abort word, which ends all later waits at once, and the kernel
// runs to its end without meaning.  Nothing here legitimately waits for longer than the kernels in
// front of it in the stream run.
struct TsWait {
    volatile int* abort_word;      // shared memory
    int* status;
    __device__ __forceinline__ void operator()(uint64_t* bar, uint32_t parity) const
    {
        const uint32_t b = smem_u32(bar);
        if (mbar_try_wait(b, parity)) return;
#pragma unroll 1
        for (uint32_t i = 0; i < kWaitSpins; i++) {
            if (mbar_try_wait(b, parity)) return;
            if ((i & 15u) == 15u && *abort_word) return;
        }
        *abort_word = 1;
        atomicOr(status, ST_TC_TIMEOUT);
    }
};

// ---- tensor memory as an operand and as a destination of registers ------------------------------------
// D[tmem] (+)= A[tmem] * B[smem]; issued by ONE thread.
// The four products of a k-step of 64 (16 k = 8 columns of A, 32 bytes of B each), in one
// statement: the issuing warp shares its scheduler with the decode warps, and what it takes to issue a k-step is
// what a short k-step takes.
__device__ __forceinline__ void tc_mma_kstep(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t accumulate)
{
    asm volatile(
        "{\n.reg .pred p, t;\n.reg .b32 a1, a2, a3;\n.reg .b64 b1, b2, b3;\n"
        "setp.ne.b32 p, %4, 0;\nsetp.eq.b32 t, 0, 0;\n"
        "add.s32 a1, %1, 8;\nadd.s32 a2, %1, 16;\nadd.s32 a3, %1, 24;\n"
        "add.s64 b1, %2, 2;\nadd.s64 b2, %2, 4;\nadd.s64 b3, %2, 6;\n"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [a1], b1, %3, t;\n"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [a2], b2, %3, t;\n"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [a3], b3, %3, t;\n}\n" ::"r"(d_tmem),
        "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
}
// 16 lanes x 32 columns: register 4 t + {0, 1, 2, 3} of lane l is column 8 t + {0, 0, 4, 4} + l % 4 of tensor-
// memory lane l / 4 + {0, 8, 0, 8}: four 16x16 fp16 fragments side by side.
__device__ __forceinline__ void tmem_st_16x32cols(uint32_t taddr, const uint32_t (&r)[16])
{
    asm volatile(
        "tcgen05.st.sync.aligned.16x128b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};\n" ::"r"(
            taddr),
        "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
        "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
        : "memory");
}
__device__ __forceinline__ bool elect_one()
{
    uint32_t p;
    asm volatile("{\n.reg .pred p;\nelect.sync _|p, 0xFFFFFFFF;\nselp.u32 %0, 1, 0, p;\n}\n" : "=r"(p));
    return p != 0;
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory"); }
// 16 consecutive fp32 columns of this thread's tensor-memory lane.
__device__ __forceinline__ void tmem_ld_16cols(uint32_t taddr, float (&v)[16])
{
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n"
        "tcgen05.wait::ld.sync.aligned;\n"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr)
        : "memory");
#pragma unroll
    for (int i = 0; i < 16; i++) v[i] = __uint_as_float(r[i]);
}

// 16 bytes that no earlier kernel of the stream writes; volatile, so that the load stays where it is written.
__device__ __forceinline__ uint4 ldg_nc_128(const __half* p)
{
    uint4 v;
    asm volatile("ld.global.nc.v4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}

// One 32-byte store (sm_100: 256-bit vector stores); p must be 32-byte aligned.
__device__ __forceinline__ void st_global_256(void* p, const uint4& a, const uint4& b)
{
    asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(p), "r"(a.x), "r"(a.y), "r"(a.z), "r"(a.w),
                 "r"(b.x), "r"(b.y), "r"(b.z), "r"(b.w)
                 : "memory");
}

// Two codewords -> (w_a, w_b) fp16, with the XOR constant as a run-time value (one LOP3).  Each word's
// halves are added by a broadcasting HADD2 and one byte permute joins the two sums.  Gathering the halves
// with two byte permutes and adding once is one operation on either side too, but the logic pipe bounds
// the decode (14 of its clocks per tile that way, 11 this way) and the multiplier pipe is half empty.
template <int CB> __device__ __forceinline__ uint32_t decode_pair_rt(uint32_t cw_a, uint32_t cw_b, uint32_t xc)
{
    const uint32_t xa = codebook_word_rt<CB>(cw_a, xc), xb = codebook_word_rt<CB>(cw_b, xc);
    if (CB == CB_MUL1) {
        const uint32_t s = xa | (xb << 16);
        return h2_as_u32(__hfma2(u32_as_h2(s), u32_as_h2(0x1EEE1EEEu), u32_as_h2(0xC931C931u)));
    }
    const __half2 ha = u32_as_h2(xa), hb = u32_as_h2(xb);
    return __byte_perm(h2_as_u32(__hadd2(__low2half2(ha), __high2half2(ha))),
                       h2_as_u32(__hadd2(__low2half2(hb), __high2half2(hb))), 0x5410);
}

// MN-major operand in the 128-byte-swizzled layout: 64 elements of the M (or N) index per 128-byte row,
// one row per k, 8-row groups 1024 bytes apart, the next 64 elements 128 rows (16 KiB) further on.
__device__ __forceinline__ uint64_t smem_desc_mn_sw128(uint32_t smem_addr)
{
    uint64_t d = 0;
    d |= (uint64_t)((smem_addr & 0x3FFFFu) >> 4);
    d |= (uint64_t)(16384 >> 4) << 16;
    d |= (uint64_t)(1024 >> 4) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)2 << 61;
    return d;
}
constexpr uint32_t kIdescMajorA = 1u << 15;          // A is MN-major

// ---- the output rotation of 128 tokens: D2 = Y H ---------------------------------------------------------
// B operand H[n][k] = (-1)^popcount(n & k), K-major: two 64-wide halves of k, 128 rows of 128 bytes each.  (As H64 and
// -H64, half of it, with products of 64 columns: room for more packed tiles, but MLP of 300 rows 188.6 -> 190.8 us.)
// (The decode warps do this before they decode.  A word's pattern depends on the low three bits of n, which are the same for
// all of a thread's pieces if `threads` is a multiple of 64: 8 of the 12 bit counts a thread are made once.  With all 36, at a
// quarter of the ordinary rate, every launch took 0.2 to 0.4 us longer: 6784 -> 768 at 330 rows 28.5 us, this way 28.1.  UNROLL
// pieces at a time: all four in the forms whose tail is long; one in JOINT, which runs for a tile only and is the quicker
// the less code it has to fetch, K = 1, 5120 x 5120 at 77 rows 16.9 / 16.6.)
template <int UNROLL> __device__ __forceinline__ void store_sylvester(uint8_t* h_mat, int thread, int threads)
{
    uint32_t w[4];
    const int n_low = (thread >> 3) & 7;
#pragma unroll
    for (int j = 0; j < 4; j++)
        w[j] = 0x3C003C00u | ((__popc(n_low & (2 * j)) & 1) ? 0x8000u : 0u) | ((__popc(n_low & (2 * j + 1)) & 1) ? 0x80000000u : 0u);
#pragma unroll UNROLL
    for (int i = thread; i < 2048; i += threads) {
        const int kh = i >> 10, n = (i >> 3) & 127, ch = i & 7;
        const uint32_t flip = (__popc(n & (64 * kh + 8 * ch)) & 1) ? 0x80008000u : 0u;
        *reinterpret_cast<uint4*>(h_mat + kh * 16384 + n * 128 + ((ch ^ (n & 7)) << 4)) = make_uint4(w[0] ^ flip, w[1] ^ flip, w[2] ^ flip, w[3] ^ flip);
    }
}
// Issued by ONE thread; `done` gets one arrival when the product is complete.
__device__ __forceinline__ void rotate_tile(uint32_t d_tmem, uint32_t y_buf, uint32_t h_mat, uint32_t done)
{
    const uint64_t yd = smem_desc_mn_sw128(y_buf), hd = smem_desc_sw128(h_mat);
#pragma unroll
    for (int kk = 0; kk < 8; kk++)
        tc_mma_f16(d_tmem, yd + 128 * kk, hd + (kk >> 2) * 1024 + (kk & 3) * 2, mma_idesc_f16(128, 128) | kIdescMajorA, kk > 0 ? 1u : 0u);
    tc_commit(done);
}

// One stretch of k-steps of one output tile.
struct TsSeg {
    int m0, rows;            // first row of xh, rows in use
    int tn0;                 // first tile column of the trellis
    int sv_off, y_col, y_row_delta;
    int k0, k1;              // k-steps
    int tile;                // tile number (dense launches)
    int member;              // sibling group: which member's output
    int first;               // first segment of this CTA's range
};

// The segments of one CTA, the same sequence for every role.
template <bool TABLE> struct TsWalk {
    // The same value in every lane already; the reduction tells the compiler, because its result is a uniform
    // register.  (Behind a shuffle or a 64-bit division all of the issuing warps' loop control and descriptors
    // lived in ordinary registers and were moved over for every instruction: 5 to 9 % of the kernel.)
    static __device__ __forceinline__ int uniform(int v) { return __reduce_max_sync(0xFFFFFFFFu, v); }
    int tile0, u, u1, u0;     // dense: the CTA's first tile; next, end and first k-step of its range, counted from that tile's
    // tables: a warp looks at 32 of its CTA's items at a time, one per lane, and takes those in use in turn
    int item;                 // first item not looked at yet
    uint32_t found;           // items in use among those looked at last
    int4 p, q;                // this lane's
    int it;
    __device__ __forceinline__ void start(const GemmArgs& a)
    {
        item = (int)blockIdx.x;
        found = 0;
        const int64_t g = gridDim.x, c = blockIdx.x, nks = a.t_in >> 2;
        if (a.ts_split) {
            const int k0 = (int)(a.n_items * nks * c / g), k1 = (int)(a.n_items * nks * (c + 1) / g);
            tile0 = uniform(k0 / (int)nks);
            u0 = uniform(k0 - tile0 * (int)nks);
            u1 = uniform(k1 - tile0 * (int)nks);
        } else {
            tile0 = uniform((int)(a.n_items * c / g));
            u0 = 0;
            u1 = uniform(((int)(a.n_items * (c + 1) / g) - tile0) * (int)nks);
        }
        u = u0;
    }
    __device__ __forceinline__ bool next(const GemmArgs& a, TsSeg& s)
    {
        const int nks = a.t_in >> 2;
        if (TABLE) {
            // Items: column halves of the table's tiles, then once more for the second part of tiles with more
            // rows than ts_tok (parts of equal size).
            while (!found) {
                if (item >= a.n_items) return false;
                it = item + (int)(threadIdx.x & 31) * (int)gridDim.x;
                const int per_part = 2 * a.n_tiles_tab, part = it / per_part, e = it - part * per_part, h = e & 1;
                bool used = it < a.n_items;
                if (used) {
                    p = reinterpret_cast<const int4*>(a.tile_tab)[e & ~1];
                    q = reinterpret_cast<const int4*>(a.tile_tab)[e | 1];
                    const int rows = p.y - p.x, parts = (rows + a.ts_tok - 1) / a.ts_tok;
                    used = rows > 0 && 128 * h < q.y && part < parts;
                    if (used) {
                        const int size = ((rows + parts - 1) / parts + 15) & ~15;
                        p.x += part * size;
                        p.y = min(size, p.y - p.x);                // now: rows of the part
                        used = p.y > 0;
                        p.z += 8 * h; p.w += 128 * h; q.x += 128 * h;
                    }
                }
                found = __ballot_sync(0xFFFFFFFFu, used);
                item += 32 * (int)gridDim.x;
            }
            const int l = __ffs(found) - 1;
            found &= found - 1;
            s.m0 = uniform(__shfl_sync(0xFFFFFFFFu, p.x, l));
            s.rows = uniform(__shfl_sync(0xFFFFFFFFu, p.y, l));
            s.tn0 = uniform(__shfl_sync(0xFFFFFFFFu, p.z, l));
            s.sv_off = __shfl_sync(0xFFFFFFFFu, p.w, l);
            s.y_col = __shfl_sync(0xFFFFFFFFu, q.x, l);
            s.y_row_delta = __shfl_sync(0xFFFFFFFFu, q.z, l);
            s.tile = __shfl_sync(0xFFFFFFFFu, it, l);
            s.k0 = 0; s.k1 = nks; s.first = 1; s.member = 0;
            return true;
        }
        if (u >= u1) return false;
        s.first = u == u0;
        s.tile = tile0 + uniform(u / nks);
        s.k0 = u - (s.tile - tile0) * nks;
        s.k1 = min(nks, s.k0 + (u1 - u));
        u += s.k1 - s.k0;
        const int tn = uniform(s.tile / a.tiles_m), tm = s.tile - tn * a.tiles_m;
        s.m0 = tm * a.ts_tok;
        s.rows = min(a.ts_tok, a.m - s.m0);
        s.tn0 = 8 * tn;
        s.sv_off = s.y_col = 128 * tn;
        s.y_row_delta = 0;
        s.member = 0;
        if (a.n_members > 1) {
            while (tn >= a.member_end[s.member]) s.member++;
            if (s.member) s.y_col -= 128 * a.member_end[s.member - 1];
            s.m0 += s.member * a.m;
            s.y_row_delta = -s.member * a.m;
        }
        return true;
    }
};

// Last step of a tile's finishing: D2 (lane = token) scaled, biased and stored; this warp's 32 columns.  `drained` is called when
// tensor memory has been read.
template <typename Drained>
__device__ __forceinline__ void store_rotated(const GemmArgs& a, const TsSeg& sg, bool used, int orow, uint32_t lane_base, int set,
                                              uint64_t* h_full, uint32_t hpar, const TsWait& wait, Drained&& drained)
{
    __half* yp = nullptr;
    if (used) {
        const int col0 = sg.y_col + 32 * set;
        yp = a.n_members > 1 ? a.member_y[sg.member] + (int64_t)orow * a.member_stride[sg.member] + col0
                             : a.y + (int64_t)orow * a.y_row_stride + col0;
    }
    // The output scales are fetched behind the product: between the stores below, which might alias
    // them, the loads would be made and waited for one after the other, and a prefetch into L1 does
    // not help.
    uint4 sv[4];
#pragma unroll
    for (int c = 0; c < 4; c++)
        sv[c] = a.svh ? ldg_nc_128(a.svh + sg.sv_off + 32 * set + 8 * c)
                      : make_uint4(0x3C003C00u, 0x3C003C00u, 0x3C003C00u, 0x3C003C00u);
    wait(h_full, hpar);
    tc_fence_after_sync();
    float f[32];
    tmem_ld_32cols(lane_base + 32 * set, f);
    drained();
    if (!used) return;
    const uint64_t scale = f32x2(EXL3_HAD_SCALE, EXL3_HAD_SCALE);
    uint4 held16 = make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
    for (int c = 0; c < 4; c++) {
        const uint32_t sw4[4] = {sv[c].x, sv[c].y, sv[c].z, sv[c].w};
        uint32_t h[4];
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const float2 w2 = __half22float2(u32_as_h2(sw4[i]));
            h[i] = f16_pair(mul_f32x2(mul_f32x2(f32x2(f[8 * c + 2 * i], f[8 * c + 2 * i + 1]), scale), f32x2(w2.x, w2.y)));
        }
        if (a.bias) {
            const uint4 bv = __ldg(reinterpret_cast<const uint4*>(a.bias + sg.sv_off + 32 * set + 8 * c));
            const uint32_t bw[4] = {bv.x, bv.y, bv.z, bv.w};
#pragma unroll
            for (int i = 0; i < 4; i++) h[i] = h2_as_u32(__hadd2(u32_as_h2(h[i]), u32_as_h2(bw[i])));
        }
        const uint4 ov = make_uint4(h[0], h[1], h[2], h[3]);
        if (!a.y_wide) {
            *reinterpret_cast<uint4*>(yp + 8 * c) = ov;
        } else if (c & 1) {
            st_global_256(yp + 8 * (c - 1), held16, ov);   // whole sectors
        } else {
            held16 = ov;
        }
    }
}

template <int K, int CB, int MODE>
__global__ void __launch_bounds__(kTsThreads, 1)
    gemm_kernel(const GemmArgs a, const __grid_constant__ CUtensorMap tm_x, const __grid_constant__ CUtensorMap tm_w)
{
    using L = TsLayout<K>;
    using F = TsForm<MODE>;
    constexpr int NS = F::kStages;
    extern __shared__ __align__(1024) uint8_t smem[];
    uint64_t* w_full = reinterpret_cast<uint64_t*>(smem);      // packed tiles landed                     [12]
    uint64_t* w_empty = w_full + kTsMaxWStages;               // ... read by the set's four warps         [12]
    uint64_t* full = w_empty + kTsMaxWStages;                   // weights decoded AND activations landed    [8]
    uint64_t* empty = full + kTsStages;                       // the k-step's MMAs are done                [8]
    uint64_t* d_full = empty + kTsStages;                      // a segment's sums are complete             [2]
    uint64_t* d_empty = d_full + 2;                            // ... and drained                          [2]
    uint64_t* h_full = d_empty + 2;                            // the rotated tile is complete
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(h_full + 1);
    volatile int* handoff = reinterpret_cast<volatile int*>(tmem_slot + 2);
    const TsWait wait{reinterpret_cast<volatile int*>(tmem_slot + 1), a.status};
    uint8_t* h_mat = smem + kTsHOff;
    uint8_t* y_buf = smem + kTsYOff;
    uint8_t* recv = smem + kTsWOff;                            // JOINT: sums from the tile's other CTAs
    uint8_t* w_ring = smem + kTsWOff + (F::kJoint ? a.ts_recv_bytes : 0);
    const int nw = a.ts_w_stages;                              // depth of ring w, a multiple of the sets
    uint8_t* x_ring = w_ring + nw * L::kWBytes;

    using Walk = TsWalk<false>;
    const int tid = threadIdx.x, warp = Walk::uniform(tid >> 5), lane = tid & 31;
    const int nx = a.stages, x_bytes = a.ts_x_bytes;           // depth and stage size of ring x
    Walk walk;
    walk.start(a);
    TsSeg sg;

    if (warp == 0) {                                           // (one thread's 40 to 60 barriers took 0.3 us)
        if (lane < nw) {
            mbar_init(smem_u32(&w_full[lane]), 1);
            mbar_init(smem_u32(&w_empty[lane]), 4);
        }
        if (lane < kTsStages) {
            mbar_init(smem_u32(&full[lane]), 5);               // a set's four warps and the activations' copy
            mbar_init(smem_u32(&empty[lane]), 1);
        }
        if (lane < 2) {
            mbar_init(smem_u32(&d_full[lane]), 1);
            mbar_init(smem_u32(&d_empty[lane]), kTsDecodeWarps);
        }
        if (lane == 0) {
            mbar_init(smem_u32(h_full), 1);
            *wait.abort_word = 0;
        }
        mbar_fence_init();
    }
    if (warp == 2) tmem_alloc(smem_u32(tmem_slot), 512);
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem_base = (uint32_t)Walk::uniform((int)*tmem_slot);
    if (F::kJoint) cluster_arrive_relaxed();                   // "my shared memory is there"
    griddep_launch_dependents();

    // The three single-issuer roles run as whole warps with one elected lane issuing: loop control,
    // addresses and descriptors then stay in uniform registers, where TMA and tcgen05.mma take them.
    // Written as one lane's code, an MMA k-step took 570 clocks to issue and a TMA box about 200.
    if (warp == 0) {
        // ------------------------------------------------------------------ packed tiles ----
        const bool leader = elect_one();
        if (leader) tma_prefetch_desc(&tm_w);
        int s = 0;
        uint32_t parity = 1;                                   // (a wait for the phase before the first passes)
        while (walk.next(a, sg)) {
            for (int ks = sg.k0; ks < sg.k1; ks++) {
                wait(&w_empty[s], parity);
                if (leader) {
                    const uint32_t bar = smem_u32(&w_full[s]);
                    mbar_arrive_expect_tx(bar, L::kWBytes);
                    tma_load_3d(smem_u32(w_ring) + s * L::kWBytes, &tm_w, 0, sg.tn0, kTsStepTiles * ks, bar);
                }
                if (++s == nw) { s = 0; parity ^= 1u; }
            }
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------------- activations ----
        const bool leader = elect_one();
        if (leader) tma_prefetch_desc(&tm_x);
        griddep_wait();
        const int box_rows = a.ts_box_rows, box_bytes = box_rows * 128;
        // The copy counts on the barrier of the k-step's tensor-memory stage.  A stage of this ring is free
        // when the MMAs of the k-step nx before are done (nx <= 8: that barrier cannot be a turn ahead).
        int s = 0, v = 0;
        while (walk.next(a, sg)) {
            const int boxes = (sg.rows + box_rows - 1) / box_rows;
            for (int ks = sg.k0; ks < sg.k1; ks++, v++) {
                const int u = v - nx;
                if (u >= 0) wait(&empty[u & (kTsStages - 1)], (uint32_t)(u / kTsStages) & 1u);
                if (leader) {
                    const uint32_t bar = smem_u32(&full[v & (kTsStages - 1)]);
                    const uint32_t dst = smem_u32(x_ring) + (uint32_t)(s * x_bytes);
                    mbar_arrive_expect_tx(bar, (uint32_t)(boxes * box_bytes));
                    tma_load_2d(dst, &tm_x, ks * 64, sg.m0, bar);
                    for (int b = 1; b < boxes; b++)
                        tma_load_2d(dst + b * box_bytes, &tm_x, ks * 64, sg.m0 + box_rows * b, bar);
                }
                if (++s == nx) s = 0;
            }
        }
    } else if (warp == 2) {
        // -------------------------------------------------------------------- MMA issuer ----
        const bool leader = elect_one();
        int xs = 0, as = 0, db = 0, v = 0;
        uint32_t dpar = 1;
        const uint32_t x0 = smem_u32(x_ring);
        while (walk.next(a, sg)) {
            wait(&d_empty[db], dpar);
            tc_fence_after_sync();
            const uint32_t d_tmem = tmem_base + (uint32_t)(128 * db);
            // (an MMA takes at most 256 tokens: a wide tile is two halves)
            const int n16 = (sg.rows + 15) & ~15, n0 = F::kWide ? ((n16 >> 1) + 15) & ~15 : n16, n1 = n16 - n0;
            const uint32_t idesc = mma_idesc_f16(128, n0), idesc1 = mma_idesc_f16(128, n1);
            uint32_t accum = 0;
            for (int ks = sg.k0; ks < sg.k1; ks++, v++) {
                const uint32_t at = tmem_base + F::kACol0 + 32 * as;
                const uint64_t xd = smem_desc_sw128(x0 + (uint32_t)(xs * x_bytes));
                wait(&full[v & (kTsStages - 1)], (uint32_t)(v / kTsStages) & 1u);
                tc_fence_after_sync();
                if (leader) {
                    tc_mma_kstep(d_tmem, at, xd, idesc, accum);
                    if (F::kWide && n1 > 0) tc_mma_kstep(d_tmem + n0, at, xd + (uint64_t)(8 * n0), idesc1, accum);   // n0 rows of 128 bytes further
                    tc_commit(smem_u32(&empty[v & (kTsStages - 1)]));
                }
                accum = 1u;
                if (++xs == nx) xs = 0;
                if (++as == NS) as = 0;
            }
            if (leader) tc_commit(smem_u32(&d_full[db]));
            if (++db == a.ts_dbuf) { db = 0; dpar ^= 1u; }
        }
    } else if (warp >= kTsFirstDecodeWarp) {
        // ------------------------------------------------- decode, and finish the tiles ----
        const int q = warp & 3, set = (warp - kTsFirstDecodeWarp) >> 2;
        const int dt = tid - 32 * kTsFirstDecodeWarp;
        const int prev_word = (lane + 31) & 31;
        const uint32_t xc = a.cb_xor;
        const int nks = a.t_in >> 2;
        LaneWords<K> lw;
        lw.init(lane);
        store_sylvester<F::kJoint ? 1 : 4>(h_mat, dt, 512);
        // A set decodes its k-steps in order, whatever tiles they belong to.  With AHEAD the warps decode as many
        // k-steps of the next tile as there are stages before they finish one, so that the tensor core has work
        // in the meantime; a CTA with hardly more than one tile is 1 us quicker without.
        int kc = 0, v = set, ws = set;                             // end of the current tile's k-steps; next one of this set, its ring stage
        uint32_t w_par = 0;
        int db = 0;
        uint32_t dpar = 0, hpar = 0;
        TsSeg nx_sg;
        bool more = walk.next(a, nx_sg);
        while (more) {
            sg = nx_sg;
            more = walk.next(a, nx_sg);
            const int n_steps = sg.k1 - sg.k0;
            kc += n_steps;
            const int v_end = kc + (F::kAhead && more ? min(NS, nx_sg.k1 - nx_sg.k0) : 0);
            for (; v < v_end; v += kTsSets) {
                // Four sets, and a multiple of them in stages of ring w and of tensor memory: a stage always belongs to the
                // same set.  (With another number a set could look at a barrier two phases early and read a stale parity.)
                const int st = v & (NS - 1), vb = v - NS;      // vb: the k-step that had the stage before
                wait(&w_full[ws], w_par);
                const uint32_t* wt = reinterpret_cast<const uint32_t*>(w_ring + ws * L::kWBytes) + 2 * q * L::kTileWords;
                auto tile_frag = [&](const uint32_t (&cw)[8], uint32_t* f) {
                    f[0] = decode_pair_rt<CB>(cw[0], cw[1], xc);
                    f[1] = decode_pair_rt<CB>(cw[4], cw[5], xc);
                    f[2] = decode_pair_rt<CB>(cw[2], cw[3], xc);
                    f[3] = decode_pair_rt<CB>(cw[6], cw[7], xc);
                };
                auto await_operand = [&]() {
                    if (vb >= 0) wait(&empty[vb & (kTsStages - 1)], (uint32_t)(vb / kTsStages) & 1u);
                    tc_fence_after_sync();
                };
                const uint32_t a_tmem = tmem_base + ((uint32_t)(32 * q) << 16) + F::kACol0 + 32 * st;
                // Tile columns 2q, 2q + 1 of all four tile rows, one after the other.  As a loop, half the code leaves the issuing
                // warps and a short call's start more of the instruction cache: for JOINT, whose CTAs have few k-steps, and for
                // K = 1.  Elsewhere the loop costs long ranges more than it gives short ones: us as a loop / unrolled / before
                // there was a loop, 5120 x 17408: K = 3, 200 rows 39.9 / 38.9 / 38.9, K = 5, 64 rows 35.1 / 33.0 / 35.6; 512 x 512,
                // K = 5, 64 rows 8.2 / 8.2 / 8.3.  The wide form, whose sets mostly wait for MMAs, reads all words first and is 2 %
                // quicker with it (an MLP of 300 rows).
                if constexpr (F::kWide) {
                    uint32_t pw[2][4][K == 4 ? 4 : 3];
#pragma unroll
                    for (int h = 0; h < 2; h++)
#pragma unroll
                        for (int tk = 0; tk < 4; tk++) {
                            const uint32_t* tw = wt + (tk * 8 + h) * L::kTileWords;
                            if constexpr (K == 4) {
                                pw[h][tk][0] = tw[lane];
                                pw[h][tk][1] = tw[prev_word];
                                pw[h][tk][2] = reinterpret_cast<const uint16_t*>(tw)[2 * lane];        // the two 16-bit aligned
                                pw[h][tk][3] = reinterpret_cast<const uint16_t*>(tw)[2 * lane + 1];    // windows
                            } else {
                                pw[h][tk][0] = tw[lw.i0];
                                pw[h][tk][1] = tw[lw.i1];
                                pw[h][tk][2] = LaneWords<K>::kThree ? tw[lw.i2] : 0u;
                            }
                        }
                    await_operand();
#pragma unroll
                    for (int h = 0; h < 2; h++) {
                        uint32_t frag[16];
#pragma unroll
                        for (int tk = 0; tk < 4; tk++) {
                            const auto& p = pw[h][tk];
                            uint32_t cw[8];
                            if constexpr (K == 4) lane_codewords_k4_halves(p[0], p[1], p[2], p[3], cw);
                            else lane_codewords<K>(p[0], p[1], p[2], lw.sh, cw);
                            tile_frag(cw, frag + 4 * tk);
                        }
                        tmem_st_16x32cols(a_tmem + ((uint32_t)(16 * h) << 16), frag);
                    }
                } else {
                    constexpr int kUnroll = F::kJoint || K == 1 ? 1 : 2;
#pragma unroll kUnroll
                    for (int h = 0; h < 2; h++) {
                        uint32_t frag[16];
#pragma unroll
                        for (int tk = 0; tk < 4; tk++) {
                            const uint32_t* tw = wt + (tk * 8 + h) * L::kTileWords;
                            uint32_t cw[8];
                            if constexpr (K == 4) lane_codewords_k4(tw[lane], tw[prev_word], cw);
                            else lane_codewords<K>(tw[lw.i0], tw[lw.i1], LaneWords<K>::kThree ? tw[lw.i2] : 0u, lw.sh, cw);
                            tile_frag(cw, frag + 4 * tk);
                        }
                        if (h == 0) await_operand();
                        tmem_st_16x32cols(a_tmem + ((uint32_t)(16 * h) << 16), frag);
                    }
                }
                // Only now is it certain that the packed words have been read: the stores above depend on them.  (With
                // the slot given back before the wait for `empty`, some loads were found to take place after it, and
                // to see the words of a later k-step.)
                __syncwarp();
                if (lane == 0) mbar_arrive(smem_u32(&w_empty[ws]));
                if ((ws += kTsSets) >= nw) { ws = set; w_par ^= 1u; }
                tmem_st_wait();
                tc_fence_before_sync();
                __syncwarp();
                if (lane == 0) mbar_arrive(smem_u32(&full[v & (kTsStages - 1)]));
            }

            // ---- finish the tile: what it needs from global memory first ----
            const int out = 32 * q + lane;                         // this thread's column of the tile
            const int n16 = (sg.rows + 15) >> 4;
            // a shared tile's first and last contributor (64-bit divisions, done behind the last MMAs)
            int cf = 0, cl = 0, slot_first = 0;
            if (n_steps != nks && dt == 0) {
                const int64_t U = (int64_t)a.n_items * nks, G = gridDim.x, f = (int64_t)sg.tile * nks;
                cf = (int)(((f + 1) * G - 1) / U);
                cl = (int)(((f + nks) * G - 1) / U);
                slot_first = U * cf / G == f ? 0 : 1;
            }
            wait(&d_full[db], dpar);
            tc_fence_after_sync();
            const uint32_t d_tmem = tmem_base + (uint32_t)(128 * db);
            const uint32_t lane_base = d_tmem + ((uint32_t)(32 * q) << 16);
            const size_t slot_floats = (size_t)kTsOuts * a.ts_tok;
            bool held = true;
            auto release_d = [&]() {                               // the next tile's MMAs may go into this D
                if (!held) return;
                held = false;
                tc_fence_before_sync();
                __syncwarp();
                if (lane == 0) mbar_arrive(smem_u32(&d_empty[db]));
            };
            if constexpr (F::kJoint) {
                // The tile's CTAs share its tokens out, sixteen at a time: chunk ch is CTA ch % n's.  The sums go to their
                // owners as they lie in tensor memory, [source][chunk][four tokens][column].
                const int n = a.ts_joint, rank = (int)(blockIdx.x % (unsigned)n), most = (a.ts_tok / 16 + n - 1) / n;
                cluster_wait();
                for (int ch = set; ch < n16; ch += kTsSets) {
                    const int owner = ch % n;
                    if (owner == rank) continue;
                    float f[16];
                    tmem_ld_16cols(lane_base + 16 * ch, f);
                    const int src = rank < owner ? rank : rank - 1;
                    const uint32_t dst = cluster_address(smem_u32(recv) + (uint32_t)(((src * most + ch / n) * 4 * kTsOuts + out) * 16), owner);
#pragma unroll
                    for (int i = 0; i < 4; i++) st_cluster_f32x4(dst + i * kTsOuts * 16, make_float4(f[4 * i], f[4 * i + 1], f[4 * i + 2], f[4 * i + 3]));
                }
                __syncwarp();
                cluster_sync();
                const int own = n16 > rank ? (n16 - rank + n - 1) / n : 0;
                if (own == 0) continue;                            // (nothing follows: a CTA has one tile)
                for (int o = set; o < own; o += kTsSets) {
                    float v[16], f[16];
                    tmem_ld_16cols(lane_base + 16 * (rank + o * n), v);
#pragma unroll
                    for (int i = 0; i < 16; i++) f[i] = 0.f;
                    for (int j = 0; j < n; j++) {                  // in CTA order
                        if (j == rank) {
#pragma unroll
                            for (int i = 0; i < 16; i++) f[i] += v[i];
                            continue;
                        }
                        const float4* part = reinterpret_cast<const float4*>(recv) + ((j < rank ? j : j - 1) * most + o) * 4 * kTsOuts + out;
#pragma unroll
                        for (int i = 0; i < 4; i++) {
                            const float4 u = part[i * kTsOuts];
                            f[4 * i] += u.x; f[4 * i + 1] += u.y; f[4 * i + 2] += u.z; f[4 * i + 3] += u.w;
                        }
                    }
                    uint32_t hv[8];
#pragma unroll
                    for (int i = 0; i < 8; i++) hv[i] = h2_as_u32(__floats2half2_rn(f[2 * i], f[2 * i + 1]));
                    uint8_t* row = y_buf + (o >> 2) * 16384 + out * 128;
                    const int piece = 2 * (o & 3), sw = out & 7;
                    *reinterpret_cast<uint4*>(row + ((piece ^ sw) << 4)) = make_uint4(hv[0], hv[1], hv[2], hv[3]);
                    *reinterpret_cast<uint4*>(row + (((piece + 1) ^ sw) << 4)) = make_uint4(hv[4], hv[5], hv[6], hv[7]);
                }
                fence_proxy_async_smem();
                tc_fence_before_sync();
                named_bar_sync(1, 512);
                if (warp == kTsFirstDecodeWarp) {
                    tc_fence_after_sync();
                    if (elect_one()) rotate_tile(d_tmem, smem_u32(y_buf), smem_u32(h_mat), smem_u32(h_full));
                    __syncwarp();
                }
                const int row = 16 * (rank + (out >> 4) * n) + (out & 15);       // lane = token now
                const bool used = out < 16 * own && row < sg.rows;
                store_rotated(a, sg, used, sg.m0 + row + sg.y_row_delta, lane_base, set, h_full, hpar, wait, [] {});
                continue;
            }
            bool finish = true;
            int c_first = 0, n_contrib = 1;
            if (n_steps != nks) {
                float4* part = reinterpret_cast<float4*>(a.ts_partials + (size_t)(2 * blockIdx.x + (sg.first ? 0 : 1)) * slot_floats) + out;
                for (int ch = set; ch < n16; ch += kTsSets) {
                    float f[16];
                    tmem_ld_16cols(lane_base + 16 * ch, f);
#pragma unroll
                    for (int i = 0; i < 4; i++)
                        __stcg(part + (4 * ch + i) * kTsOuts, make_float4(f[4 * i], f[4 * i + 1], f[4 * i + 2], f[4 * i + 3]));
                }
                named_bar_sync(1, 512);
                if (dt == 0) {
                    // as in the streamed GEMV: the barrier orders the CTA's stores before this release, the
                    // count wraps to zero with the last arrival and is an acquire for the reads below
                    unsigned old;
                    asm volatile("atom.acq_rel.gpu.global.inc.u32 %0, [%1], %2;"
                                 : "=r"(old) : "l"(a.ts_ctr + cf), "r"((unsigned)(cl - cf)) : "memory");
                    handoff[0] = old == (unsigned)(cl - cf) ? 1 : 0;
                    handoff[1] = cf;
                    handoff[2] = cl - cf + 1;
                    handoff[3] = slot_first;
                }
                named_bar_sync(1, 512);
                finish = handoff[0] != 0;
                c_first = handoff[1];
                n_contrib = handoff[2];
                slot_first = handoff[3];
            }
            if (finish) {
                // The rotated half goes over D's first 128 columns, which have been read by then.
#pragma unroll 1
                for (int tg = 0; 128 * tg < sg.rows; tg++) {       // 128 tokens at a time
                    if (n_steps == nks) {
#pragma unroll 1
                        for (int ch = 8 * tg + set; ch < min(8 * tg + 8, n16); ch += kTsSets) {
                            float f[16];
                            tmem_ld_16cols(lane_base + 16 * ch, f);
                            uint32_t hv[8];
#pragma unroll
                            for (int i = 0; i < 8; i++) hv[i] = h2_as_u32(__floats2half2_rn(f[2 * i], f[2 * i + 1]));
                            const int c16 = ch & 7;                // 16 tokens = two 16-byte pieces of a 64-token row
                            uint8_t* row = y_buf + (c16 >> 2) * 16384 + out * 128;
                            const int piece = 2 * (c16 & 3), sw = out & 7;
                            *reinterpret_cast<uint4*>(row + ((piece ^ sw) << 4)) = make_uint4(hv[0], hv[1], hv[2], hv[3]);
                            *reinterpret_cast<uint4*>(row + (((piece + 1) ^ sw) << 4)) = make_uint4(hv[4], hv[5], hv[6], hv[7]);
                        }
                    } else {
                        // The contributors' sums, added in CTA order: eight tokens at a time, the slots of four CTAs
                        // in flight at once.  (The round trips to L2 are what this costs.)
#pragma unroll 1
                        for (int u8 = 16 * tg + set; u8 < min(16 * tg + 16, 2 * n16); u8 += kTsSets) {
                            float f[8];
#pragma unroll
                            for (int i = 0; i < 8; i++) f[i] = 0.f;
#pragma unroll 1
                            for (int j0 = 0; j0 < n_contrib; j0 += 4) {
                                float4 p[4][2];
#pragma unroll
                                for (int j = 0; j < 4; j++) {
                                    const bool in = j0 + j < n_contrib;
                                    const int c = in ? 2 * (c_first + j0 + j) + (j0 + j == 0 ? slot_first : 0) : 0;
                                    const float4* q4 = reinterpret_cast<const float4*>(a.ts_partials + (size_t)c * slot_floats) + out + 2 * u8 * kTsOuts;
                                    p[j][0] = p[j][1] = make_float4(0.f, 0.f, 0.f, 0.f);
                                    if (in) { p[j][0] = __ldcg(q4); p[j][1] = __ldcg(q4 + kTsOuts); }
                                }
#pragma unroll
                                for (int j = 0; j < 4; j++) {
                                    f[0] += p[j][0].x; f[1] += p[j][0].y; f[2] += p[j][0].z; f[3] += p[j][0].w;
                                    f[4] += p[j][1].x; f[5] += p[j][1].y; f[6] += p[j][1].z; f[7] += p[j][1].w;
                                }
                            }
                            uint32_t hv[4];
#pragma unroll
                            for (int i = 0; i < 4; i++) hv[i] = h2_as_u32(__floats2half2_rn(f[2 * i], f[2 * i + 1]));
                            const int c8 = u8 & 15;                // 8 tokens = one 16-byte piece of a 64-token row
                            *reinterpret_cast<uint4*>(y_buf + (c8 >> 3) * 16384 + out * 128 + (((c8 & 7) ^ (out & 7)) << 4)) =
                                make_uint4(hv[0], hv[1], hv[2], hv[3]);
                        }
                    }
                    fence_proxy_async_smem();
                    tc_fence_before_sync();
                    named_bar_sync(1, 512);
                    if (warp == kTsFirstDecodeWarp) {
                        tc_fence_after_sync();
                        if (elect_one()) rotate_tile(d_tmem, smem_u32(y_buf), smem_u32(h_mat), smem_u32(h_full));
                        __syncwarp();
                    }
                    const bool used = 128 * tg + out < sg.rows;    // lane = token now
                    store_rotated(a, sg, used, sg.m0 + 128 * tg + out + sg.y_row_delta, lane_base, set, h_full, hpar, wait,
                                  [&] { if (128 * tg + 128 >= sg.rows) release_d(); });    // the last reads of D
                    hpar ^= 1u;
                }
            }
            release_d();
            // (handoff and y_buf are read by all warps before any of them comes here again: the next use is
            // behind the named barrier of the next tile)
            if (++db == a.ts_dbuf) { db = 0; dpar ^= 1u; }
        }
    }
    __syncwarp();
    if (F::kJoint && warp < kTsFirstDecodeWarp) {              // all threads take part in the cluster's barriers
        cluster_wait();
        cluster_sync();
    }
    tc_fence_before_sync();
    __syncthreads();
    if (warp == 2) {
        tc_fence_after_sync();
        tmem_dealloc(tmem_base, 512);
    }
}

}  // namespace exl3

#include "exl3_gemm_tiles.cuh"

namespace exl3 {

// ---- host side ----------------------------------------------------------------------------------

// Bytes of partial sums a dense launch may use: two slots of 128 columns x (tokens of a tile) per CTA.
inline size_t gemm_tile_partial_bytes(int tok, int ctas) { return (size_t)ctas * 2 * kTsOuts * (size_t)tok * sizeof(float); }

TsPlan gemm_plan(int64_t rows, int64_t tiles_n, int nks, int sms, size_t partial_bytes, int tok, int tok_wide);

inline int gemm_tensor_maps(CUtensorMap* tm_x, CUtensorMap* tm_w, const GemmArgs& a, int tile_words, const __half* xh, const uint32_t* trellis)
{
    const uint64_t in = (uint64_t)a.t_in * 16;
    const uint64_t xdims[2] = {in, (uint64_t)a.xh_rows};
    const uint64_t xstrides[1] = {in * 2};
    const uint32_t xbox[2] = {64u, (uint32_t)a.ts_box_rows};
    const int rc = make_tensor_map(tm_x, CU_TENSOR_MAP_DATA_TYPE_UINT16, 2, xh, xdims, xstrides, xbox, CU_TENSOR_MAP_SWIZZLE_128B);
    if (rc) return rc;
    const uint64_t dims[3] = {(uint64_t)tile_words, (uint64_t)a.t_out, (uint64_t)a.t_in};
    const uint64_t strides[2] = {(uint64_t)tile_words * 4, (uint64_t)a.t_out * tile_words * 4};
    const uint32_t box[3] = {(uint32_t)tile_words, 8u, (uint32_t)kTsStepTiles};
    return make_tensor_map(tm_w, CU_TENSOR_MAP_DATA_TYPE_UINT32, 3, trellis, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_NONE);
}

// Makes a kernel's whole shared memory available, once per device.
template <typename Kernel> static int gemm_shared_memory(Kernel kernel, bool (&done)[kMaxDevices])
{
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= kMaxDevices) return EXL3_E_UNSUPPORTED;
    if (done[dev]) return EXL3_OK;
    const int rc = note_cuda(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kTsSmemBytes));
    if (rc == EXL3_OK) done[dev] = true;
    return rc;
}

struct JointLaunch {
    cudaLaunchAttribute attr[2];
    cudaLaunchConfig_t cfg = {};
    JointLaunch(int grid, int n, cudaStream_t s)
    {
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = (unsigned)n;
        attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
        attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[1].val.programmaticStreamSerializationAllowed = 1;
        cfg.gridDim = dim3((unsigned)grid);
        cfg.blockDim = dim3(kTsThreads);
        cfg.dynamicSmemBytes = kTsSmemBytes;
        cfg.stream = s;
        cfg.attrs = attr;
        cfg.numAttrs = 2;
    }
};
// Clusters of n CTAs that the device holds at a time (a cluster lies in one part of the chip); asked once.
template <typename Kernel> static int gemm_clusters(Kernel kernel, int n)
{
    static int known[kMaxDevices][kTsJointMost + 1] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= kMaxDevices || n < 1 || n > kTsJointMost) return 0;
    int& k = known[dev][n];
    if (k == 0) {
        JointLaunch l(n, n, nullptr);
        l.cfg.numAttrs = 1;
        int c = 0;
        if (cudaOccupancyMaxActiveClusters(&c, kernel, &l.cfg) != cudaSuccess) { cudaGetLastError(); c = 0; }
        k = c > 0 ? c : -1;
    }
    return k;
}

template <int K, int CB> static int launch_gemm_tiles_t(GemmArgs a, const __half* xh, const uint32_t* trellis, cudaStream_t s)
{
    static bool attr_set[kMaxDevices] = {};
    int rc = gemm_shared_memory(gemm_tiles_kernel<K, CB>, attr_set);
    if (rc) return rc;
    a.cb_xor = 0x3B603B60u;
    a.ts_split = 0;
    // Rows of a tile: what nearly all tiles need if the caller says how many rows a tile has on average (the activation
    // ring is as deep as its stages are small, and up to 192 there are two accumulators), the table's 256 if not.  Tiles
    // with more are taken in parts.  Below 128 more parts are looked through than the smaller stages are worth: at least
    // 64 / 128, K = 4, 17 tokens of 16 experts, 1024 / 256 dims, 29.8 / 28.4 us; 16 tokens of 256 experts, 2048 / 512, 116.2 / 114.9.
    a.ts_tok = kTsMaxTok;
    a.ts_box_rows = 64;
    if (a.rows_hint > 0 && a.rows_hint < 200) {
        const double most = a.rows_hint + 2.5 * std::sqrt((double)a.rows_hint);
        a.ts_tok = std::max(128, std::min(kTsMaxTok, ((int)most + 31) / 32 * 32));
        a.ts_box_rows = 32;
    }
    a.n_items = 2 * a.n_tiles_tab * ((kTsMaxTok + a.ts_tok - 1) / a.ts_tok);
    a.ts_x_bytes = (a.ts_tok + a.ts_box_rows - 1) / a.ts_box_rows * a.ts_box_rows * 128;
    a.stages = std::min(kGtMaxXStages, (kTsSmemBytes - gt_x_off<K>()) / a.ts_x_bytes);
    a.ts_dbuf = a.ts_tok <= kGtTokTwice ? 2 : 1;
    CUtensorMap tm_x, tm_w;
    rc = gemm_tensor_maps(&tm_x, &tm_w, a, TsLayout<K>::kTileWords, xh, trellis);
    if (rc) return rc;
    // an odd stride: which items are in use repeats with a period of 2 or 4
    const int grid = std::min(a.n_items, (device_sm_count() - 1) | 1);
    return launch_kernel(gemm_tiles_kernel<K, CB>, dim3((unsigned)grid), dim3(kGtThreads), kTsSmemBytes, s, true, a, tm_x, tm_w);
}

template <int K, int CB> static int launch_gemm_t(GemmArgs a, const __half* xh, const uint32_t* trellis, cudaStream_t s)
{
    using L = TsLayout<K>;
    static bool attr_set[4][kMaxDevices] = {};
    int rc = gemm_shared_memory(gemm_kernel<K, CB, TS_PLAIN>, attr_set[TS_PLAIN]);
    if (rc == EXL3_OK) rc = gemm_shared_memory(gemm_kernel<K, CB, TS_AHEAD>, attr_set[TS_AHEAD]);
    if (rc == EXL3_OK) rc = gemm_shared_memory(gemm_kernel<K, CB, TS_WIDE>, attr_set[TS_WIDE]);
    if (rc == EXL3_OK) rc = gemm_shared_memory(gemm_kernel<K, CB, TS_JOINT>, attr_set[TS_JOINT]);
    if (rc) return rc;
    a.cb_xor = 0x3B603B60u;
    const int sms = device_sm_count(), nks = a.t_in / kTsStepTiles;
    a.tiles_n = a.t_out / 8;
    TsPlan plan = gemm_plan(a.m, a.tiles_n, nks, sms, a.ts_partial_bytes, L::kTok, L::kTokWide);
    const TsRings rings = {L::kRoom, L::kWBytes};
    a.ts_joint = ts_joint(plan, a.tiles_n, nks, sms, rings);
    while (a.ts_joint && gemm_clusters(gemm_kernel<K, CB, TS_JOINT>, a.ts_joint) < plan.tiles_m * a.tiles_n)
        a.ts_joint = ts_joint(plan, a.tiles_n, nks, sms, rings, a.ts_joint - 1);
    if (a.ts_joint) { plan.grid = (int)(plan.tiles_m * a.tiles_n) * a.ts_joint; plan.split = 1; }
    a.ts_tok = plan.tok;
    a.tiles_m = plan.tiles_m;
    if (!ts_countable(plan, a.tiles_n, nks)) return EXL3_E_SHAPE;
    a.n_items = a.tiles_m * a.tiles_n;
    a.ts_box_rows = a.ts_tok > 256 ? a.ts_tok / 2 : a.ts_tok;                      // (a box has at most 256 rows)
    a.ts_split = plan.split;
    const int mode = a.ts_joint ? TS_JOINT : plan.wide ? TS_WIDE : a.n_items >= 2 * plan.grid ? TS_AHEAD : TS_PLAIN;
    a.ts_x_bytes = (a.ts_tok + a.ts_box_rows - 1) / a.ts_box_rows * a.ts_box_rows * 128;
    // Ring x has up to eight stages beside eight of ring w (four in the wide form); what is left goes to ring w, up to three
    // stages per set (more do not pay: 28 stages delay the first activations behind them, 17408 -> 512 16.4 -> 17.4 us).
    a.ts_recv_bytes = ts_recv_bytes(a.ts_tok, a.ts_joint);
    a.stages = ts_x_stages(rings, a.ts_recv_bytes, mode == TS_WIDE ? 4 : 8, a.ts_x_bytes, kTsStages);
    a.ts_w_stages = std::min(kTsMaxWStages, (L::kRoom - a.ts_recv_bytes - a.stages * a.ts_x_bytes) / L::kWBytes) / kTsSets * kTsSets;
    if (a.stages < kTsLeastStages || a.ts_w_stages < kTsSets) return EXL3_E_UNSUPPORTED;        // (never for a plan as above: no ring, no launch)
    a.ts_dbuf = a.ts_tok <= 128 ? 2 : 1;
    CUtensorMap tm_x, tm_w;
    rc = gemm_tensor_maps(&tm_x, &tm_w, a, L::kTileWords, xh, trellis);
    if (rc) return rc;
    if (mode == TS_JOINT) {
        const JointLaunch l(plan.grid, a.ts_joint, s);
        return note_cuda(cudaLaunchKernelEx(&l.cfg, gemm_kernel<K, CB, TS_JOINT>, (const GemmArgs)a, (const CUtensorMap)tm_x, (const CUtensorMap)tm_w));
    }
    const auto kernel = mode == TS_AHEAD ? gemm_kernel<K, CB, TS_AHEAD> : mode == TS_WIDE ? gemm_kernel<K, CB, TS_WIDE> : gemm_kernel<K, CB, TS_PLAIN>;
    return launch_kernel(kernel, dim3((unsigned)plan.grid), dim3(kTsThreads), kTsSmemBytes, s, true, a, tm_x, tm_w);
}

template <int K>
int launch_gemm_k(const GemmArgs& a, int cb, const __half* xh, const uint32_t* trellis, cudaStream_t s)
{
    switch (cb) {
        case CB_3INST:
            return a.tile_tab ? launch_gemm_tiles_t<K, CB_3INST>(a, xh, trellis, s) : launch_gemm_t<K, CB_3INST>(a, xh, trellis, s);
        case CB_MCG:
            return a.tile_tab ? launch_gemm_tiles_t<K, CB_MCG>(a, xh, trellis, s) : launch_gemm_t<K, CB_MCG>(a, xh, trellis, s);
        case CB_MUL1:
            return a.tile_tab ? launch_gemm_tiles_t<K, CB_MUL1>(a, xh, trellis, s) : launch_gemm_t<K, CB_MUL1>(a, xh, trellis, s);
        default: return EXL3_E_CODEBOOK;
    }
}

}  // namespace exl3
