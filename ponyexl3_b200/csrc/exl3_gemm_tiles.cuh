// GEMM over a device table of output tiles (SwitchGLU prefill): each tile names its trellis columns, activation rows,
// scales and output rows.  The product, the operands' layouts and the finishing steps are those of the dense kernel
// (exl3_gemm.cuh); what differs is who does what, because a CTA runs through many short tiles (8 to 32 k-steps each):
//   warp 0       packed tiles: one TMA box per k-step (ring w, two stages per set)
//   warps 1, 3   activations: TMA boxes (ring x), every other k-step each
//   warp 2       issues the MMAs
//   warps 4-11   finish the tiles
//   warps 12-27  decode: four sets of four warps, the sets take the k-steps in turn
// Tensor memory: one stage of weights per set (4 x 32 columns) and 384 columns of sums, two accumulators of up to 192
// tokens or one of up to 256.  A set decodes half of its k-step before it waits for the MMAs of its previous one, so
// a stage per set is enough.
//
// What bounds it: for gate|up (many k-steps a tile) the round trip of ring x.  A k-step's boxes take 4,000 clocks from the
// request to the MMAs that free them, and the shared memory left holds seven of them: 580 clocks a k-step, where four
// sets of 1300 .. 1650 clocks a k-step each would decode one in 410 at most.  That is why ring x gets all memory that the rest does not need (H64 for
// H128, two stages per set in ring w).  For down (few k-steps, one stored tile each) the finishing warps: eight are quicker
// than four (155 -> 133 us), and with two accumulators they work beside the next tile's MMAs.
// 4096 tokens, 256 experts, top-8, 2048 / 512, K = 4: gate|up 221 -> 187 us, down 175 -> 133 us against the dense kernel's
// organisation (16 decode warps that also finish the tiles), which this kernel had before.
#pragma once

namespace exl3 {

constexpr int kGtSets = 4, kGtFirstDecodeWarp = 12, kGtFirstEpiWarp = 4;
constexpr int kGtEpiThreads = 32 * (kGtFirstDecodeWarp - kGtFirstEpiWarp);
constexpr int kGtThreads = 32 * (kGtFirstDecodeWarp + 4 * kGtSets);
constexpr int kGtSumCols = 512 - 32 * kGtSets, kGtTokTwice = kGtSumCols / 2;
constexpr int kGtHBytes = 2 * 64 * 64 * 2;             // H64 and -H64
constexpr int kGtScaleOff = 1024, kGtHOff = 2048, kGtYOff = kGtHOff + kGtHBytes, kGtWOff = kGtYOff + kTsYBytes;
constexpr int kGtWStages = 2 * kGtSets, kGtMaxXStages = 16;
template <int K> constexpr int gt_x_off() { return kGtWOff + kGtWStages * TsLayout<K>::kWBytes; }

// The output rotation as H128 = [[H64, H64], [H64, -H64]]: a quarter of the operand, and what that saves is one more stage of ring
// x.  (Products of 64 columns take the tensor cores longer, but here nobody waits for them; see rotate_tile.)
__device__ __forceinline__ void store_h64(uint8_t* h_mat, int thread, int threads)
{
    for (int i = thread; i < 1024; i += threads) {
        const int n = (i >> 3) & 63, ch = i & 7;
        const uint32_t flip = ((__popc(n & (8 * ch)) ^ (i >> 9)) & 1) ? 0x80008000u : 0u;
        uint32_t w[4];
#pragma unroll
        for (int j = 0; j < 4; j++)
            w[j] = flip ^ (0x3C003C00u | ((__popc(n & (2 * j)) & 1) ? 0x8000u : 0u) | ((__popc(n & (2 * j + 1)) & 1) ? 0x80000000u : 0u));
        *reinterpret_cast<uint4*>(h_mat + (i >> 9) * 8192 + n * 128 + ((ch ^ (n & 7)) << 4)) = make_uint4(w[0], w[1], w[2], w[3]);
    }
}
__device__ __forceinline__ void rotate_tile_h64(uint32_t d_tmem, uint32_t y_buf, uint32_t h_mat, uint32_t done)
{
    const uint64_t yd = smem_desc_mn_sw128(y_buf), hd = smem_desc_sw128(h_mat);
#pragma unroll
    for (int nh = 0; nh < 2; nh++)
#pragma unroll
        for (int kk = 0; kk < 8; kk++)
            tc_mma_f16(d_tmem + 64 * nh, yd + 128 * kk, hd + (nh & (kk >> 2)) * 512 + (kk & 3) * 2, mma_idesc_f16(128, 64) | kIdescMajorA,
                       kk > 0 ? 1u : 0u);
    tc_commit(done);
}

template <int K, int CB>
__global__ void __launch_bounds__(kGtThreads, 1)
    gemm_tiles_kernel(const GemmArgs a, const __grid_constant__ CUtensorMap tm_x, const __grid_constant__ CUtensorMap tm_w)
{
    using L = TsLayout<K>;
    using Walk = TsWalk<true>;
    constexpr int S = kGtSets, NW = kGtWStages;
    extern __shared__ __align__(1024) uint8_t smem[];
    uint64_t* w_full = reinterpret_cast<uint64_t*>(smem);      // packed tiles landed                      [NW]
    uint64_t* w_empty = w_full + NW;                           // ... read by the set's four warps          [NW]
    uint64_t* full = w_empty + NW;                             // weights decoded                           [S]
    uint64_t* empty = full + S;                                // the k-step's MMAs are done                [S]
    uint64_t* x_full = empty + S;                              // activations landed                       [nx]
    uint64_t* x_empty = x_full + kGtMaxXStages;                // ... and their MMAs are done              [nx]
    uint64_t* d_full = x_empty + kGtMaxXStages;                            // a tile's sums are complete                [2]
    uint64_t* d_empty = d_full + 2;                            // ... and drained                           [2]
    uint64_t* h_full = d_empty + 2;                            // the rotated tile is complete
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(h_full + 1);
    const TsWait wait{reinterpret_cast<volatile int*>(tmem_slot + 1), a.status};
    float* scales = reinterpret_cast<float*>(smem + kGtScaleOff);      // of two tiles
    uint8_t* h_mat = smem + kGtHOff;
    uint8_t* y_buf = smem + kGtYOff;
    uint8_t* w_ring = smem + kGtWOff;
    uint8_t* x_ring = smem + gt_x_off<K>();

    const int tid = threadIdx.x, warp = Walk::uniform(tid >> 5), lane = tid & 31;
    const int nx = a.stages, x_bytes = a.ts_x_bytes;           // depth and stage size of ring x
    Walk walk;
    walk.start(a);
    TsSeg sg;

    if (warp == 0) {
        if (lane < NW) {
            mbar_init(smem_u32(&w_full[lane]), 1);
            mbar_init(smem_u32(&w_empty[lane]), 4);
        }
        if (lane < S) {
            mbar_init(smem_u32(&full[lane]), 4);
            mbar_init(smem_u32(&empty[lane]), 1);
        }
        if (lane < nx) {
            mbar_init(smem_u32(&x_full[lane]), 1);
            mbar_init(smem_u32(&x_empty[lane]), 1);
        }
        if (lane < 2) {
            mbar_init(smem_u32(&d_full[lane]), 1);
            mbar_init(smem_u32(&d_empty[lane]), kGtEpiThreads / 32);
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
    griddep_launch_dependents();

    if (warp == 0) {
        // ------------------------------------------------------------------ packed tiles ----
        const bool leader = elect_one();
        if (leader) tma_prefetch_desc(&tm_w);
        griddep_wait();                                        // the table belongs to an earlier kernel
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
                if (++s == NW) { s = 0; parity ^= 1u; }
            }
        }
    } else if (warp == 1 || warp == 3) {
        // ------------------------------------------------------------------- activations ----
        // From a stage's release to its next data in use takes some 3.5 K clocks, of which the boxes' issue is 400: hence as deep a
        // ring as there is room for, with barriers of its own, and two warps.
        const bool leader = elect_one();
        if (leader) tma_prefetch_desc(&tm_x);
        griddep_wait();
        const int box_rows = a.ts_box_rows, box_bytes = box_rows * 128;
        const int mine = warp >> 1;                            // even or odd k-steps
        int v = 0, s = mine;                                   // k-step; the ring stage of this warp's next one
        uint32_t parity = 1;
        while (walk.next(a, sg)) {
            const int boxes = (sg.rows + box_rows - 1) / box_rows;
            for (int ks = sg.k0; ks < sg.k1; ks++, v++) {
                if ((v & 1) != mine) continue;
                wait(&x_empty[s], parity);
                if (leader) {
                    const uint32_t bar = smem_u32(&x_full[s]);
                    const uint32_t dst = smem_u32(x_ring) + (uint32_t)(s * x_bytes);
                    mbar_arrive_expect_tx(bar, (uint32_t)(boxes * box_bytes));
                    for (int i = 0; i < boxes; i++)
                        tma_load_2d(dst + i * box_bytes, &tm_x, ks * 64, sg.m0 + box_rows * i, bar);
                }
                if ((s += 2) >= nx) { s -= nx; parity ^= 1u; }
            }
        }
    } else if (warp == 2) {
        // -------------------------------------------------------------------- MMA issuer ----
        const bool leader = elect_one();
        griddep_wait();
        int xs = 0, as = 0, db = 0;
        uint32_t dpar = 1, par = 0, x_par = 0;
        const uint32_t x0 = smem_u32(x_ring);
        while (walk.next(a, sg)) {
            wait(&d_empty[db], dpar);
            tc_fence_after_sync();
            const uint32_t d_tmem = tmem_base + (uint32_t)(kGtTokTwice * db);
            const uint32_t idesc = mma_idesc_f16(128, (sg.rows + 15) & ~15);
            uint32_t accum = 0;
            for (int ks = sg.k0; ks < sg.k1; ks++) {
                const uint32_t at = tmem_base + kGtSumCols + 32 * as;
                const uint64_t xd = smem_desc_sw128(x0 + (uint32_t)(xs * x_bytes));
                wait(&x_full[xs], x_par);
                wait(&full[as], par);
                tc_fence_after_sync();
                if (leader) {
                    tc_mma_kstep(d_tmem, at, xd, idesc, accum);
                    tc_commit(smem_u32(&empty[as]));
                    tc_commit(smem_u32(&x_empty[xs]));
                }
                accum = 1u;
                if (++xs == nx) { xs = 0; x_par ^= 1u; }
                if (++as == S) { as = 0; par ^= 1u; }
            }
            if (leader) tc_commit(smem_u32(&d_full[db]));
            if (++db == a.ts_dbuf) { db = 0; dpar ^= 1u; }
        }
    } else if (warp >= kGtFirstDecodeWarp) {
        // ------------------------------------------------------------------------ decode ----
        const int q = warp & 3, set = (warp - kGtFirstDecodeWarp) >> 2;
        const int prev_word = (lane + 31) & 31;
        const uint32_t xc = a.cb_xor;
        LaneWords<K> lw;
        lw.init(lane);
        const uint32_t a_tmem = tmem_base + ((uint32_t)(32 * q) << 16) + kGtSumCols + 32 * set;
        griddep_wait();
        // The k-steps of all tiles in one sequence.
        int end = 0, v = set, ws = set;                        // (NW is a multiple of S: a stage of ring w is one set's, too)
        uint32_t par = 0, w_par = 0;
        while (walk.next(a, sg)) {
            end += sg.k1 - sg.k0;
            for (; v < end; v += S, par ^= 1u) {
                wait(&w_full[ws], w_par);
                const uint32_t* wt = reinterpret_cast<const uint32_t*>(w_ring + ws * L::kWBytes) + 2 * q * L::kTileWords;
                // (As a loop for K >= 4.  Up to 3 it cost more than its smaller code gave: 17 tokens of 16 experts, 2048 / 512 dims,
                // K = 2, 41.7 us as a loop, 40.5 without; K = 4 the other way round, 1000 tokens of 256 experts +3 % without.)
                constexpr int kUnroll = K <= 3 ? 2 : 1;
#pragma unroll kUnroll
                for (int h = 0; h < 2; h++) {                  // tile columns 2q, 2q + 1 of all four tile rows
                    uint32_t frag[16];
#pragma unroll
                    for (int tk = 0; tk < 4; tk++) {
                        const uint32_t* tw = wt + (tk * 8 + h) * L::kTileWords;
                        uint32_t cw[8];
                        if constexpr (K == 4) lane_codewords_k4(tw[lane], tw[prev_word], cw);
                        else lane_codewords<K>(tw[lw.i0], tw[lw.i1], LaneWords<K>::kThree ? tw[lw.i2] : 0u, lw.sh, cw);
                        frag[4 * tk + 0] = decode_pair_rt<CB>(cw[0], cw[1], xc);
                        frag[4 * tk + 1] = decode_pair_rt<CB>(cw[4], cw[5], xc);
                        frag[4 * tk + 2] = decode_pair_rt<CB>(cw[2], cw[3], xc);
                        frag[4 * tk + 3] = decode_pair_rt<CB>(cw[6], cw[7], xc);
                    }
                    if (h == 0) {                              // the MMAs of this set's k-step before
                        if (v >= S) wait(&empty[set], par ^ 1u);
                        tc_fence_after_sync();
                    }
                    tmem_st_16x32cols(a_tmem + ((uint32_t)(16 * h) << 16), frag);
                }
                // Only now is it certain that the packed words have been read: the stores above depend on them.
                __syncwarp();
                if (lane == 0) mbar_arrive(smem_u32(&w_empty[ws]));
                if ((ws += S) >= NW) { ws = set; w_par ^= 1u; }
                tmem_st_wait();
                tc_fence_before_sync();
                __syncwarp();
                if (lane == 0) mbar_arrive(smem_u32(&full[set]));
            }
        }
    } else if (warp >= kGtFirstEpiWarp) {
        // -------------------------------------------------------------- finish the tiles ----
        // Two warps per quarter of the tensor-memory lanes, each with every other piece of sixteen columns.
        const int q = warp & 3, part = (warp - kGtFirstEpiWarp) >> 2, out = 32 * q + lane;     // column of the tile, then token of the group
        store_h64(h_mat, tid - 32 * kGtFirstEpiWarp, kGtEpiThreads);
        griddep_wait();
        int db = 0;
        uint32_t dpar = 0, hpar = 0;
        float* scale_of = scales;
        while (walk.next(a, sg)) {
            const int n16 = (sg.rows + 15) >> 4;
            auto out_row = [&](int tg) {                       // output row of this thread's token
                const int row = 128 * tg + out, grow = sg.m0 + row + sg.y_row_delta;
                return a.y_row_map && row < sg.rows ? a.y_row_map[grow] : grow;
            };
            int orow = out_row(0);
            // (two tiles' worth: a warp may still be storing the tile before)
            scale_of = scale_of == scales ? scales + 128 : scales;
            if (part == 0) scale_of[out] = a.svh ? __half2float(a.svh[sg.sv_off + out]) : 1.f;
            wait(&d_full[db], dpar);
            tc_fence_after_sync();
            const uint32_t d_tmem = tmem_base + (uint32_t)(kGtTokTwice * db);
            const uint32_t lane_base = d_tmem + ((uint32_t)(32 * q) << 16);
#pragma unroll 1
            for (int tg = 0; 128 * tg < sg.rows; tg++) {       // 128 tokens at a time
#pragma unroll 1
                for (int ch = 8 * tg + part; ch < min(8 * tg + 8, n16); ch += 2) {
                    float f[16];
                    tmem_ld_16cols(lane_base + 16 * ch, f);
                    uint32_t hv[8];
#pragma unroll
                    for (int i = 0; i < 8; i++) hv[i] = h2_as_u32(__floats2half2_rn(f[2 * i], f[2 * i + 1]));
                    const int c16 = ch & 7;                    // 16 tokens = two 16-byte pieces of a 64-token row
                    uint8_t* row = y_buf + (c16 >> 2) * 16384 + out * 128;
                    const int piece = 2 * (c16 & 3), sw = out & 7;
                    *reinterpret_cast<uint4*>(row + ((piece ^ sw) << 4)) = make_uint4(hv[0], hv[1], hv[2], hv[3]);
                    *reinterpret_cast<uint4*>(row + (((piece + 1) ^ sw) << 4)) = make_uint4(hv[4], hv[5], hv[6], hv[7]);
                }
                fence_proxy_async_smem();
                tc_fence_before_sync();
                named_bar_sync(1, kGtEpiThreads);
                if (warp == kGtFirstEpiWarp) {
                    tc_fence_after_sync();
                    if (elect_one()) rotate_tile_h64(d_tmem, smem_u32(y_buf), smem_u32(h_mat), smem_u32(h_full));
                    __syncwarp();
                }
                const bool used = 128 * tg + out < sg.rows;    // lane = token now
                __half* yp = nullptr;
                if (used) {
                    if (a.n_peer > 0) {                        // the row belongs to the GPU that holds its token
                        const int pr = orow / a.rows_per_peer;
                        yp = a.y_peer[pr] + (int64_t)(orow - pr * a.rows_per_peer) * a.y_row_stride + sg.y_col;
                    } else {
                        yp = a.y + (int64_t)orow * a.y_row_stride + sg.y_col;
                    }
                }
                if (128 * tg + 128 < sg.rows) orow = out_row(tg + 1);
                wait(h_full, hpar);
                hpar ^= 1u;
                tc_fence_after_sync();
                if (128 * tg + 32 * q < sg.rows) {
                    const uint64_t had = f32x2(EXL3_HAD_SCALE, EXL3_HAD_SCALE);
#pragma unroll 1
                    for (int c = part; c < 8; c += 2) {
                        float f[16];
                        tmem_ld_16cols(lane_base + 16 * c, f);
                        uint32_t h[8];
#pragma unroll
                        for (int i = 0; i < 4; i++) {
                            const float4 w = *reinterpret_cast<const float4*>(scale_of + 16 * c + 4 * i);
                            h[2 * i] = f16_pair(mul_f32x2(mul_f32x2(f32x2(f[4 * i], f[4 * i + 1]), had), f32x2(w.x, w.y)));
                            h[2 * i + 1] = f16_pair(mul_f32x2(mul_f32x2(f32x2(f[4 * i + 2], f[4 * i + 3]), had), f32x2(w.z, w.w)));
                        }
                        if (used) {
                            const uint4 lo = make_uint4(h[0], h[1], h[2], h[3]), hi = make_uint4(h[4], h[5], h[6], h[7]);
                            if (a.y_wide) {
                                st_global_256(yp + 16 * c, lo, hi);   // whole sectors, also into another GPU
                            } else {
                                *reinterpret_cast<uint4*>(yp + 16 * c) = lo;
                                *reinterpret_cast<uint4*>(yp + 16 * c + 8) = hi;
                            }
                        }
                    }
                }
            }
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&d_empty[db]));    // the next tile but one may go into this accumulator
            if (++db == a.ts_dbuf) { db = 0; dpar ^= 1u; }
        }
    }
    __syncwarp();
    tc_fence_before_sync();
    __syncthreads();
    if (warp == 2) {
        tc_fence_after_sync();
        tmem_dealloc(tmem_base, 512);
    }
    if (a.n_peer > 0 && tid == 0) {
        // Rows were stored into other GPUs' memory: every CTA is counted on a local counter (the
        // barrier above orders the CTA's stores before this thread's fence), and the CTA that
        // completes the count announces this GPU's rows to every peer.
        __threadfence();
        const unsigned done = atomicAdd(a.done_ctr, 1u) + 1u;
        if (done == gridDim.x) {
            atomicExch(a.done_ctr, 0u);           // re-armed for the next launch on this workspace
            __threadfence_system();
            for (int p = 0; p < a.n_peer; p++)
                asm volatile("red.relaxed.sys.global.add.u32 [%0], 1;" ::"l"(a.ctr_peer[p]) : "memory");
        }
    }
}

}  // namespace exl3
