// Codec kernels outside the matmul: tile unpack, full decode to fp16 (the
// bit-exact test target), the codebook table, and the stand-alone Hadamard-128
// rotation.  All are HBM-trivial; the matmul kernels reuse the same device
// functions, so a bit-exact decode here proves the arithmetic they run.
#include <type_traits>

#include "exl3_internal.h"

namespace exl3 {

// ---- unpack: one warp per tile ------------------------------------------------------------
template <int K>
__global__ void __launch_bounds__(256) unpack_kernel(const uint32_t* __restrict__ trellis,
                                                     int64_t n_tiles, uint16_t* __restrict__ out)
{
    const int lane = threadIdx.x & 31;
    LaneWords<K> lw;
    lw.init(lane);
    const int64_t warp0 = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const int64_t nwarps = (int64_t)gridDim.x * (blockDim.x >> 5);
    for (int64_t tile = warp0; tile < n_tiles; tile += nwarps) {
        const uint32_t* w = trellis + tile * (8 * K);
        uint32_t cw[8];
        lane_codewords<K>(w[lw.i0], w[lw.i1], LaneWords<K>::kThree ? w[lw.i2] : 0u, lw.sh, cw);
        uint4 v;
        v.x = cw[0] | (cw[1] << 16);
        v.y = cw[2] | (cw[3] << 16);
        v.z = cw[4] | (cw[5] << 16);
        v.w = cw[6] | (cw[7] << 16);
        reinterpret_cast<uint4*>(out + tile * 256)[lane] = v;
    }
}

// ---- decode: one warp per tile, fp16 W written at its matrix position ------------------------
template <int K, int CB>
__global__ void __launch_bounds__(256)
    decode_kernel(const uint32_t* __restrict__ trellis, int64_t t_in, int64_t t_out, int64_t tn0,
                  int64_t tn_count, __half* __restrict__ w, int64_t ld)
{
    const int lane = threadIdx.x & 31;
    LaneWords<K> lw;
    lw.init(lane);
    const int64_t warp0 = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const int64_t nwarps = (int64_t)gridDim.x * (blockDim.x >> 5);
    const int64_t n_tiles = t_in * tn_count;
    for (int64_t i = warp0; i < n_tiles; i += nwarps) {
        const int64_t tk = i / tn_count, tl = i % tn_count;
        const uint32_t* p = trellis + (tk * t_out + tn0 + tl) * (8 * K);
        uint32_t cw[8];
        lane_codewords<K>(p[lw.i0], p[lw.i1], LaneWords<K>::kThree ? p[lw.i2] : 0u, lw.sh, cw);
#pragma unroll
        for (int j = 0; j < 8; j += 2) {
            const __half2 v = u32_as_h2(decode_pair<CB>(cw[j], cw[j + 1]));
            __half* dst = w + (tk * 16) * ld + tl * 16;
            dst[(int64_t)frag_row(lane, j) * ld + frag_col(lane, j)] = __low2half(v);
            dst[(int64_t)frag_row(lane, j + 1) * ld + frag_col(lane, j + 1)] = __high2half(v);
        }
    }
}

template <int CB> __global__ void table_kernel(__half* __restrict__ table)
{
    const uint32_t w = blockIdx.x * blockDim.x + threadIdx.x;
    if (w < 65536u) table[w] = decode_one<CB>(w);
}

// ---- Hadamard-128: one warp per (row, block) ----------------------------------------------
template <typename T> __device__ __forceinline__ void load4(const T* p, float (&v)[4]);
template <> __device__ __forceinline__ void load4<__half>(const __half* p, float (&v)[4])
{
    const uint2 u = *reinterpret_cast<const uint2*>(p);
    const float2 a = __half22float2(u32_as_h2(u.x)), b = __half22float2(u32_as_h2(u.y));
    v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
}
template <> __device__ __forceinline__ void load4<__nv_bfloat16>(const __nv_bfloat16* p, float (&v)[4])
{
    const uint2 u = *reinterpret_cast<const uint2*>(p);
    v[0] = __uint_as_float(u.x << 16); v[1] = __uint_as_float(u.x & 0xFFFF0000u);
    v[2] = __uint_as_float(u.y << 16); v[3] = __uint_as_float(u.y & 0xFFFF0000u);
}
template <> __device__ __forceinline__ void load4<float>(const float* p, float (&v)[4])
{
    const float4 f = *reinterpret_cast<const float4*>(p);
    v[0] = f.x; v[1] = f.y; v[2] = f.z; v[3] = f.w;
}

// Both rotation kernels are launched as programmatic dependents: their blocks are set up while the
// previous kernel of the stream drains.  With EXL3_FLAG_PDL (early_trigger) the next kernel, the matmul
// that consumes `out`, may start streaming its weights right away; without the flag it may do so once
// everything before this kernel is complete, so that weights written just before the call are seen.
__device__ __forceinline__ void rotation_dependency(int early_trigger)
{
    if (early_trigger) griddep_launch_dependents();
    griddep_wait();
    if (!early_trigger) griddep_launch_dependents();
}

// Rows of x may be gathered (row_src) and the scale vectors chosen per output row
// (pre_row / post_row give the row of the pre / post matrix to use), which is what the
// sibling-group and MoE paths need; the plain rotation passes NULL for all three.
template <typename T>
__global__ void __launch_bounds__(256)
    hadamard_kernel(const T* __restrict__ x, int64_t rows, int64_t n, int64_t x_row_stride,
                    const __half* __restrict__ pre, const __half* __restrict__ post,
                    __half* __restrict__ out, const int32_t* __restrict__ row_src,
                    const int32_t* __restrict__ pre_row, const int32_t* __restrict__ post_row,
                    int early_trigger, int out_mode, int glu, int member_rows)
{
    rotation_dependency(early_trigger);
    // 32-bit block arithmetic (the launcher refuses more than 2^31 blocks): 64-bit divisions that split
    // a block index into (row, block of the row) cost more than the butterfly itself
    const int lane = threadIdx.x & 31;
    const uint32_t nblk = (uint32_t)(n >> 7);
    const uint32_t total = (uint32_t)rows * nblk;
    const uint32_t warp0 = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const uint32_t nwarps = gridDim.x * (blockDim.x >> 5);
    // Four 128-blocks per warp and turn: the loads of all four are in flight before the first
    // butterfly starts (one 256-byte load per warp at a time left the kernel latency-bound).
    constexpr int U = 4;
    for (uint32_t i0 = warp0; i0 < total; i0 += nwarps * U) {
        float v[U][4], sp[U][4];
        int64_t rr[U], cc[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
            const uint32_t i = i0 + u * nwarps;      // strided: small problems still use every warp
            const bool ok = i < total && i >= i0;    // (i >= i0: no wrap-around)
            const uint32_t rq = ok ? i / nblk : 0u;
            const int64_t r = rq, b = ok ? i - rq * nblk : 0u;
            rr[u] = ok ? r : -1;
            cc[u] = b * 128 + lane * 4;
            // members of a sibling group rotate the same rows with their own signs, one after the other (a 32-bit
            // division here was 0.5 us slower for two members of 17408 columns: 56.1 -> 56.6)
            const int64_t member = member_rows ? r / member_rows : 0;
            const int64_t rs = row_src ? row_src[r] : r - member * member_rows;
            load4<T>(x + rs * x_row_stride + cc[u], v[u]);
            if (glu && ok) {
                // the row holds [gate (n) | up (n)]: the input is fp16(act(gate) * up)
                float up[4];
                load4<T>(x + rs * x_row_stride + n + cc[u], up);
#pragma unroll
                for (int q = 0; q < 4; q++) v[u][q] = glu_value(v[u][q], up[q], glu);
            }
            if (pre) load4<__half>(pre + (pre_row ? (int64_t)pre_row[r] : member) * n + cc[u], sp[u]);
        }
#pragma unroll
        for (int u = 0; u < U; u++) {
            // the reference rounds x to fp16 first (ponyexl3/ref/forward.py:26)
#pragma unroll
            for (int q = 0; q < 4; q++) {
                v[u][q] = __half2float(__float2half_rn(v[u][q]));
                if (pre) v[u][q] *= sp[u][q];
            }
            had128_warp(v[u], lane);
        }
#pragma unroll
        for (int u = 0; u < U; u++) {
            if (rr[u] < 0) continue;
            const int64_t r = rr[u], col = cc[u];
#pragma unroll
            for (int q = 0; q < 4; q++) v[u][q] *= EXL3_HAD_SCALE;
            if (post) {
                float s[4];
                load4<__half>(post + (post_row ? (int64_t)post_row[r] * n : 0) + col, s);
#pragma unroll
                for (int q = 0; q < 4; q++) v[u][q] *= s[q];
            }
            uint2 o;
            o.x = h2_as_u32(__floats2half2_rn(v[u][0], v[u][1]));
            o.y = h2_as_u32(__floats2half2_rn(v[u][2], v[u][3]));
            if (out_mode == HAD_OUT_F16) {
                *reinterpret_cast<uint2*>(out + r * n + col) = o;
            } else {
                // one 32-bit word per element for the GEMV's two-slot fragments:
                // (x, 0) keeps exactly-decoded weights, (x, x) lets the MMA add the two
                // codebook halves itself
                uint4 e;
                const uint32_t m = (out_mode == HAD_OUT_PAIR_X0) ? 0u : 0x00010000u;
                e.x = (o.x & 0xFFFFu) * (1u + m);
                e.y = (o.x >> 16) * (1u + m);
                e.z = (o.y & 0xFFFFu) * (1u + m);
                e.w = (o.y >> 16) * (1u + m);
                *reinterpret_cast<uint4*>(reinterpret_cast<uint32_t*>(out) + r * n + col) = e;
            }
        }
    }
}

// ---- the rotation of many rows, on the tensor cores ---------------------------------------------
// had128(x * suh) for blocks of 16 rows x 128 columns.  H128 = H8 (x) H16: the 16-point transform over four
// of the seven column bits is a product with the +-1 matrix H16 (mma.sync m16n8k16, 16 of them per block),
// the 8-point one over the other three is butterflies between the eight accumulator groups, two values per
// instruction.  fp16 inputs times +-1 are exact and the sums are fp32, as in the butterfly kernel; only the
// order of the fp32 additions differs.  As one 128-point product (128 MMAs per block) the kernel was bound
// by the rate of mma.sync: 42 us for 8192 x 5120 and 138 us for 65,536 x 2048.
//
// A lane loads 16 contiguous bytes (8 columns) of rows g and g + 8 per quarter of the block: column
// 32 q + 8 t + 4 s + c, c = 0..3.  The MMA's k index is a free bijection as long as A and B agree: group
// (q, s) takes its sixteen columns as k = 2 t + (c & 1) + 8 (c >> 1), so the four bits of k are the column
// bits 0 (c), 3, 4 (t) and 1 (c); the bits of n are given the same meaning, which makes B the plain H16 for
// every group and leaves a lane, after the butterflies over q and s, with the same 8 contiguous columns
// per quarter that it loaded: stores are as wide as the loads.
//
// x * pre is rounded to fp16, which is exact for +-1 only.  With SPLIT it is two fp16 parts and two products: for
// the rows of a sibling group that one by one would be few enough for the butterfly kernel, which does not round
// it (multipliers of 0.5 to 1.5, 40 rows: 5.0e-4 off the oracle without, 7e-5 with it).  A group of 5120 + 2 x 1024
// columns and 24 to 63 rows takes 19.4 .. 21.0 us without, 19.6 .. 21.2 with it, 23.1 .. 27.2 by the butterfly kernel.  (And for
// EXL3_FLAG_WIDE_SCALES where the number of rows is on the device, which the butterfly kernel does not read.)
//
// COPIES: output rows r, r + base, r + 2 base, .. are the same row of x with other multipliers (gate and up of a
// SwitchGLU, the members of a sibling group), and a block's loads of x serve all of them.
template <typename T> struct Load8;
template <> struct Load8<__half> {
    static __device__ __forceinline__ uint4 at(const __half* p) { return *reinterpret_cast<const uint4*>(p); }
};
template <> struct Load8<__nv_bfloat16> {
    static __device__ __forceinline__ uint4 at(const __nv_bfloat16* p)
    {
        const uint4 u = *reinterpret_cast<const uint4*>(p);
        const uint32_t w[4] = {u.x, u.y, u.z, u.w};
        uint32_t o[4];
#pragma unroll
        for (int i = 0; i < 4; i++)
            o[i] = h2_as_u32(__floats2half2_rn(__uint_as_float(w[i] << 16), __uint_as_float(w[i] & 0xFFFF0000u)));
        return make_uint4(o[0], o[1], o[2], o[3]);
    }
};
template <> struct Load8<float> {
    static __device__ __forceinline__ uint4 at(const float* p)
    {
        const float4 a = *reinterpret_cast<const float4*>(p), b = *reinterpret_cast<const float4*>(p + 4);
        return make_uint4(h2_as_u32(__floats2half2_rn(a.x, a.y)), h2_as_u32(__floats2half2_rn(a.z, a.w)),
                          h2_as_u32(__floats2half2_rn(b.x, b.y)), h2_as_u32(__floats2half2_rn(b.z, b.w)));
    }
};

__device__ __forceinline__ uint32_t glu_pair(uint32_t gate, uint32_t up, int glu)
{
    const float2 gf = __half22float2(u32_as_h2(gate)), uf = __half22float2(u32_as_h2(up));
    return h2_as_u32(__floats2half2_rn(glu_value(gf.x, uf.x, glu), glu_value(gf.y, uf.y, glu)));
}

// x * p as the rounded product (in place of x) and what that leaves out, exact but for what is below 2^-24.
__device__ __forceinline__ void split_product(uint32_t& x, uint32_t p, uint32_t& rest)
{
    const __half2 x2 = u32_as_h2(x), p2 = u32_as_h2(p), h = __hmul2_rn(x2, p2);
    x = h2_as_u32(h);
    rest = h2_as_u32(__hfma2(x2, p2, __hneg2(h)));
}

template <typename T, bool SPLIT, bool COPIES>
__global__ void __launch_bounds__(256, 2)
    hadamard_mma_kernel(const T* __restrict__ x, int64_t rows, int64_t n, int64_t x_row_stride,
                        const __half* __restrict__ pre, __half* __restrict__ out,
                        const int32_t* __restrict__ row_src, const int32_t* __restrict__ pre_row,
                        const int32_t* __restrict__ rows_dev, int early_trigger, int glu, int member_rows, int copies)
{
    rotation_dependency(early_trigger);
    if (COPIES) rows /= copies;
    if (rows_dev) {           // the number of rows in use was left on the device by an earlier kernel
        const int64_t r = *rows_dev;
        rows = r < 0 ? 0 : (r < rows ? r : rows);
    }
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    // B fragments of H16[k][n] = (-1)^popcount(k & n), constant per lane: n = 8 nt + g, k = 2 t + {0, 1} (+ 8)
    uint32_t hb[2][2];
#pragma unroll
    for (int nt = 0; nt < 2; nt++)
#pragma unroll
        for (int j = 0; j < 2; j++) {
            const int n16 = 8 * nt + g, k = 2 * t + 8 * j;
            hb[nt][j] = 0x3C003C00u | ((__popc(n16 & k) & 1) ? 0x8000u : 0u) | ((__popc(n16 & (k + 1)) & 1) ? 0x80000000u : 0u);
        }
    const uint32_t nblk = (uint32_t)(n >> 7);
    const uint32_t total = (uint32_t)((rows + 15) >> 4) * nblk;
    const uint32_t warp0 = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const uint32_t nwarps = gridDim.x * (blockDim.x >> 5);
    for (uint32_t blk = warp0; blk < total; blk += nwarps) {
        const uint32_t rb = blk / nblk, cb = blk - rb * nblk;
        const int64_t r0 = (int64_t)rb * 16 + g, r1 = r0 + 8;
        const bool ok0 = r0 < rows, ok1 = r1 < rows;
        const int64_t col = (int64_t)cb * 128 + 8 * t;
        // (see hadamard_kernel)
        const int64_t mb0 = !COPIES && member_rows && ok0 ? (uint32_t)r0 / (uint32_t)member_rows : 0;
        const int64_t mb1 = !COPIES && member_rows && ok1 ? (uint32_t)r1 / (uint32_t)member_rows : 0;
        uint4 xa[4], xb[4];
        {
            const int64_t s0 = ok0 ? (row_src ? row_src[r0] : r0 - mb0 * member_rows) : 0;
            const int64_t s1 = ok1 ? (row_src ? row_src[r1] : r1 - mb1 * member_rows) : 0;
            const T* p0 = x + s0 * x_row_stride + col;
            const T* p1 = x + s1 * x_row_stride + col;
#pragma unroll
            for (int q = 0; q < 4; q++) {
                xa[q] = ok0 ? Load8<T>::at(p0 + 32 * q) : make_uint4(0u, 0u, 0u, 0u);
                xb[q] = ok1 ? Load8<T>::at(p1 + 32 * q) : make_uint4(0u, 0u, 0u, 0u);
            }
            if (glu) {
                // the row holds [gate (n) | up (n)]: the input is fp16(act(gate) * up); all loads in flight first
                uint4 ua[4], ub[4];
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    ua[q] = ok0 ? Load8<T>::at(p0 + n + 32 * q) : make_uint4(0u, 0u, 0u, 0u);
                    ub[q] = ok1 ? Load8<T>::at(p1 + n + 32 * q) : make_uint4(0u, 0u, 0u, 0u);
                }
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    xa[q] = make_uint4(glu_pair(xa[q].x, ua[q].x, glu), glu_pair(xa[q].y, ua[q].y, glu),
                                       glu_pair(xa[q].z, ua[q].z, glu), glu_pair(xa[q].w, ua[q].w, glu));
                    xb[q] = make_uint4(glu_pair(xb[q].x, ub[q].x, glu), glu_pair(xb[q].y, ub[q].y, glu),
                                       glu_pair(xb[q].z, ub[q].z, glu), glu_pair(xb[q].w, ub[q].w, glu));
                }
            }
        }
        const int n_copies = COPIES ? copies : 1;
#pragma unroll 1
        for (int v = 0; v < n_copies; v++) {
            const int64_t o0 = COPIES ? r0 + v * rows : r0, o1 = COPIES ? r1 + v * rows : r1;
            uint4 la[4], lb[4];                                  // SPLIT: the second parts
            uint4 ya[4], yb[4];                                  // the products
#pragma unroll
            for (int q = 0; q < 4; q++) { ya[q] = xa[q]; yb[q] = xb[q]; }
            if (SPLIT && !pre)
#pragma unroll
                for (int q = 0; q < 4; q++) la[q] = lb[q] = make_uint4(0u, 0u, 0u, 0u);
            if (pre) {
                // (without pre_row, only the members of a group have multipliers of their own; a row out of use has the first ones)
                const int64_t mv = COPIES && member_rows ? v : 0;
                const __half* q0 = pre + (ok0 && pre_row ? (int64_t)pre_row[o0] : mb0 + mv) * n + col;
                const __half* q1 = pre + (ok1 && pre_row ? (int64_t)pre_row[o1] : mb1 + mv) * n + col;
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    const uint4 a = *reinterpret_cast<const uint4*>(q0 + 32 * q);
                    const uint4 b = *reinterpret_cast<const uint4*>(q1 + 32 * q);
                    if constexpr (SPLIT) {
                        split_product(ya[q].x, a.x, la[q].x); split_product(ya[q].y, a.y, la[q].y);
                        split_product(ya[q].z, a.z, la[q].z); split_product(ya[q].w, a.w, la[q].w);
                        split_product(yb[q].x, b.x, lb[q].x); split_product(yb[q].y, b.y, lb[q].y);
                        split_product(yb[q].z, b.z, lb[q].z); split_product(yb[q].w, b.w, lb[q].w);
                        continue;
                    }
                    ya[q].x = h2_as_u32(__hmul2(u32_as_h2(ya[q].x), u32_as_h2(a.x)));
                    ya[q].y = h2_as_u32(__hmul2(u32_as_h2(ya[q].y), u32_as_h2(a.y)));
                    ya[q].z = h2_as_u32(__hmul2(u32_as_h2(ya[q].z), u32_as_h2(a.z)));
                    ya[q].w = h2_as_u32(__hmul2(u32_as_h2(ya[q].w), u32_as_h2(a.w)));
                    yb[q].x = h2_as_u32(__hmul2(u32_as_h2(yb[q].x), u32_as_h2(b.x)));
                    yb[q].y = h2_as_u32(__hmul2(u32_as_h2(yb[q].y), u32_as_h2(b.y)));
                    yb[q].z = h2_as_u32(__hmul2(u32_as_h2(yb[q].z), u32_as_h2(b.z)));
                    yb[q].w = h2_as_u32(__hmul2(u32_as_h2(yb[q].w), u32_as_h2(b.w)));
                }
            }
            // c[2 q + s][nt]: columns 32 q' + 8 t + 4 s' + 2 nt + {0, 1} of rows g (first pair) and g + 8, for the
            // 16-point transform of group (q, s); the butterflies turn (q, s) into (q', s')
            uint64_t c[8][2][2];
#pragma unroll
            for (int q = 0; q < 4; q++)
#pragma unroll
                for (int s = 0; s < 2; s++) {
                    const uint32_t af[4] = {s ? ya[q].z : ya[q].x, s ? yb[q].z : yb[q].x, s ? ya[q].w : ya[q].y, s ? yb[q].w : yb[q].y};
#pragma unroll
                    for (int nt = 0; nt < 2; nt++) {
                        float d[4] = {0.f, 0.f, 0.f, 0.f};
                        mma_16816(d, af, hb[nt][0], hb[nt][1]);
                        if constexpr (SPLIT) {
                            const uint32_t lf[4] = {s ? la[q].z : la[q].x, s ? lb[q].z : lb[q].x, s ? la[q].w : la[q].y, s ? lb[q].w : lb[q].y};
                            mma_16816(d, lf, hb[nt][0], hb[nt][1]);
                        }
                        c[2 * q + s][nt][0] = f32x2(d[0], d[1]);
                        c[2 * q + s][nt][1] = f32x2(d[2], d[3]);
                    }
                }
            const uint64_t minus = f32x2(-1.f, -1.f), scale = f32x2(EXL3_HAD_SCALE, EXL3_HAD_SCALE);
#pragma unroll
            for (int h = 1; h < 8; h <<= 1)
#pragma unroll
                for (int i = 0; i < 8; i++) {
                    if (i & h) continue;
#pragma unroll
                    for (int nt = 0; nt < 2; nt++)
#pragma unroll
                        for (int r = 0; r < 2; r++) {
                            const uint64_t u = c[i][nt][r], v = c[i + h][nt][r];
                            c[i][nt][r] = add_f32x2(u, v);
                            c[i + h][nt][r] = fma_f32x2(v, minus, u);
                        }
                }
            auto put = [&](int64_t row, int r) {
                __half* o = out + row * n + col;
#pragma unroll
                for (int q = 0; q < 4; q++)
                    *reinterpret_cast<uint4*>(o + 32 * q) =
                        make_uint4(f16_pair(mul_f32x2(c[2 * q][0][r], scale)), f16_pair(mul_f32x2(c[2 * q][1][r], scale)),
                                   f16_pair(mul_f32x2(c[2 * q + 1][0][r], scale)), f16_pair(mul_f32x2(c[2 * q + 1][1][r], scale)));
            };
            if (ok0) put(o0, 0);
            if (ok1) put(o1, 1);
        }
    }
}

// ---- launchers ------------------------------------------------------------------------------

static int grid_for(int64_t warps_needed, int warps_per_block)
{
    int64_t blocks = (warps_needed + warps_per_block - 1) / warps_per_block;
    const int64_t cap = (int64_t)device_sm_count() * 8;
    if (blocks > cap) blocks = cap;
    if (blocks < 1) blocks = 1;
    return (int)blocks;
}

template <int K> static void launch_unpack_k(const uint32_t* t, int64_t n, uint16_t* o, cudaStream_t s)
{
    unpack_kernel<K><<<grid_for(n, 8), 256, 0, s>>>(t, n, o);
}

int launch_unpack(const uint32_t* trellis, int64_t n_tiles, int k, uint16_t* out, cudaStream_t s)
{
    switch (k) {
        case 1: launch_unpack_k<1>(trellis, n_tiles, out, s); break;
        case 2: launch_unpack_k<2>(trellis, n_tiles, out, s); break;
        case 3: launch_unpack_k<3>(trellis, n_tiles, out, s); break;
        case 4: launch_unpack_k<4>(trellis, n_tiles, out, s); break;
        case 5: launch_unpack_k<5>(trellis, n_tiles, out, s); break;
        case 6: launch_unpack_k<6>(trellis, n_tiles, out, s); break;
        case 7: launch_unpack_k<7>(trellis, n_tiles, out, s); break;
        case 8: launch_unpack_k<8>(trellis, n_tiles, out, s); break;
        default: return EXL3_E_K;
    }
    return check_launch();
}

template <int K>
static int launch_decode_k(const uint32_t* t, int64_t t_in, int64_t t_out, int cb, int64_t tn0,
                           int64_t tnc, __half* w, int64_t ld, cudaStream_t s)
{
    const int g = grid_for(t_in * tnc, 8);
    switch (cb) {
        case CB_3INST: decode_kernel<K, CB_3INST><<<g, 256, 0, s>>>(t, t_in, t_out, tn0, tnc, w, ld); break;
        case CB_MCG: decode_kernel<K, CB_MCG><<<g, 256, 0, s>>>(t, t_in, t_out, tn0, tnc, w, ld); break;
        case CB_MUL1: decode_kernel<K, CB_MUL1><<<g, 256, 0, s>>>(t, t_in, t_out, tn0, tnc, w, ld); break;
        default: return EXL3_E_CODEBOOK;
    }
    return check_launch();
}

int launch_decode(const uint32_t* trellis, int64_t t_in, int64_t t_out, int k, int cb, int64_t tn0,
                  int64_t tn_count, __half* w, int64_t ld, cudaStream_t s)
{
    switch (k) {
        case 1: return launch_decode_k<1>(trellis, t_in, t_out, cb, tn0, tn_count, w, ld, s);
        case 2: return launch_decode_k<2>(trellis, t_in, t_out, cb, tn0, tn_count, w, ld, s);
        case 3: return launch_decode_k<3>(trellis, t_in, t_out, cb, tn0, tn_count, w, ld, s);
        case 4: return launch_decode_k<4>(trellis, t_in, t_out, cb, tn0, tn_count, w, ld, s);
        case 5: return launch_decode_k<5>(trellis, t_in, t_out, cb, tn0, tn_count, w, ld, s);
        case 6: return launch_decode_k<6>(trellis, t_in, t_out, cb, tn0, tn_count, w, ld, s);
        case 7: return launch_decode_k<7>(trellis, t_in, t_out, cb, tn0, tn_count, w, ld, s);
        case 8: return launch_decode_k<8>(trellis, t_in, t_out, cb, tn0, tn_count, w, ld, s);
        default: return EXL3_E_K;
    }
}

int launch_table(int cb, __half* table, cudaStream_t s)
{
    switch (cb) {
        case CB_3INST: table_kernel<CB_3INST><<<256, 256, 0, s>>>(table); break;
        case CB_MCG: table_kernel<CB_MCG><<<256, 256, 0, s>>>(table); break;
        case CB_MUL1: table_kernel<CB_MUL1><<<256, 256, 0, s>>>(table); break;
        default: return EXL3_E_CODEBOOK;
    }
    return check_launch();
}

int launch_hadamard(const void* x, int x_dtype, int64_t rows, int64_t n, int64_t x_row_stride,
                    const __half* pre, const __half* post, __half* out, const int32_t* row_src,
                    const int32_t* pre_row, const int32_t* post_row, bool pdl, int out_mode,
                    cudaStream_t s, int glu, const int32_t* rows_dev, int member_rows, bool row_pairs,
                    bool wide_scales)
{
    if (rows * (n >> 7) >= ((int64_t)1 << 31)) return EXL3_E_RANGE;   // the kernel counts blocks in 32 bits
    // Many rows into a plain fp16 matrix (the prefill GEMM's operand): 16-row blocks on the tensor cores.
    // (a GLU over bf16 / fp32 rows stays on the butterfly kernel, which applies it before the fp16 rounding)
    // (a row count read from the device always takes this kernel, however few rows there may be)
    const bool mma = out_mode == HAD_OUT_F16 && !post && !post_row && ((rows >= kHadamardMmaMinRows && !wide_scales) || rows_dev) &&
                     (!glu || x_dtype == EXL3_DT_F16) &&
                     x_row_stride % 8 == 0 && (reinterpret_cast<uintptr_t>(x) & 15) == 0 &&
                     (!pre || (reinterpret_cast<uintptr_t>(pre) & 15) == 0) && (reinterpret_cast<uintptr_t>(out) & 15) == 0;
    if (rows_dev && !mma) return EXL3_E_UNSUPPORTED;
    // Rows that share a row of x: worth it where there are blocks enough without splitting them (below, 592 x 4 warps).
    int copies = !mma || rows_dev || glu ? 1 : row_pairs ? 2 : member_rows >= kHadamardMmaMinRows ? (int)(rows / member_rows) : 1;
    if (((rows / copies + 15) >> 4) * (n >> 7) < 4 * 16 * (int64_t)device_sm_count()) copies = 1;
    const int g = mma ? grid_for(((rows / copies + 15) >> 4) * (n >> 7), 8) : grid_for(rows * (n >> 7), 8);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(g);
    cfg.blockDim = dim3(256);
    cfg.dynamicSmemBytes = 0;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    const int early = pdl ? 1 : 0;
    cudaError_t e;
    if (mma) {
        const bool split = (member_rows > 0 && member_rows < kHadamardMmaMinRows) || wide_scales;
        auto launch = [&](auto* xt) {
            using T = std::remove_const_t<std::remove_pointer_t<decltype(xt)>>;
            const auto kernel = copies > 1 ? hadamard_mma_kernel<T, false, true> : split ? hadamard_mma_kernel<T, true, false> : hadamard_mma_kernel<T, false, false>;
            return cudaLaunchKernelEx(&cfg, kernel, xt, rows, n, x_row_stride, pre, out, row_src, pre_row, rows_dev, early, glu, member_rows, copies);
        };
        switch (x_dtype) {
            case EXL3_DT_F16: e = launch((const __half*)x); break;
            case EXL3_DT_BF16: e = launch((const __nv_bfloat16*)x); break;
            case EXL3_DT_F32: e = launch((const float*)x); break;
            default: return EXL3_E_DTYPE;
        }
        return note_cuda(e);
    }
    switch (x_dtype) {
        case EXL3_DT_F16:
            e = cudaLaunchKernelEx(&cfg, hadamard_kernel<__half>, (const __half*)x, rows, n,
                                   x_row_stride, pre, post, out, row_src, pre_row, post_row, early, out_mode, glu, member_rows);
            break;
        case EXL3_DT_BF16:
            e = cudaLaunchKernelEx(&cfg, hadamard_kernel<__nv_bfloat16>, (const __nv_bfloat16*)x,
                                   rows, n, x_row_stride, pre, post, out, row_src, pre_row, post_row,
                                   early, out_mode, glu, member_rows);
            break;
        case EXL3_DT_F32:
            e = cudaLaunchKernelEx(&cfg, hadamard_kernel<float>, (const float*)x, rows, n,
                                   x_row_stride, pre, post, out, row_src, pre_row, post_row, early, out_mode, glu, member_rows);
            break;
        default: return EXL3_E_DTYPE;
    }
    return note_cuda(e);
}

}  // namespace exl3
