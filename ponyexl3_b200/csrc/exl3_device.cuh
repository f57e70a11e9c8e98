// Device-only building blocks shared by the kernels: exact fp16 codebook
// arithmetic, the m16n8k16 fragment multiply, the 128-point Hadamard butterfly
// of one warp, and thin wrappers over the sm_100a asynchronous-copy / mbarrier /
// programmatic-launch instructions.  Every wait on an mbarrier is bounded.
#pragma once
#include <cuda_fp16.h>
#include <cuda_bf16.h>
#include <stdint.h>

#include "exl3_bits.cuh"

namespace exl3 {

// Status bits a kernel may set in the workspace status word.
enum : int {
    ST_WAIT_FULL_TIMEOUT = 1,    // a consumer gave up waiting for a staged item
    ST_WAIT_EMPTY_TIMEOUT = 2,   // the producer gave up waiting for a free stage
    ST_TC_TIMEOUT = 4,           // a tensor-core pipeline wait gave up
    ST_BAD_LAUNCH = 8,           // a kernel found its launch (shared memory, cluster) not as planned
    ST_PEER_TIMEOUT = 16,        // a wait for the other GPUs' output blocks gave up
};

// ---- codebooks: exact fp16 arithmetic -------------------------------------------------

__device__ __forceinline__ uint32_t h2_as_u32(__half2 h) { return *reinterpret_cast<uint32_t*>(&h); }
__device__ __forceinline__ __half2 u32_as_h2(uint32_t u) { return *reinterpret_cast<__half2*>(&u); }

// Two codewords -> one register holding (w_a, w_b) as fp16, bit-exact with the
// reference codebooks (ponyexl3/ref/codebook.py:66-91): 3INST / MCG add the two
// fp16 halves of the scrambled word with one rounding; MUL1 sends the fp16
// pattern 0x6400 + byte-sum through one fused multiply-add.
template <int CB> __device__ __forceinline__ uint32_t decode_pair(uint32_t cw_a, uint32_t cw_b)
{
    const uint32_t xa = codebook_word<CB>(cw_a);
    const uint32_t xb = codebook_word<CB>(cw_b);
    if (CB == CB_MUL1) {
        const uint32_t s = xa | (xb << 16);
        const __half2 kinv = u32_as_h2(0x1EEE1EEEu), kbias = u32_as_h2(0xC931C931u);
        return h2_as_u32(__hfma2(u32_as_h2(s), kinv, kbias));
    }
    const uint32_t lo = __byte_perm(xa, xb, 0x5410);   // (lo_a, lo_b)
    const uint32_t hi = __byte_perm(xa, xb, 0x7632);   // (hi_a, hi_b)
    return h2_as_u32(__hadd2(u32_as_h2(lo), u32_as_h2(hi)));
}

template <int CB> __device__ __forceinline__ __half decode_one(uint32_t cw)
{
    return __low2half(u32_as_h2(decode_pair<CB>(cw, cw)));
}

// ---- tensor-core fragment multiply ------------------------------------------------------

// D(16x8, f32) += A(16x16, f16, row) * B(16x8, f16, col).  The packed tile order of
// EXL3 is exactly the A-fragment order of W^T (out x in), so decoded registers feed
// this directly (a0: codewords 0,1; a1: 4,5; a2: 2,3; a3: 6,7 of the lane).
__device__ __forceinline__ void mma_16816(float (&d)[4], const uint32_t (&a)[4], uint32_t b0,
                                          uint32_t b1)
{
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, "
        "{%8,%9}, {%0,%1,%2,%3};\n"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// ---- two fp32 values per instruction ----------------------------------------------------------

__device__ __forceinline__ uint64_t f32x2(float lo, float hi)
{
    return (uint64_t)__float_as_uint(lo) | ((uint64_t)__float_as_uint(hi) << 32);
}
__device__ __forceinline__ uint64_t add_f32x2(uint64_t a, uint64_t b)
{
    uint64_t r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ uint64_t mul_f32x2(uint64_t a, uint64_t b)
{
    uint64_t r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ uint64_t fma_f32x2(uint64_t a, uint64_t b, uint64_t c)
{
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ uint32_t f16_pair(uint64_t v)
{
    return h2_as_u32(__floats2half2_rn(__uint_as_float((uint32_t)v), __uint_as_float((uint32_t)(v >> 32))));
}

// ---- Hadamard ---------------------------------------------------------------------------

// In-place 128-point Sylvester Hadamard of a block spread over one warp, lane l
// holding elements 4l..4l+3; un-normalised (caller scales by 1/sqrt(128)).
__device__ __forceinline__ void had128_warp(float (&v)[4], int lane)
{
    float a = v[0] + v[1], b = v[0] - v[1], c = v[2] + v[3], d = v[2] - v[3];
    v[0] = a + c; v[1] = b + d; v[2] = a - c; v[3] = b - d;
#pragma unroll
    for (int m = 1; m < 32; m <<= 1) {
        const bool upper = (lane & m) != 0;
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const float o = __shfl_xor_sync(0xFFFFFFFFu, v[i], m);
            v[i] = upper ? (o - v[i]) : (v[i] + o);
        }
    }
}

#define EXL3_HAD_SCALE 0.08838834764831845f

// ---- gated linear unit ------------------------------------------------------------------------

// act(g) * u in fp32 (the caller rounds to fp16): mode 1 = SiLU, 2 = tanh-GELU, the two
// activations of the reference's SwitchGLU (ponyexl3/mlx/exl3_moe.py:62-75).
enum : int { GLU_NONE = 0, GLU_SILU = 1, GLU_GELU = 2 };
// g / (1 + exp(-g)).  The division is a product with the approximate reciprocal and one correction by the
// residual (Markstein, IBM J. Res. Dev. 34, 1990), without the division's branch, which kept a rotation from
// overlapping the elements of a row: SwitchGLU of 4096 tokens 507 -> 499 us, MLP of 300 rows 167 -> 162.  Outside
// (-87, 87), where the reciprocal would leave fp32, the result is g or -0 (NaN for NaN and minus infinity), so that
// bf16 and fp32 gates of any size are right too.  All 65,536 fp16 gates give the division's float where that is
// above 1e-35 (only -0 gives +0).
__device__ __forceinline__ float silu(float g)
{
    const float d = 1.f + __expf(-g);
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(d));
    const float q = g * r;
    return fabsf(g) < 87.f ? __fmaf_rn(__fmaf_rn(-q, d, g), r, q) : g * __saturatef(g);
}
__device__ __forceinline__ float glu_value(float g, float u, int mode)
{
    if (mode == GLU_GELU)
        return 0.5f * g * (1.f + tanhf(0.797884560803f * (g + 0.044715f * g * g * g))) * u;
    return silu(g) * u;
}

// ---- shared-memory barriers and bulk copies ------------------------------------------------

__device__ __forceinline__ uint32_t smem_u32(const void* p)
{
    return (uint32_t)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(bar), "r"(count));
}

__device__ __forceinline__ void mbar_fence_init()
{
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
}

__device__ __forceinline__ void mbar_arrive(uint32_t bar)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(bar) : "memory");
}

__device__ __forceinline__ void mbar_arrive_expect_tx(uint32_t bar, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(bar), "r"(bytes)
                 : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity)
{
    uint32_t ok;
    asm volatile(
        "{\n.reg .pred p;\n"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        "selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}

// Bounded wait: false after kWaitSpins unsuccessful polls (each poll already
// blocks for a hardware-defined interval).
constexpr uint32_t kWaitSpins = 1u << 20;
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity)
{
    for (uint32_t i = 0; i < kWaitSpins; i++)
        if (mbar_try_wait(bar, parity)) return true;
    return false;
}

__device__ __forceinline__ void prefetch_l1(const void* p) { asm volatile("prefetch.global.L1 [%0];\n" ::"l"(p)); }
__device__ __forceinline__ void prefetch_l2(const void* p) { asm volatile("prefetch.global.L2 [%0];\n" ::"l"(p)); }

// Programmatic dependent launch: let the next kernel of the stream start its
// independent prologue / wait until the kernels this one depends on have finished.
__device__ __forceinline__ void griddep_launch_dependents()
{
    asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
}
__device__ __forceinline__ void griddep_wait() { asm volatile("griddepcontrol.wait;\n" ::: "memory"); }

__device__ __forceinline__ void named_bar_sync(int id, int threads)
{
    asm volatile("bar.sync %0, %1;\n" ::"r"(id), "r"(threads) : "memory");
}

// ---- thread-block clusters: barrier, and the shared memory of CTA `rank` ----
__device__ __forceinline__ void cluster_sync()
{
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}
__device__ __forceinline__ void cluster_arrive_relaxed() { asm volatile("barrier.cluster.arrive.relaxed.aligned;\n" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory"); }
__device__ __forceinline__ uint32_t cluster_address(uint32_t addr, int rank)
{
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
__device__ __forceinline__ void st_cluster_f32x4(uint32_t addr, const float4& v)
{
    asm volatile("st.shared::cluster.v4.f32 [%0], {%1,%2,%3,%4};\n" ::"r"(addr), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w) : "memory");
}
__device__ __forceinline__ float ld_cg_f32(const float* p)
{
    float v;
    asm volatile("ld.global.cg.f32 %0, [%1];\n" : "=f"(v) : "l"(p));
    return v;
}

}  // namespace exl3
