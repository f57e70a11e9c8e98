// Trellis encoder: exact Viterbi search of 16x16 tiles over the bitshift trellis, the
// converter's side of the EXL3 format (reference: quantize_tile_reference,
// ponyexl3/convert/reference_search.py:30-87, itself the parity oracle of the reference's
// search kernel).
//
// A tile is 256 weights in codeword order.  The trellis has 65,536 states (the 16-bit windows);
// a step appends K bits, s' = ((s << K) | j) & 0xFFFF, so the predecessors of s' are
// (s' >> K) | (j << (16 - K)), j = 0 .. 2^K - 1.  Path cost = sum of (codebook(s_t) - w[t])^2 in
// float64 with the product and the sum rounded separately, the FIRST minimum winning among
// predecessors and among final states, exactly as the reference's numpy code, so the chosen
// states are bit-identical.  The bitstream is tail-biting (codeword 0's window reaches back into
// codeword 255's): a free pass proposes the closing state, pinned passes start from it until
// the path's pre-state of step 0 and its last state both equal the pin (at most max_pins passes).
//
// search_kernel runs the recursion from the tile's end: B_t[b], the least cost of steps t .. 255 from base b = s_t >> K,
//   B_t[b] = min_n ( (codebook(b << K | n) - w_t)^2 + B_t+1[(b << K | n) mod 2^(16-K)] )
// with the chosen n kept for every base and step.  One such pass answers the free search (the cheapest of all
// B_0) and every pinned one (the path from the pinned base), where the reference's recursion from the start needs a
// pass of 255 steps for each: two for most tiles, up to five.  The sums are rounded in another order, so a result
// is only taken if it cannot depend on that: every decision on the path is further from its runner-up than the
// rounding of float64 sums of that size (2^-42), or a tie of equal errors at either end of the path, where both orders take
// the first.  Tiles where that fails (exact ties: one tile in some thousands at K <= 6, one in three at K = 8 with MUL1's
// thousand values) are marked, and encode_kernel searches them from the start, in the reference's order.
//
// The 2^K bases with the same b mod 2^(16-2K) share their successors, so all that a step hands on is one cost per base,
// 2^(16-K) numbers instead of 65,536.  For K >= 2 they fit the SM's shared memory and a tile is searched by
// one CTA without leaving it; only the pointers (one byte per base and step) go to L2.
//   * A thread owns the same 128 of the 65,536 (base, n) pairs in every step and keeps their codebook values in
//     registers; its bases are taken from one group where K allows.  A group's successors are neighbours, read
//     16 bytes at a time.
//   * The minimum over n is found in fp32 (two values per instruction) on keys with n in their low
//     bits, relative to a lower bound of all costs, together with the gap to the runner-up; the
//     winner's cost is then computed in float64.  Where the gap is inside the
//     error bound of the fp32 keys (about one base in a thousand; exact ties too) the thread takes the
//     minimum over all n in float64.  fp32 rounding therefore never reaches a result.
//   * K = 2 has 16,384 bases, 192 KiB for one set of costs: the group of a thread (four reads, four
//     writes) is updated in place, which rotates the address of a base by K bits per step.
//   * K = 1 (32,768 bases, 384 KiB) keeps its costs in L2 and compares its two successors in float64.
//   * The walk along the pointers streams them through shared memory, 32 KiB at a time, 20 K clocks a tile (as a
//     chain of L2 round trips it took 90 K); a pinned path is only walked to where it meets the one before.
// Tiles are handed out by a counter.
//
// Bound: instruction issue (some 60 % of the slots, the logic pipe as busy), 8 warp instructions per 32 states and step (the
// keys, their minimum and the gap are three of them).  592 tiles of a 256 x 592 matrix, K = 4: 10.0 -> 3.8 ms
// against the search from the start; at K = 2, 3, 5, 6, 7, 8 (3INST) 9.4, 4.9, 3.4, 3.2, 3.4, 6.4 ms (518 tiles of the
// search from the start: 29.0, 12.5, 7.0, 7.2, 7.9, 10.2; K = 8 leaves one tile to encode_kernel).  1024 threads of half the
// registers, for more warps to choose from, took 4.3 ms at K = 4.

#include <cuda_fp16.h>

#include <algorithm>

#include "exl3_bits.cuh"
#include "exl3_device.cuh"
#include "exl3_internal.h"

namespace exl3 {

constexpr int kEncStates = 65536;
constexpr int kEncThreads = 512;
constexpr size_t kEncCounterBytes = 256;                 // counters in front of the slots
constexpr size_t kEncBackBytes = 256 * (size_t)(kEncStates / 2);
constexpr size_t kEncCostBytes = 2 * (size_t)(kEncStates / 2) * sizeof(double);   // K = 1, and odd tiles
constexpr size_t kEncSlotBytes = kEncBackBytes + kEncCostBytes;

// With weights up to here a path costs less than 256 x 1e26, far from the 1e30 of states that the pinned one cannot
// reach, which a cost can therefore be told from, and every cost is a number.
constexpr float kEncLargest = 1e13f;

struct EncodeArgs {
    const float* w;        // (n_tiles, 256) codeword order
    int64_t n_tiles;
    int max_pins;
    uint16_t* states;      // (n_tiles, 256) the 16-bit window of every codeword
    uint32_t* packed;      // NULL or (n_tiles, 8K) packed tile words
    unsigned* counter;     // tiles handed out so far by this kernel
    unsigned* left;        // tiles that search_kernel has left: [0] in doubt, [1] odd
    uint8_t* slots;        // gridDim.x workspace slots
};

// A tile that search_kernel leaves is marked in its first two states, which are no trellis path for any K.
enum : int { kEncDoubt = 0, kEncOdd = 1 };

constexpr int kEncClose = 64;
struct EncodeShared {
    double red_c[32];
    double red_u[32];
    int red_s[32];
    float w[256];
    uint16_t states[256];
    uint32_t words[64];
    unsigned smin[3];
    int fin, pin, done;
    unsigned tile;
    // search_kernel
    float sums[32];
    int merged;
    int n_close;                       // decisions that might be: step << 16 | base, and by how much
    uint32_t close_at[kEncClose];
    double close_gap[kEncClose];
};

__device__ __forceinline__ double sq_err(double c, double w)
{
    const double d = c - w;
    return __dmul_rn(d, d);
}
// (Converted to float64 by the instruction, here and below: as six integer ones, 592 tiles of K = 1 took 11.2 ms for 10.5, and
// tiles of zeros at K = 8 with MUL1, which the search from the start answers, 50.2 for 43.9.)
template <int CB> __device__ __forceinline__ float codebook_f32(uint32_t s) { return __half2float(decode_one<CB>(s)); }

// The cheapest final state, the lowest index among equals, over the CTA; (bc, bs) is the thread's own.
__device__ __forceinline__ void final_state(EncodeShared& sh, double bc, int bs, int warps)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        const double oc = __shfl_down_sync(0xFFFFFFFFu, bc, off);
        const int os = __shfl_down_sync(0xFFFFFFFFu, bs, off);
        if (oc < bc || (oc == bc && os < bs)) { bc = oc; bs = os; }
    }
    if (lane == 0) { sh.red_c[warp] = bc; sh.red_s[warp] = bs; }
    __syncthreads();
    if (warp == 0) {
        bc = sh.red_c[lane < warps ? lane : 0];
        bs = sh.red_s[lane < warps ? lane : 0];
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) {
            const double oc = __shfl_down_sync(0xFFFFFFFFu, bc, off);
            const int os = __shfl_down_sync(0xFFFFFFFFu, bs, off);
            if (oc < bc || (oc == bc && os < bs)) { bc = oc; bs = os; }
        }
        if (lane == 0) sh.fin = bs;
    }
    __syncthreads();
}

// Walk of one warp over the back-pointers, two steps per round trip to L2.
template <int K> __device__ __forceinline__ void walk_back(EncodeShared& sh, const uint8_t* back, int pass)
{
    constexpr int NB = kEncStates >> K, J = 1 << K, R = (J + 31) / 32;
    const int lane = threadIdx.x & 31;
    uint32_t s = (uint32_t)sh.fin;
    for (int t = 255; t >= 0; t -= 2) {
        const uint32_t j0 = __ldcg(back + (size_t)t * NB + (s >> K));
        uint32_t v[R];
#pragma unroll
        for (int r = 0; r < R; r++) {
            const uint32_t j = (uint32_t)(lane + 32 * r) & (J - 1);
            v[r] = __ldcg(back + (size_t)(t - 1) * NB + ((s | (j << 16)) >> (2 * K)));
        }
        if (lane == 0) sh.states[t] = (uint16_t)s;
        s = (s >> K) | (j0 << (16 - K));
        if (lane == 0) sh.states[t - 1] = (uint16_t)s;
        uint32_t j1 = v[0];
#pragma unroll
        for (int r = 1; r < R; r++)
            if ((int)(j0 >> 5) == r) j1 = v[r];
        j1 = __shfl_sync(0xFFFFFFFFu, j1, (int)(j0 & 31));
        s = (s >> K) | (j1 << (16 - K));
    }
    __syncwarp();
    if (lane == 0) {
        const int last = sh.states[255];
        if (pass > 0 && (int)s == sh.pin && last == sh.pin) sh.done = 1;
        sh.pin = last;
    }
}

// States and, when asked for, the packed tile: the low K bits of every codeword, MSB first in codeword
// order, as little-endian 32-bit words (ponyexl3/ref/trellis.py:12-50).
template <int K> __device__ __forceinline__ void store_tile(EncodeShared& sh, const EncodeArgs& a, int64_t tile)
{
    const int tid = threadIdx.x;
    if (tid < 256) a.states[tile * 256 + tid] = sh.states[tid];
    if (a.packed) {
        if (tid < 64) sh.words[tid] = 0u;
        __syncthreads();
        if (tid < 256) {
            const uint32_t v = sh.states[tid] & (uint32_t)((1 << K) - 1);
            for (int b = 0; b < K; b++)
                if ((v >> (K - 1 - b)) & 1u) {
                    const int pos = tid * K + b;
                    atomicOr(&sh.words[pos >> 5], 1u << (31 - (pos & 31)));
                }
        }
        __syncthreads();
        if (tid < 8 * K) a.packed[tile * 8 * K + tid] = sh.words[tid];
    }
    __syncthreads();
}

// The next tile for this CTA (n_tiles or more: none left), its weights in shared memory; MARK: of those that
// search_kernel has marked so.
template <int MARK = -1> __device__ __forceinline__ int64_t next_tile(EncodeShared& sh, const EncodeArgs& a)
{
    const int tid = threadIdx.x;
    if (tid == 0) {
        unsigned t;
        do {
            t = atomicAdd(a.counter, 1u);
        } while (MARK >= 0 && t < a.n_tiles && !(a.states[(int64_t)t * 256] == 0xFFFF && (int)a.states[(int64_t)t * 256 + 1] == MARK));
        sh.tile = t;
        sh.pin = -1;
        sh.done = 0;
    }
    __syncthreads();
    const int64_t tile = sh.tile;
    if (tile < a.n_tiles && tid < 256) sh.w[tid] = a.w[tile * 256 + tid];
    __syncthreads();
    return tile;
}

// (k & ~(J - 1)) | j as one three-input operation (written in C, ptxas made two of it).
template <int J> __device__ __forceinline__ uint32_t key_with_index(uint32_t k, uint32_t j)
{
    uint32_t r;
    asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(r) : "r"(k), "n"(~(J - 1)), "r"(j));
    return r;
}

// How the 65,536 (b, n) pairs of a step of the backward search are dealt to the threads.  The bases b with the same
// h = b mod 2^(16-2K) have the same successors, (h << K) | n.
template <int K> struct SearchSplit {
    static constexpr int NT = kEncThreads;               // threads
    static constexpr int kPairs = kEncStates / NT;       // pairs per thread
    static constexpr int NB = kEncStates >> K;           // bases
    static constexpr int J = 1 << K;
    static constexpr int HB = 16 - 2 * K;                // bits of h
    static constexpr int NH = 1 << HB;                   // groups
    static constexpr int JT = J < kPairs ? J : kPairs;   // n values per thread and base
    static constexpr int TB = J / JT;                    // threads of a base: more than one for the largest K
    static constexpr int NG = NH < NT ? NH : NT;
    static constexpr int G = NH / NG;                    // groups per thread
    static constexpr int L = kPairs / JT / G;            // bases per thread and group: (l0 + T i) << HB | h, i < L
    static constexpr int T = J / L;
    static constexpr int JC = JT < 16 ? JT : 16;         // n values per turn
    static constexpr int BL = L < 4 ? L : 4;             // bases whose costs are made at a time (all of them at once spill)
    static constexpr bool kInPlace = K == 2;
    // Every how many steps a tile with too many close decisions is left.  At K = 8 MUL1's thousand values tie at most bases of a
    // zero weight: 592 tiles of zeros take 44 ms this way, nearly all of it the search from the start, and 20 more with the whole
    // search before they are left; others take 1 % longer.  At lower K such tiles are few, or fill the list up late.
    static constexpr int kLook = K == 8 ? 16 : 256;
    static constexpr size_t kCost = (size_t)NB * (kInPlace ? 1 : 2) * (sizeof(double) + sizeof(float));
    static constexpr int kChunk = 32768;                 // bytes of pointers fetched at a time by the walk
    static constexpr int kRowBytes = NB;                 // pointers of a step
    static constexpr int kRows = kChunk / kRowBytes;     // ... steps
    static constexpr size_t kSmem = kCost > 2 * kChunk ? kCost : 2 * kChunk;
    static constexpr int kThreads = NT;
    // The byte of a step's row that holds base b's pointer (a thread's L pointers lie side by side), and the pointer in it.
    static __device__ __forceinline__ uint32_t at(uint32_t b)
    {
        if (TB > 1) return b;
        const uint32_t h = b & (NH - 1), q = b >> HB;
        return ((h / NG) * NT + (q % T) * NG + (h & (NG - 1))) * L + q / T;
    }
    static __device__ __forceinline__ uint32_t pick(uint8_t byte, uint32_t) { return byte; }
};
// K = 1: 1024 threads, a pointer is a bit.
template <> struct SearchSplit<1> {
    static constexpr int NB = kEncStates / 2, J = 2, HB = 14, NH = 1 << HB;
    static constexpr int NT = 1024, kThreads = 1024, kRowBytes = NB / 8;
    static constexpr int kChunk = 32768, kRows = kChunk / kRowBytes;
    static constexpr size_t kSmem = 2 * kChunk;
    static __device__ __forceinline__ uint32_t at(uint32_t b) { return b >> 3; }
    static __device__ __forceinline__ uint32_t pick(uint8_t byte, uint32_t b) { return (byte >> (b & 7)) & 1u; }
};

// The path from base b0 over the pointers, 32 KiB of them at a time through shared memory, by one thread.  From where
// it meets the path in sh.states (MEET) it is that path.
template <int K> __device__ __forceinline__ void walk_ahead(EncodeShared& sh, uint8_t* stage, const uint8_t* ptr, uint32_t b0, bool meet)
{
    using E = SearchSplit<K>;
    const int tid = threadIdx.x;
    auto fetch = [&](int c) {
        for (int o = 16 * tid; o < E::kChunk; o += 16 * E::kThreads)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(stage + (c & 1) * E::kChunk + o)),
                         "l"(ptr + (size_t)c * E::kChunk + o)
                         : "memory");
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    constexpr int kChunks = 256 / E::kRows;
    if (tid == 0) sh.merged = 0;
    fetch(0);
    uint32_t b = b0;
    for (int c = 0; c < kChunks; c++) {
        if (c + 1 < kChunks) {
            fetch(c + 1);
            asm volatile("cp.async.wait_group 1;" ::: "memory");
        } else {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
        }
        __syncthreads();
        if (tid == 0) {
            const uint8_t* rows = stage + (c & 1) * E::kChunk;
            for (int r = 0; r < E::kRows; r++) {
                const uint32_t s = (b << K) | E::pick(rows[r * E::kRowBytes + E::at(b)], b);
                b = s & (E::NB - 1);
                const int t = c * E::kRows + r;
                const bool met = meet && ((sh.states[t] ^ s) & (E::NB - 1)) == 0;
                sh.states[t] = (uint16_t)s;
                if (met) { sh.merged = 1; break; }
            }
        }
        __syncthreads();
        if (sh.merged) break;
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
}

// A tile that the search leaves to the kernels behind it.
__device__ __forceinline__ void leave_tile(const EncodeArgs& a, int64_t tile, int why)
{
    a.states[tile * 256] = 0xFFFF;
    a.states[tile * 256 + 1] = (uint16_t)why;
    atomicAdd(a.left + why, 1u);
}

// What a tile's paths should cost at most: far more than K bits usually leave, and what lies beyond the bulk of the
// codebooks, twice where one or two bits cannot follow large weights of changing sign.  (A tile whose path costs more is in
// doubt.  592 tiles of standard deviation 10, K = 1 with 3INST and K = 2 with MUL1: 38.9 and 25.3 ms without the 2, 11.3 and 8.2
// with it.)  Two paths whose float64 costs, summed in any order, are further apart than 2^-42 of the cost are in the right
// order; a decision that fp32 leaves unsure, or by less than twice `close`, 2^-41 of the bound, is made in float64, and noted
// if it is closer than that.  False: the tile is not for this search.
__device__ __forceinline__ bool cost_bound(EncodeShared& sh, float per_weight, float per_outlier, float& bound)
{
    const int tid = threadIdx.x;
    const float w = tid < 256 ? sh.w[tid] : 0.f, over = fmaxf(fabsf(w) - 2.5f, 0.f);
    float sum = over * over;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xFFFFFFFFu, sum, o);
    if ((tid & 31) == 0) sh.sums[tid >> 5] = sum;
    if (tid == 0) sh.n_close = 0;
    if (__syncthreads_or(!(fabsf(w) < kEncLargest))) return false;
    bound = 256.f * per_weight;
#pragma unroll
    for (int i = 0; i < 8; i++) bound += per_outlier * sh.sums[i];
    return true;
}
__device__ __forceinline__ void note_close(EncodeShared& sh, int t, uint32_t base, double gap)
{
    const int at = atomicAdd(&sh.n_close, 1);
    if (at < kEncClose) {
        sh.close_at[at] = ((uint32_t)t << 16) | base;
        sh.close_gap[at] = gap;
    }
}

// For all threads, between two steps: whether more decisions have been noted than there is room for, which leaves the tile
// in doubt whatever comes.
__device__ __forceinline__ bool too_close(EncodeShared& sh)
{
    return __syncthreads_or(sh.n_close > kEncClose);
}

// The paths of a tile from the pointers of all its bases, `cost` giving a base's cost to the end of the tile: the free
// path, then the pinned ones until one closes.  False: a decision on one of them is too close to be told.
template <int K, int CB, typename Cost>
__device__ __forceinline__ bool search_paths(EncodeShared& sh, uint8_t* stage, const uint8_t* ptr, int max_pins, float bound, Cost&& cost)
{
    using E = SearchSplit<K>;
    constexpr int NB = E::NB, kWarps = E::kThreads / 32;
    const int tid = threadIdx.x;
    // The free path starts at the cheapest base.  Bases of a group whose first codewords have the same error cost the
    // same to the bit, and the lowest wins, in whatever order the costs are summed, if the paths behind are one.  (Totals that
    // are the same to the bit do not say so: the search from the start compares the first errors alone, and two that
    // differ by less than the total's last place decide it.)
    uint32_t b0;
    bool unsure_start;
    {
        double bc = 1e300, second = 1e300;
        int bs = 0;
        auto merge = [&](double oc, double ou, int os) {
            if (oc == bc && ((os ^ bs) & (E::NH - 1)) == 0) {
                second = fmin(second, ou);
                bs = min(bs, os);
            } else {
                second = fmin(fmax(bc, oc), fmin(second, ou));
                if (oc < bc) { bc = oc; bs = os; }
            }
        };
        for (int b = tid; b < NB; b += E::kThreads) merge(cost((uint32_t)b), 1e300, b);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const double oc = __shfl_xor_sync(0xFFFFFFFFu, bc, o), ou = __shfl_xor_sync(0xFFFFFFFFu, second, o);
            const int os = __shfl_xor_sync(0xFFFFFFFFu, bs, o);
            merge(oc, ou, os);
        }
        if ((tid & 31) == 0) { sh.red_c[tid >> 5] = bc; sh.red_u[tid >> 5] = second; sh.red_s[tid >> 5] = bs; }
        __syncthreads();
        bc = sh.red_c[0]; second = sh.red_u[0]; bs = sh.red_s[0];
        for (int i = 1; i < kWarps; i++) merge(sh.red_c[i], sh.red_u[i], sh.red_s[i]);
        b0 = (uint32_t)bs;
        bool other = false;
        if (tid < E::J) {
            const uint32_t b = ((uint32_t)tid << E::HB) | (b0 & (E::NH - 1));
            const uint32_t s = (b << K) | E::pick(__ldcg(ptr + E::at(b)), b), s0 = (b0 << K) | E::pick(__ldcg(ptr + E::at(b0)), b0);
            auto first = [&](uint32_t state) { return sq_err((double)codebook_f32<CB>(state), (double)sh.w[0]); };
            other = cost(b) == bc && ((s ^ s0) & (E::J - 1) || first(s) != first(s0));
        }
        unsure_start = __syncthreads_or(other) || !(second - bc > bc * 2.3e-13);       // 2^-42
    }
    for (int pass = 0; pass <= max_pins; pass++) {
        const int pin = pass ? (int)sh.states[255] : -1;
        __syncthreads();
        walk_ahead<K>(sh, stage, ptr, pass ? (uint32_t)pin & (NB - 1) : b0, pass > 0);
        // its cost, and whether one of its decisions is too close to be told
        double e = 0.0;
        if (tid < 256) e = sq_err((double)codebook_f32<CB>(sh.states[tid]), (double)sh.w[tid]);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) e += __shfl_xor_sync(0xFFFFFFFFu, e, o);
        if ((tid & 31) == 0) sh.red_c[tid >> 5] = e;
        __syncthreads();
        double total = 0.0;
#pragma unroll
        for (int i = 0; i < 8; i++) total += sh.red_c[i];
        bool doubt = sh.n_close > kEncClose || (pass == 0 && unsure_start) || !(total <= (double)bound);
        for (int i = tid; i < min(sh.n_close, kEncClose); i += E::kThreads) {
            const uint32_t at = sh.close_at[i];
            if ((uint32_t)(sh.states[at >> 16] >> K) == (at & 0xFFFFu) && !(sh.close_gap[i] > total * 2.3e-13)) doubt = true;
        }
        if (__syncthreads_or(doubt)) return false;
        if (pass > 0 && (int)sh.states[255] == pin) break;
    }
    return true;
}

template <int K, int CB>
__global__ void __launch_bounds__(kEncThreads, 1) search_kernel(const EncodeArgs a)
{
    using E = SearchSplit<K>;
    constexpr int NB = E::NB, J = E::J, L = E::L, G = E::G, JC = E::JC, BL = E::BL, HB = E::HB, LB = 16 - K;
    // Two fp32 keys whose bit patterns differ by less than this may be in the wrong order: the low K
    // bits hold n (2^K units), the arithmetic before is off by at most four units on either side; twice
    // that, rounded up.
    constexpr uint32_t kGap = 4u * J + 32u;
    extern __shared__ __align__(16) uint8_t smem[];
    __shared__ EncodeShared sh;
    double* md0 = reinterpret_cast<double*>(smem);
    float* mf0 = reinterpret_cast<float*>(md0 + (E::kInPlace ? 1 : 2) * NB);
    const int tid = threadIdx.x;
    uint8_t* ptr = a.slots + (size_t)blockIdx.x * kEncSlotBytes;

    const uint32_t h0 = (uint32_t)tid & (E::NG - 1);
    const uint32_t l0 = (uint32_t)(tid / E::NG);
    // several threads of a base are lanes 32 / TB apart
    constexpr int kLanes = 32 / E::TB;
    const uint32_t b_own = (uint32_t)((tid & (kLanes - 1)) | ((tid >> 5) * kLanes));
    const uint32_t n_first = (uint32_t)(((tid & 31) / kLanes) * E::JT);
    auto base = [&](int g, int i) -> uint32_t { return E::TB > 1 ? b_own : ((l0 + E::T * i) << HB) | (h0 + E::NG * g); };

    uint32_t cbr[G * L][E::JT / 2];
#pragma unroll
    for (int g = 0; g < G; g++)
#pragma unroll
        for (int i = 0; i < L; i++)
#pragma unroll
            for (int q = 0; q < E::JT / 2; q++) {
                const uint32_t s = (base(g, i) << K) + n_first + 2 * q;
                cbr[g * L + i][q] = decode_pair<CB>(s, s + 1);
            }

    // Address of base b.  The fp32 costs of a group's successors are read as 16-byte pieces: piece c of row r = b >> K lies
    // at c ^ row_xor(r), so that a quarter warp's reads of neighbouring rows fall into different banks.  In place, b is rotated by
    // the bits of the steps taken so far, and its low nibble XOR-ed with the others, because neighbours are then at
    // any power-of-two stride.
    auto row_xor = [](uint32_t r) -> uint32_t { return K == 3 ? (r >> 2) & 1u : K == 4 ? (r >> 1) & 3u : K == 8 ? 0u : r & 7u; };
    auto slot = [&](uint32_t b, int rot) -> uint32_t {
        if (!E::kInPlace) return b;
        b = ((b << rot) | (b >> (LB - rot))) & (NB - 1);
        return b ^ (((b >> 4) ^ (b >> 8) ^ (b >> 12)) & 15u);
    };
    // (row_xor does not depend on i or g: base(g, i) lies T << HB and 512 apart, above the bits that it takes)
    const uint32_t first_f = E::kInPlace ? 0u : base(0, 0) ^ (row_xor(base(0, 0) >> K) << 2);

    for (;;) {
        const int64_t tile = next_tile(sh, a);
        if (tile >= a.n_tiles) return;
        if (tid == 0) sh.smin[0] = sh.smin[1] = 0x7F800000u;
        for (int b = tid; b < NB; b += E::NT) { md0[b] = 0.0; mf0[b] = 0.f; }
        float bound;
        if (!cost_bound(sh, 32.f / (float)(1 << (2 * K)), K == 2 ? 2.f : 1.f, bound)) {
            if (tid == 0) leave_tile(a, tile, kEncOdd);
            continue;
        }
        const double close = (double)bound * 0x1p-41;
        // ... so fp32 keys of at least `near` decide if their bit patterns are kGap apart: that is 2^-20 of them or more
        const uint32_t near = __float_as_uint(bound * 0x1p-20f);

        double off = 0.0;                                // lower bound of every cost of the step
        bool left = false;
#pragma unroll 1
        for (int u = 0; u < 256; u++) {
            const int t = 255 - u;
            const int cur = E::kInPlace ? 0 : (u & 1), nxt = E::kInPlace ? 0 : cur ^ 1;
            const int rot = E::kInPlace ? (K * u) % LB : 0;
            const double* mdc = md0 + cur * NB;
            const float* mfc = mf0 + cur * NB;
            double* mdn = md0 + nxt * NB;
            float* mfn = mf0 + nxt * NB;
            const float w = sh.w[t];
            // costs in mfc are relative to the bound of the step before
            if (u > 0) off += (double)__uint_as_float(sh.smin[u % 3]) * (1.0 - 2.4e-7);
            if (tid == 0) sh.smin[(u + 2) % 3] = 0x7F800000u;
            const uint64_t nw = f32x2(-w, -w);
            uint32_t low_new = 0x7F800000u;
#pragma unroll
            for (int g = 0; g < G; g++) {
                const uint32_t row = (E::TB > 1 ? b_own & (E::NH - 1) : h0 + E::NG * g) << K;       // the successors of this group
                uint8_t* pp = ptr + (size_t)t * NB + (E::TB > 1 ? b_own : (uint32_t)(E::NT * g + tid) * L);
                uint32_t pk[(L + 3) / 4];
                uint64_t mf2[JC / 2];
                auto load = [&](int c) {
                    if constexpr (E::kInPlace) {
#pragma unroll
                        for (int q = 0; q < JC / 2; q++)
                            mf2[q] = f32x2(mfc[slot(row | (2 * q), rot)], mfc[slot(row | (2 * q + 1), rot)]);
                    } else {
#pragma unroll
                        for (int q = 0; q < JC / 4; q++) {
                            const uint32_t piece = (n_first + c * JC + 4 * q) ^ (row_xor(row >> K) << 2);
                            const float4 v = *reinterpret_cast<const float4*>(mfc + (row | piece));
                            mf2[2 * q] = f32x2(v.x, v.y);
                            mf2[2 * q + 1] = f32x2(v.z, v.w);
                        }
                    }
                };
                if (E::JT == JC) load(0);
#pragma unroll
                for (int i0 = 0; i0 < L; i0 += BL) {
                    uint32_t m1[BL], m2[BL];
#pragma unroll
                    for (int c = 0; c < E::JT / JC; c++) {
                        if (E::JT != JC) load(c);
#pragma unroll
                        for (int i = 0; i < BL; i++) {
                            uint32_t key[JC];
#pragma unroll
                            for (int q = 0; q < JC / 2; q++) {
                                uint32_t pair = cbr[g * L + i0 + i][c * (JC / 2) + q];
                                asm volatile("" : "+r"(pair));   // converted here: hoisted, the floats spill
                                const float2 cf = __half22float2(u32_as_h2(pair));
                                const uint64_t d = add_f32x2(f32x2(cf.x, cf.y), nw);
                                const uint64_t k2 = fma_f32x2(d, d, mf2[q]);
                                const uint32_t n = c * JC + 2 * q;
                                key[2 * q] = key_with_index<J>((uint32_t)k2, n);
                                key[2 * q + 1] = key_with_index<J>((uint32_t)(k2 >> 32), n + 1);
                            }
                            uint32_t lo = key[0];
#pragma unroll
                            for (int q = 1; q < JC; q++) lo = min(lo, key[q]);
                            // gap to the runner-up: the winner itself wraps to the largest number
                            uint32_t gap = 0xFFFFFFFFu;
#pragma unroll
                            for (int q = 0; q < JC; q++) gap = __viaddmin_u32(key[q], ~lo, gap);
                            const uint32_t up = lo + 1u + gap;
                            if (c == 0) {
                                m1[i] = lo;
                                m2[i] = up;
                            } else {
                                m2[i] = min(max(m1[i], lo), min(m2[i], up));
                                m1[i] = min(m1[i], lo);
                            }
                        }
                    }
                    // the winners' costs in float64, several bases at once; then the bases where fp32 could not decide
                    double val[BL];
                    uint32_t bn[BL], unsure = 0;
                    const double wd = (double)w;
#pragma unroll
                    for (int i = 0; i < BL; i++) {
                        uint32_t lo = m1[i], up = m2[i];
                        if constexpr (E::TB > 1) {       // the other threads' n values
                            lo |= n_first;               // (the low bits hold 0 .. JT - 1 so far)
                            up |= n_first;
#pragma unroll
                            for (int o = kLanes; o < 32; o <<= 1) {
                                const uint32_t lo2 = __shfl_xor_sync(0xFFFFFFFFu, lo, o), up2 = __shfl_xor_sync(0xFFFFFFFFu, up, o);
                                up = min(max(lo, lo2), min(up, up2));
                                lo = min(lo, lo2);
                            }
                        }
                        bn[i] = lo & (J - 1);
                        const uint32_t s = (base(g, i0 + i) << K) | bn[i];
                        val[i] = __dadd_rn(mdc[slot(row | bn[i], rot)], sq_err((double)codebook_f32<CB>(s), wd));
                        if (up - lo < kGap || up < near) unsure |= 1u << i;
                    }
                    if (unsure) {
#pragma unroll
                        for (int i = 0; i < BL; i++) {
                            if (!((unsure >> i) & 1u)) continue;
                            const uint32_t s = base(g, i0 + i) << K;
                            double second = 1e300;
                            bn[i] = 0;
                            val[i] = __dadd_rn(mdc[slot(row, rot)], sq_err((double)codebook_f32<CB>(s), wd));
#pragma unroll 4
                            for (int q = 1; q < J; q++) {
                                const double v = __dadd_rn(mdc[slot(row | (uint32_t)q, rot)], sq_err((double)codebook_f32<CB>(s | (uint32_t)q), wd));
                                // (final states with equal errors: the first of them, in whatever order the costs are summed)
                                if (v < val[i]) { second = val[i]; val[i] = v; bn[i] = q; }
                                else if (v < second && (u > 0 || v > val[i])) second = v;
                            }
                            if (second - val[i] < close && n_first == 0) note_close(sh, t, base(g, i0 + i), second - val[i]);
                        }
                    }
                    if (n_first == 0) {
#pragma unroll
                        for (int i = 0; i < BL; i++) {
                            // in place, base (i << HB) | h of the next step takes the address of (h << K) | i
                            const uint32_t ad = E::kInPlace ? slot(row | (i0 + i), rot) : base(g, i0 + i);
                            const uint32_t af = E::kInPlace ? ad : first_f + (i0 + i) * (E::T << HB) + E::NG * g;
                            const float rel = fmaxf((float)(val[i] - off), 0.f);
                            mdn[ad] = val[i];
                            mfn[af] = rel;
                            low_new = min(low_new, __float_as_uint(rel));
                            const int q = i0 + i;
                            pk[q >> 2] = (q & 3) ? pk[q >> 2] | (bn[i] << (8 * (q & 3))) : bn[i];
                        }
                    }
                }
                if (n_first == 0) {
                    if constexpr (L == 8) __stcg(reinterpret_cast<uint2*>(pp), make_uint2(pk[0], pk[1]));
                    else if constexpr (L == 4) __stcg(reinterpret_cast<uint32_t*>(pp), pk[0]);
                    else if constexpr (L == 2) __stcg(reinterpret_cast<uint16_t*>(pp), (uint16_t)pk[0]);
                    else __stcg(pp, (uint8_t)pk[0]);
                }
            }
            low_new = __reduce_min_sync(0xFFFFFFFFu, low_new);
            if ((tid & 31) == 0) atomicMin(&sh.smin[(u + 1) % 3], low_new);
            __syncthreads();
            if constexpr (E::kLook < 256)
                if (u % E::kLook == E::kLook - 1 && (left = too_close(sh))) break;
        }
        constexpr int end_rot = E::kInPlace ? (K * 256) % LB : 0;
        if (!left && search_paths<K, CB>(sh, smem, ptr, a.max_pins, bound, [&](uint32_t b) { return md0[slot(b, end_rot)]; })) store_tile<K>(sh, a, tile);
        else if (tid == 0) leave_tile(a, tile, kEncDoubt);
    }
}

// ---- the search from the start, in the reference's order: tiles that search_kernel leaves ----------------------
//   m_t+1[b'] = min_j ( m_t[(b' >> K) | (j << (16-2K))] + (codebook(b' | j << (16-K)) - w_t)^2 )
// with the same arithmetic; float64 costs are what the reference computes, to the bit.  The walk over the back-pointers reads
// two steps per L2 round trip: while the warp fetches step t's pointer its lanes fetch step t - 1's for every value
// that pointer can have.

// How the 65,536 (b', j) pairs of a step are dealt to the threads.
template <int K> struct EncodeSplit {
    static constexpr int NB = kEncStates >> K;           // bases
    static constexpr int J = 1 << K;
    static constexpr int JT = J < 128 ? J : 128;         // j values per thread and base (K = 8: two threads a base)
    static constexpr int BPT = 128 / JT;                 // bases per thread
    static constexpr int L = BPT < J ? BPT : J;          // ... of them in one group (same b' >> K)
    static constexpr int G = BPT / L;                    // groups per thread
    static constexpr int JC = JT < 16 ? JT : 16;         // j values per turn
    static constexpr bool kInPlace = K == 2;
    static constexpr size_t kSmem = (size_t)NB * (kInPlace ? 1 : 2) * (sizeof(double) + sizeof(float));
};

template <int K, int CB>
__global__ void __launch_bounds__(kEncThreads, 1) encode_kernel(const EncodeArgs a)
{
    using E = EncodeSplit<K>;
    constexpr int NB = E::NB, J = E::J, L = E::L, G = E::G, JC = E::JC, LB = 16 - K;
    // Two fp32 keys whose bit patterns differ by less than this may be in the wrong order: the low K
    // bits hold j (2^K units), the arithmetic before is off by at most four units on either side; twice
    // that, rounded up.
    constexpr uint32_t kGap = 4u * J + 32u;
    extern __shared__ __align__(16) uint8_t smem[];
    __shared__ EncodeShared sh;
    double* md0 = reinterpret_cast<double*>(smem);
    float* mf0 = reinterpret_cast<float*>(md0 + (E::kInPlace ? 1 : 2) * NB);
    const int tid = threadIdx.x;
    uint8_t* back = a.slots + (size_t)blockIdx.x * kEncSlotBytes;
    if (*a.left == 0u) return;

    // this thread's bases: groups h(g) = h0 + 512 g, bases (h << K) | (l0 + i)
    constexpr int TPG = K == 8 ? 512 : J / L;            // threads per group
    const uint32_t h0 = (uint32_t)(tid / TPG);
    const uint32_t l0 = K == 8 ? (uint32_t)(tid >> 1) : (uint32_t)(tid % TPG) * L;
    const uint32_t j_first = K == 8 ? 128u * (tid & 1) : 0u;

    uint32_t cbr[G * L][E::JT / 2];
#pragma unroll
    for (int g = 0; g < G; g++)
#pragma unroll
        for (int i = 0; i < L; i++)
#pragma unroll
            for (int q = 0; q < E::JT / 2; q++) {
                const uint32_t b = ((h0 + 512u * g) << K) | (l0 + i), j = j_first + 2 * q;
                cbr[g * L + i][q] = decode_pair<CB>(b | (j << LB), b | ((j + 1) << LB));
            }

    // Address of base b.  Its low four bits are XOR-ed with the next four, so that a warp's stores (a
    // few consecutive bases per thread) fall into different banks.  In place, b is first rotated by
    // the bits of the steps taken so far and the XOR takes all its nibbles, because sixteen neighbours
    // are then at any power-of-two stride.
    auto slot = [&](uint32_t b, int rot) -> uint32_t {
        if (E::kInPlace) {
            b = ((b >> rot) | (b << (LB - rot))) & (NB - 1);
            return b ^ (((b >> 4) ^ (b >> 8) ^ (b >> 12)) & 15u);
        }
        return b ^ ((b >> 4) & 15u);
    };
    // ... of the j-th predecessor base of group h (hs = slot(h)): the high bits pass through the XOR
    // unless they are among the eight low ones
    auto pred_slot = [&](uint32_t h, uint32_t hs, uint32_t j, int rot) -> uint32_t {
        if (!E::kInPlace && LB - K >= 8) return hs + (j << (LB - K));
        return slot(h | (j << (LB - K)), rot);
    };
    for (;;) {
        const int64_t tile = next_tile<kEncDoubt>(sh, a);
        if (tile >= a.n_tiles) return;
        for (int pass = 0; pass <= a.max_pins; pass++) {
            const int pin = sh.pin;
            for (int b = tid; b < NB; b += kEncThreads) {
                const bool home = pin >= 0 && b == (pin & (NB - 1));
                const double m = pin < 0 || home ? 0.0 : 1e30;
                const uint32_t at = slot((uint32_t)b, 0);
                md0[at] = m;
                mf0[at] = (float)m;
                __stcg(back + b, (uint8_t)(home ? pin >> LB : 0));
            }
            if (tid == 0) sh.smin[1] = 0x7F800000u;
            __syncthreads();
            double off = 0.0;                            // lower bound of every m_t[b]
            for (int t = 0; t < 255; t++) {
                const int cur = E::kInPlace ? 0 : (t & 1), nxt = E::kInPlace ? 0 : cur ^ 1;
                const int rot = E::kInPlace ? (K * t) % LB : 0;
                const double* mdc = md0 + cur * NB;
                const float* mfc = mf0 + cur * NB;
                double* mdn = md0 + nxt * NB;
                float* mfn = mf0 + nxt * NB;
                const float w = sh.w[t];
                const bool tame = fabsf(w) < 1e6f;
                // costs in mfc are relative to the bound of the step before
                const float near = (float)off * 9.3e-10f;   // 2^-30: closer than this, float64 roundings decide
                if (t > 0) {
                    const float low = __uint_as_float(sh.smin[t % 3]);
                    if (low < 1e29f) off += (double)low * (1.0 - 2.4e-7);
                }
                if (tid == 0) sh.smin[(t + 2) % 3] = 0x7F800000u;
                const uint64_t nw = f32x2(-w, -w);
                uint32_t low_new = 0x7F800000u;
#pragma unroll
                for (int g = 0; g < G; g++) {
                    const uint32_t h = h0 + 512u * g, hs = slot(h, 0);
                    uint32_t m1[L], m2[L];
#pragma unroll
                    for (int c = 0; c < E::JT / JC; c++) {
                        uint64_t mf2[JC / 2];
#pragma unroll
                        for (int q = 0; q < JC / 2; q++) {
                            const uint32_t j = j_first + c * JC + 2 * q;
                            mf2[q] = f32x2(mfc[pred_slot(h, hs, j, rot)], mfc[pred_slot(h, hs, j + 1, rot)]);
                        }
#pragma unroll
                        for (int i = 0; i < L; i++) {
                            uint32_t key[JC];
#pragma unroll
                            for (int q = 0; q < JC / 2; q++) {
                                uint32_t pair = cbr[g * L + i][c * (JC / 2) + q];
                                asm volatile("" : "+r"(pair));   // converted here: hoisted, 128 floats spill
                                const float2 cf = __half22float2(u32_as_h2(pair));
                                const uint64_t d = add_f32x2(f32x2(cf.x, cf.y), nw);
                                const uint64_t k2 = fma_f32x2(d, d, mf2[q]);
                                const uint32_t j = c * JC + 2 * q;
                                key[2 * q] = key_with_index<J>((uint32_t)k2, j);
                                key[2 * q + 1] = key_with_index<J>((uint32_t)(k2 >> 32), j + 1);
                            }
                            uint32_t lo = key[0];
#pragma unroll
                            for (int q = 1; q < JC; q++) lo = min(lo, key[q]);
                            // gap to the runner-up: the winner itself wraps to the largest number
                            uint32_t gap = 0xFFFFFFFFu;
#pragma unroll
                            for (int q = 0; q < JC; q++) gap = __viaddmin_u32(key[q], ~lo, gap);
                            const uint32_t up = lo + 1u + gap;
                            if (c == 0) {
                                m1[i] = lo;
                                m2[i] = up;
                            } else {
                                m2[i] = min(max(m1[i], lo), min(m2[i], up));
                                m1[i] = min(m1[i], lo);
                            }
                        }
                    }
                    // the winners' costs in float64, all bases at once; then the bases where fp32 could not decide
                    double val[L];
                    uint32_t bj[L], unsure = 0;
                    const double wd = (double)w;
#pragma unroll
                    for (int i = 0; i < L; i++) {
                        uint32_t lo = m1[i], up = m2[i];
                        if (K == 8) {                    // the other half of the j values
                            lo |= j_first;               // (the low bits hold 0 .. 127 so far)
                            up |= j_first;
                            const uint32_t lo2 = __shfl_xor_sync(0xFFFFFFFFu, lo, 1), up2 = __shfl_xor_sync(0xFFFFFFFFu, up, 1);
                            up = min(max(lo, lo2), min(up, up2));
                            lo = min(lo, lo2);
                        }
                        bj[i] = lo & (J - 1);
                        const uint32_t s = ((h << K) | (l0 + i)) | (bj[i] << LB);
                        val[i] = __dadd_rn(mdc[pred_slot(h, hs, bj[i], rot)], sq_err((double)codebook_f32<CB>(s), wd));
                        if (up - lo < kGap || __uint_as_float(up) < near) unsure |= 1u << i;
                    }
                    if (unsure) {
#pragma unroll
                        for (int i = 0; i < L; i++) {
                            if (!((unsure >> i) & 1u)) continue;
                            const uint32_t b = (h << K) | (l0 + i);
                            bj[i] = 0;
                            if (val[i] >= 9e29 && tame) {   // not reachable from the pinned state yet: all exactly 1e30
                                val[i] = 1e30;
                                continue;
                            }
                            val[i] = __dadd_rn(mdc[pred_slot(h, hs, 0, rot)], sq_err((double)codebook_f32<CB>(b), wd));
#pragma unroll 1
                            for (int q = 1; q < J; q++) {
                                const uint32_t sq = b | ((uint32_t)q << LB);
                                const double v = __dadd_rn(mdc[pred_slot(h, hs, (uint32_t)q, rot)], sq_err((double)codebook_f32<CB>(sq), wd));
                                if (v < val[i]) { val[i] = v; bj[i] = q; }
                            }
                        }
                    }
                    if (K != 8 || (tid & 1) == 0) {
#pragma unroll
                        for (int i = 0; i < L; i++) {
                            const uint32_t b = (h << K) | (l0 + i);
                            // in place, base b' = (h << K) | l of the next step takes the address of h | l << (LB - K)
                            const uint32_t at = E::kInPlace ? slot(h | (i << (LB - K)), rot) : slot(b, 0);
                            const float rel = fmaxf((float)(val[i] - off), 0.f);
                            mdn[at] = val[i];
                            mfn[at] = rel;
                            low_new = min(low_new, __float_as_uint(rel));
                        }
                        uint8_t* bp = back + (size_t)(t + 1) * NB + ((h << K) | l0);
                        uint32_t pk[(L + 3) / 4];
#pragma unroll
                        for (int i = 0; i < (L + 3) / 4; i++) pk[i] = 0u;
#pragma unroll
                        for (int i = 0; i < L; i++) pk[i >> 2] |= bj[i] << (8 * (i & 3));
                        if constexpr (L == 8) __stcg(reinterpret_cast<uint2*>(bp), make_uint2(pk[0], pk[1]));
                        else if constexpr (L == 4) __stcg(reinterpret_cast<uint32_t*>(bp), pk[0]);
                        else if constexpr (L == 2) __stcg(reinterpret_cast<uint16_t*>(bp), (uint16_t)pk[0]);
                        else __stcg(bp, (uint8_t)pk[0]);
                    }
                }
                low_new = __reduce_min_sync(0xFFFFFFFFu, low_new);
                if ((tid & 31) == 0) atomicMin(&sh.smin[(t + 1) % 3], low_new);
                __syncthreads();
            }
            // step 255: every final state in float64
            {
                const int cur = E::kInPlace ? 0 : 1, rot = E::kInPlace ? (K * 255) % LB : 0;
                const double* mdc = md0 + cur * NB;
                const double wd = (double)sh.w[255];
                double bc = 0.0;
                int bs = -1;
#pragma unroll 4
                for (int s = tid; s < kEncStates; s += kEncThreads) {
                    const double v = __dadd_rn(mdc[slot((uint32_t)s >> K, rot)], sq_err((double)codebook_f32<CB>((uint32_t)s), wd));
                    if (bs < 0 || v < bc) { bc = v; bs = s; }
                }
                final_state(sh, bc, bs, kEncThreads / 32);
            }
            if (tid < 32) walk_back<K>(sh, back, pass);
            __syncthreads();
            if (sh.done) break;
        }
        store_tile<K>(sh, a, tile);
    }
}

// The tiles that encode_kernel leaves (K >= 2), with weights that are no numbers or beyond kEncLargest: in float64
// throughout, the costs in the slot (L2).  Not worth more: such a tile has no good path, only a defined one.  In
// encode_kernel, carrying NaN and telling such costs from the 1e30 took 1 % (K = 4) to 3 % (K = 6) from every tile; as a
// launch behind it, looking all tiles through takes 5 us of 9 ms.
template <int K, int CB> __global__ void __launch_bounds__(kEncThreads, 1) encode_odd_kernel(const EncodeArgs a)
{
    constexpr int NB = kEncStates >> K, J = 1 << K, LB = 16 - K;
    __shared__ EncodeShared sh;
    const int tid = threadIdx.x;
    uint8_t* back = a.slots + (size_t)blockIdx.x * kEncSlotBytes;
    double* cost0 = reinterpret_cast<double*>(back + kEncBackBytes);
    double* cost1 = cost0 + NB;
    if (*a.left == 0u) return;
    for (;;) {
        const int64_t tile = next_tile<kEncOdd>(sh, a);
        if (tile >= a.n_tiles) return;
        for (int pass = 0; pass <= a.max_pins; pass++) {
            const int pin = sh.pin;
            for (int b = tid; b < NB; b += kEncThreads) {
                const bool home = pin >= 0 && b == (pin & (NB - 1));
                __stcg(cost0 + b, pin < 0 || home ? 0.0 : 1e30);
                __stcg(back + b, (uint8_t)(home ? pin >> LB : 0));
            }
            __syncthreads();
            double* cur = cost0;
            double* nxt = cost1;
            for (int t = 0; t < 255; t++) {
                const double wd = (double)sh.w[t];
                for (int b = tid; b < NB; b += kEncThreads) {
                    double best = 0.0;
                    int bj = 0;
#pragma unroll 1
                    for (int j = 0; j < J; j++) {
                        const double v = __dadd_rn(__ldcg(cur + ((b >> K) | (j << (LB - K)))),
                                                   sq_err((double)codebook_f32<CB>((uint32_t)(b | (j << LB))), wd));
                        if (j == 0 || v < best) { best = v; bj = j; }
                    }
                    __stcg(nxt + b, best);
                    __stcg(back + (size_t)(t + 1) * NB + b, (uint8_t)bj);
                }
                __syncthreads();
                double* tmp = cur; cur = nxt; nxt = tmp;
            }
            const double wd = (double)sh.w[255];
            double bc = 0.0;
            int bs = -1;
            for (int s = tid; s < kEncStates; s += kEncThreads) {
                const double v = __dadd_rn(__ldcg(cur + (s >> K)), sq_err((double)codebook_f32<CB>((uint32_t)s), wd));
                if (bs < 0 || v < bc) { bc = v; bs = s; }
            }
            final_state(sh, bc, bs, kEncThreads / 32);
            if (tid < 32) walk_back<K>(sh, back, pass);
            __syncthreads();
            if (sh.done) break;
        }
        store_tile<K>(sh, a, tile);
    }
}

// K = 1: 32,768 bases of two predecessors; the costs stay in L2.
constexpr int kEncThreads1 = 1024;
template <int CB> __global__ void __launch_bounds__(kEncThreads1) encode_kernel_k1(const EncodeArgs a)
{
    constexpr int NB = kEncStates / 2;
    __shared__ EncodeShared sh;
    const int tid = threadIdx.x;
    uint8_t* back = a.slots + (size_t)blockIdx.x * kEncSlotBytes;
    double* cost0 = reinterpret_cast<double*>(back + kEncBackBytes);
    double* cost1 = cost0 + NB;
    if (*a.left == 0u) return;
    for (;;) {
        const int64_t tile = next_tile<kEncDoubt>(sh, a);
        if (tile >= a.n_tiles) return;
        for (int pass = 0; pass <= a.max_pins; pass++) {
            const int pin = sh.pin;
            for (int b = tid; b < NB; b += kEncThreads1) {
                const bool home = pin >= 0 && b == (pin & (NB - 1));
                __stcg(cost0 + b, pin < 0 || home ? 0.0 : 1e30);
                __stcg(back + b, (uint8_t)(home ? pin >> 15 : 0));
            }
            __syncthreads();
            double* cur = cost0;
            double* nxt = cost1;
            for (int t = 0; t < 255; t++) {
                const double wd = (double)sh.w[t];
                uint8_t* bp = back + (size_t)(t + 1) * NB;
                // bases 2h and 2h + 1 share the predecessor bases h and h + 2^14
#pragma unroll 4
                for (int h = tid; h < NB / 2; h += kEncThreads1) {
                    const double c0 = __ldcg(cur + h), c1 = __ldcg(cur + h + NB / 2);
                    double m[2];
                    uint32_t bj = 0;
#pragma unroll
                    for (int l = 0; l < 2; l++) {
                        const uint32_t b = 2 * h + l;
                        const double v0 = __dadd_rn(c0, sq_err((double)codebook_f32<CB>(b), wd));
                        const double v1 = __dadd_rn(c1, sq_err((double)codebook_f32<CB>(b | 0x8000u), wd));
                        m[l] = v1 < v0 ? v1 : v0;
                        if (v1 < v0) bj |= 1u << (8 * l);
                    }
                    __stcg(reinterpret_cast<double2*>(nxt + 2 * h), make_double2(m[0], m[1]));
                    __stcg(reinterpret_cast<uint16_t*>(bp + 2 * h), (uint16_t)bj);
                }
                __syncthreads();
                double* tmp = cur; cur = nxt; nxt = tmp;
            }
            const double wd = (double)sh.w[255];
            double bc = 0.0;
            int bs = -1;
#pragma unroll 4
            for (int s = tid; s < kEncStates; s += kEncThreads1) {
                const double v = __dadd_rn(__ldcg(cur + (s >> 1)), sq_err((double)codebook_f32<CB>((uint32_t)s), wd));
                if (bs < 0 || v < bc) { bc = v; bs = s; }
            }
            final_state(sh, bc, bs, kEncThreads1 / 32);
            if (tid < 32) walk_back<1>(sh, back, pass);
            __syncthreads();
            if (sh.done) break;
        }
        store_tile<1>(sh, a, tile);
    }
}

// K = 1, the backward search: bases h and h + 2^14 share the successors 2h and 2h + 1; the costs stay in L2, compared in
// float64.
template <int CB> __global__ void __launch_bounds__(kEncThreads1, 1) search_kernel_k1(const EncodeArgs a)
{
    using E = SearchSplit<1>;
    constexpr int NB = E::NB;
    extern __shared__ __align__(16) uint8_t smem[];
    __shared__ EncodeShared sh;
    const int tid = threadIdx.x;
    uint8_t* ptr = a.slots + (size_t)blockIdx.x * kEncSlotBytes;
    double* cost0 = reinterpret_cast<double*>(ptr + kEncBackBytes);
    for (;;) {
        const int64_t tile = next_tile(sh, a);
        if (tile >= a.n_tiles) return;
        for (int b = tid; b < NB; b += kEncThreads1) __stcg(cost0 + b, 0.0);
        float bound;
        if (!cost_bound(sh, 8.f, 2.f, bound)) {
            if (tid == 0) leave_tile(a, tile, kEncDoubt);
            continue;
        }
        const double close = (double)bound * 0x1p-41;
#pragma unroll 1
        for (int u = 0; u < 256; u++) {
            const int t = 255 - u;
            const double* cur = cost0 + (u & 1) * NB;
            double* nxt = cost0 + ((u & 1) ^ 1) * NB;
            const double wd = (double)sh.w[t];
            uint32_t* row = reinterpret_cast<uint32_t*>(ptr + (size_t)t * E::kRowBytes);
#pragma unroll 4
            for (int h = tid; h < NB / 2; h += kEncThreads1) {
                const double2 c = __ldcg(reinterpret_cast<const double2*>(cur) + h);
#pragma unroll
                for (int g = 0; g < 2; g++) {
                    const uint32_t b = (uint32_t)(h | (g << E::HB)), pair = decode_pair<CB>(2 * b, 2 * b + 1);
                    const double v0 = __dadd_rn(c.x, sq_err((double)__low2float(u32_as_h2(pair)), wd));
                    const double v1 = __dadd_rn(c.y, sq_err((double)__high2float(u32_as_h2(pair)), wd));
                    const double gap = fabs(v1 - v0);
                    // (final states with equal errors: the first of them, in whatever order the costs are summed)
                    if (gap < close && (u > 0 || gap > 0.0)) note_close(sh, t, b, gap);
                    __stcg(nxt + b, v1 < v0 ? v1 : v0);
                    const uint32_t bits = __ballot_sync(0xFFFFFFFFu, v1 < v0);
                    if ((tid & 31) == 0) __stcg(row + (b >> 5), bits);
                }
            }
            __syncthreads();
        }
        if (search_paths<1, CB>(sh, smem, ptr, a.max_pins, bound, [&](uint32_t b) { return __ldcg(cost0 + b); })) store_tile<1>(sh, a, tile);
        else if (tid == 0) leave_tile(a, tile, kEncDoubt);
    }
}

template <int K, int CB> static int launch_encode(const EncodeArgs& a, unsigned slots, cudaStream_t s)
{
    if constexpr (K == 1) {
        static bool attr_set[kMaxDevices] = {};
        int dev = 0;
        cudaGetDevice(&dev);
        if (dev < 0 || dev >= kMaxDevices) return EXL3_E_UNSUPPORTED;
        if (!attr_set[dev]) {
            const cudaError_t e = cudaFuncSetAttribute(search_kernel_k1<CB>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                       (int)SearchSplit<1>::kSmem);
            if (e != cudaSuccess) return note_cuda(e);
            attr_set[dev] = true;
        }
        search_kernel_k1<CB><<<slots, kEncThreads1, SearchSplit<1>::kSmem, s>>>(a);
        const int rc = check_launch();
        if (rc) return rc;
        EncodeArgs rest = a;
        rest.counter = a.counter + 1;
        encode_kernel_k1<CB><<<slots, kEncThreads1, 0, s>>>(rest);
        return check_launch();
    } else {
        static bool attr_set[kMaxDevices] = {};
        int dev = 0;
        cudaGetDevice(&dev);
        if (dev < 0 || dev >= kMaxDevices) return EXL3_E_UNSUPPORTED;
        if (!attr_set[dev]) {
            cudaError_t e = cudaFuncSetAttribute(search_kernel<K, CB>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                 (int)SearchSplit<K>::kSmem);
            if (e == cudaSuccess)
                e = cudaFuncSetAttribute(encode_kernel<K, CB>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)EncodeSplit<K>::kSmem);
            if (e != cudaSuccess) return note_cuda(e);
            attr_set[dev] = true;
        }
        search_kernel<K, CB><<<slots, SearchSplit<K>::NT, SearchSplit<K>::kSmem, s>>>(a);
        int rc = check_launch();
        if (rc) return rc;
        EncodeArgs rest = a;
        rest.counter = a.counter + 1;
        rest.left = a.left + kEncDoubt;
        encode_kernel<K, CB><<<slots, kEncThreads, EncodeSplit<K>::kSmem, s>>>(rest);
        rc = check_launch();
        if (rc) return rc;
        rest.counter = a.counter + 2;
        rest.left = a.left + kEncOdd;
        encode_odd_kernel<K, CB><<<slots, kEncThreads, 0, s>>>(rest);
        return check_launch();
    }
}

template <int K> static int launch_encode_k(const EncodeArgs& a, int cb, unsigned slots, cudaStream_t s)
{
    switch (cb) {
        case CB_3INST: return launch_encode<K, CB_3INST>(a, slots, s);
        case CB_MCG: return launch_encode<K, CB_MCG>(a, slots, s);
        default: return launch_encode<K, CB_MUL1>(a, slots, s);
    }
}

}  // namespace exl3

using namespace exl3;

extern "C" size_t exl3_encode_workspace_bytes(int64_t n_tiles)
{
    if (n_tiles < 1) n_tiles = 1;
    int64_t slots = device_sm_count();
    if (slots < 1) slots = 1;
    if (n_tiles < slots) slots = n_tiles;
    return kEncCounterBytes + (size_t)slots * kEncSlotBytes;
}

extern "C" int exl3_encode_tiles(const float* w, int64_t n_tiles, int k, int cb, int max_pins, uint16_t* states,
                                 uint16_t* packed, void* workspace, size_t workspace_bytes, exl3_stream_t stream)
{
    if (!w || !states) return EXL3_E_NULL;
    if (k < 1 || k > 8) return EXL3_E_K;
    if (cb < 0 || cb > 2) return EXL3_E_CODEBOOK;
    // the tile counter is 32 bits wide
    if (n_tiles < 0 || n_tiles > ((int64_t)1 << 32) || max_pins < 0 || max_pins > 64) return EXL3_E_RANGE;
    if ((reinterpret_cast<uintptr_t>(w) & 3) || (reinterpret_cast<uintptr_t>(states) & 1) ||
        (packed && (reinterpret_cast<uintptr_t>(packed) & 3)))
        return EXL3_E_ALIGN;
    if (!workspace || workspace_bytes < kEncCounterBytes + kEncSlotBytes) return EXL3_E_WORKSPACE;
    if (reinterpret_cast<uintptr_t>(workspace) & 255) return EXL3_E_ALIGN;
    if (n_tiles == 0) return EXL3_OK;
    int64_t slots = (int64_t)((workspace_bytes - kEncCounterBytes) / kEncSlotBytes);
    slots = std::min<int64_t>(slots, std::min<int64_t>(n_tiles, (int64_t)device_sm_count()));
    EncodeArgs a;
    a.max_pins = max_pins;
    a.counter = static_cast<unsigned*>(workspace);
    a.left = a.counter + 3;
    a.slots = static_cast<uint8_t*>(workspace) + kEncCounterBytes;
    cudaStream_t s = (cudaStream_t)stream;
    constexpr int64_t kMost = (int64_t)1 << 31;      // tiles per launch: the counter must not wrap
    for (int64_t t0 = 0; t0 < n_tiles; t0 += kMost) {
        a.w = w + t0 * 256;
        a.n_tiles = std::min<int64_t>(kMost, n_tiles - t0);
        a.states = states + t0 * 256;
        a.packed = packed ? reinterpret_cast<uint32_t*>(packed) + t0 * 8 * k : nullptr;
        int rc = note_cuda(cudaMemsetAsync(a.counter, 0, 5 * sizeof(unsigned), s));
        if (rc) return rc;
        switch (k) {
            case 1: rc = launch_encode_k<1>(a, cb, (unsigned)slots, s); break;
            case 2: rc = launch_encode_k<2>(a, cb, (unsigned)slots, s); break;
            case 3: rc = launch_encode_k<3>(a, cb, (unsigned)slots, s); break;
            case 4: rc = launch_encode_k<4>(a, cb, (unsigned)slots, s); break;
            case 5: rc = launch_encode_k<5>(a, cb, (unsigned)slots, s); break;
            case 6: rc = launch_encode_k<6>(a, cb, (unsigned)slots, s); break;
            case 7: rc = launch_encode_k<7>(a, cb, (unsigned)slots, s); break;
            default: rc = launch_encode_k<8>(a, cb, (unsigned)slots, s); break;
        }
        if (rc) return rc;
    }
    return EXL3_OK;
}
