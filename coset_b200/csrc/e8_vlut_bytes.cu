// Few-token product of a layer that keeps its weight in a decode-ready layout: y[T, N] = x[T, K] * Wq^T (+ bias).
//
// The code-domain kernels of e8_vlut.cu rebuild every weight block from two table gathers and a few dozen integer
// instructions per call (10-20 us for one token and a 4096 x 4096 weight).  Twice the reconstruction is an integer in
// [-35, 55], so a layer can hold t + 64 as one byte per weight instead, laid out once in the order in which the tensor
// cores want it.  The product then has no gather: a PRMT puts two bytes under the exponent 0x43 (bf16 128 + byte), one
// bf16x2 subtraction leaves t exactly, and mma.sync multiplies it UNSCALED with the activations; the scale is applied to
// the float32 inner products -- once per row when a scale covers whole rows, once per block otherwise (m16n8k8 then
// spans exactly one block).  Every product is exact, nothing is rounded to bf16 but the result.
//   * float32 activations are the exact sum of three bf16 terms and take three products, summed so that the error against 64 bits
//     is no larger than that of a chain of fused multiply-adds (8e-8 of the result at any K; one accumulator for all three
//     gave 2.2e-7; time for 4096 x 4096 float32, one scale per row with a clamp: 11.5 -> 12.5 us for one token, 24.8 -> 26.3 for 16);
//   * a clamp that can bind (|t| > clip 2 beta for some possible t) is a second product of the clamped signs, so the
//     clamped weights are exact too.
// Bound: 1 byte per weight (+ 4 per 8 weights of per-block scales), 2.6-3.9 us of HBM traffic for 4096 x 4096.  Measured
// there (graph replay, before -> now), one scale per row with a clamp: 14.4 -> 5.5 us for one token, 22.4 -> 9.5 for 16;
// one per block: 9.9 -> 6.9, 22.8 -> 10.3 (before the codes were read too, see below); float32 tokens with a scale per row: 15.2 -> 9.7, 118 -> 20.6.  8192 x 8192, one
// token, scale per row: 48 -> 16 us (4.2 TB/s).  What is left at 16 tokens is latency: two warps' worth of shared-memory
// round trips per unit at 16 warps per SM (staging the activations once per CTA, deeper cp.async rings with the weights in
// them and two-stage rings at higher occupancy were measured within 10 % of this form, and slower for few tokens).
// The per-block scales are applied to pairs of sums (f32x2), the same bits: 16 tokens 12.5 -> 11.9 us a call, for a third of the 320 instructions of a unit
// were multiply-adds and the issue of instructions is half of its time.
// A warp owns 16 rows and every KW-th unit of K; KW depends on K alone, so a row's sum does
// not depend on how many rows the matrix has (a row-sharded layer returns the same bits), and the partial sums are added
// in a fixed order through shared memory.
//
// Layout: [groups of 16 rows][units of 8 blocks][2][32 lanes] of 16 bytes; a lane's 32 bytes are eight words, word b =
// coordinates 2c, 2c + 1 of block b of the unit for row g | the same for row g + 8, with g = lane / 4, c = lane % 4: the A
// fragment of one m16n8k8 step, and two neighbouring words that of one m16n8k16 step.
// Behind the tiles, one 64-bit hash of the codes for every group and every residue of the unit modulo 16.
//
// The copy must never answer for codes that have changed since: the host sees neither a write through another alias of the
// codes nor one by a collective or a replayed graph.  So a warp of the product reads the codes of its units beside their
// bytes, hashes them, and where the hash is not the kept one does its units again with words made from the codes, as the
// layout kernel makes them.  The hash is a sum of the codes times odd keys modulo 2^64: one changed code always shows, other
// changes go unseen once in about 2^64.  Price (4096 x 4096, one scale per row with a clamp, 12 weights in turn): 6.1 -> 8.6 us for
// one token, 10.8 -> 12.6 for 16.  Comparing every unit with a copy of its codes cost more (11.6, 12.9), and so did hashing inside
// the loop over the units, from registers (11.0) or through cp.async (8.8, 13.0): the loop has no registers to spare, which is
// also why the second time round is a copy of it.
#include <cuda_bf16.h>

#include <math.h>

#include <type_traits>

#include "common.cuh"
#include "e8_fast2.cuh"
#include "e8_io.cuh"

using namespace coset;

namespace {

constexpr int kMaxTargets = 16;
struct Targets {  // where a result row goes: one buffer, or the result buffer of every rank (peer memory, plain stores)
    void* y[kMaxTargets];
    int n;
    int bf16;
};
__device__ __forceinline__ void store_result(const Targets& out, int64_t idx, float r) {
    for (int k = 0; k < out.n; ++k) {
        if (out.bf16) reinterpret_cast<__nv_bfloat16*>(out.y[k])[idx] = __float2bfloat16_rn(r);
        else reinterpret_cast<float*>(out.y[k])[idx] = r;
    }
}

constexpr float kMaxTwice = 55.0f;  // largest |2 x_hat| of any code
constexpr int kByteBias = 64;

// d = a b (FRESH) or d += a b
template <bool FRESH>
__device__ __forceinline__ void mma_16816(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    if (FRESH)
        asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
                     : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.0f));
    else
        asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                     : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
template <bool FRESH>
__device__ __forceinline__ void mma_1688(float (&d)[4], const uint32_t (&a)[2], uint32_t b0) {
    if (FRESH)
        asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%7,%7,%7,%7};"
                     : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(b0), "f"(0.0f));
    else
        asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};"
                     : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(b0));
}

// Bytes 0, 1 (HIGH: 2, 3) of a word as two exact bf16 integers byte - 64.
template <bool HIGH>
__device__ __forceinline__ uint32_t twice_pair(uint32_t w) {
    uint32_t r;
    asm("sub.rn.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(__byte_perm(w, 0x43434343u, HIGH ? 0x4342 : 0x4140)), "r"(0x43404340u));
    return r;
}
// The clamp in units of t: lanes with |t| > k become 0 in `t` and +-1 in the result.
__device__ __forceinline__ uint32_t clamp_signs(uint32_t& t, uint32_t k2) {
    const uint32_t a = t & 0x7fff7fffu;
    const uint32_t over = __hgt2_mask(*reinterpret_cast<const __nv_bfloat162*>(&a), *reinterpret_cast<const __nv_bfloat162*>(&k2));
    const uint32_t sign = ((t & 0x80008000u) | 0x3f803f80u) & over;
    t &= ~over;
    return sign;
}
// floor(clip / |scale|) in both halves (64 where nothing can exceed it)
__device__ __forceinline__ uint32_t clamp_limit(float clip, float scale) {
    const __nv_bfloat162 h = __float2bfloat162_rn(fminf(floorf(__fdividef(clip, fabsf(scale))), 64.0f));
    return *reinterpret_cast<const uint32_t*>(&h);
}
// 1 / v: rounded to nearest for float32 tokens, to about an ulp for bf16 ones
template <bool EXACT>
__device__ __forceinline__ float reciprocal(float v) {
    if (EXACT) return __frcp_rn(v);
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(v));
    return r;
}
// The exact three-term bf16 split of two floats, packed: out[p] = (p-th term of a, p-th term of b).
__device__ __forceinline__ void split3(float a, float b, uint32_t (&out)[3]) {
#pragma unroll
    for (int p = 0; p < 3; ++p) {
        const uint32_t ua = __float_as_uint(a), ub = __float_as_uint(b);
        out[p] = __byte_perm(ua, ub, 0x7632);  // truncation keeps 8 significand bits, the rest is exact
        const float ra = a - __uint_as_float(ua & 0xffff0000u), rb = b - __uint_as_float(ub & 0xffff0000u);
        a = p > 0 || ra == ra ? ra : 0.0f;  // an infinity stays in the first term
        b = p > 0 || rb == rb ? rb : 0.0f;
    }
}

// ---------------------------------------------------------------------------------------------
// codes -> layout, once per weight.  One warp per (group, unit).
__device__ __forceinline__ uint2 code_bytes_of(const uint2* table, uint32_t code) {
    const uint2 t0 = __ldg(table + (code & 0xffffu)), t1 = __ldg(table + (code >> 16));
    const uint32_t shift = (kByteBias - 5 * e8::kTableBias) * 0x01010101u;  // 2 x_hat + 35 -> + 64, at most 119
    return make_uint2(t0.x + 4u * t1.x + shift, t0.y + 4u * t1.y + shift);
}

struct TileWords {
    uint4 lo, hi;
};
// The eight words of this lane from the codes; the whole warp calls it.
__device__ __forceinline__ TileWords tile_words(const uint32_t* __restrict__ codes, int n_out, int kb, int64_t group, int unit, const uint2* __restrict__ table) {
    const int lane = threadIdx.x & 31, g = lane >> 2, c = lane & 3;
    uint2 b[2][2];  // [row g, g + 8][block 2c, 2c + 1]
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const int64_t row = group * 16 + g + 8 * h;
            const int blk = unit * 8 + 2 * c + q;
            const uint32_t code = row < n_out && blk < kb ? __ldg(codes + row * kb + blk) : 0u;
            b[h][q] = code_bytes_of(table, code);
        }
    uint32_t w[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        const int src = (lane & ~3) + (k >> 1);
        const uint32_t gx = __shfl_sync(0xffffffffu, b[0][k & 1].x, src), gy = __shfl_sync(0xffffffffu, b[0][k & 1].y, src);
        const uint32_t hx = __shfl_sync(0xffffffffu, b[1][k & 1].x, src), hy = __shfl_sync(0xffffffffu, b[1][k & 1].y, src);
        w[k] = __byte_perm(c < 2 ? gx : gy, c < 2 ? hx : hy, c & 1 ? 0x7632 : 0x5410);
    }
    return {make_uint4(w[0], w[1], w[2], w[3]), make_uint4(w[4], w[5], w[6], w[7])};
}
// The hash takes the codes of a group of 16 rows as the one array that they are, in parts of 128 codes (four per lane), one part
// per unit, so that the reads are coalesced.  A lane's four codes, zero beyond the array; WIDE: it is 16-byte aligned.
template <bool WIDE>
__device__ __forceinline__ uint4 group_codes(const uint32_t* __restrict__ codes, int n_out, int kb, int64_t group, int part) {
    const int64_t at = (int64_t)part * 128 + 4 * (threadIdx.x & 31);
    const int64_t rows = n_out - group * 16 < 16 ? n_out - group * 16 : 16, left = rows * kb - at;
    const uint32_t* p = codes + group * 16 * kb + at;
    if (WIDE && left >= 4) return __ldcs(reinterpret_cast<const uint4*>(p));
    return make_uint4(left > 0 ? __ldcs(p) : 0u, left > 1 ? __ldcs(p + 1) : 0u, left > 2 ? __ldcs(p + 2) : 0u, left > 3 ? __ldcs(p + 3) : 0u);
}
__device__ __forceinline__ unsigned long long hash_codes(const uint4& c, int part) {
    const unsigned long long x = (unsigned long long)((uint32_t)part * 32u + (threadIdx.x & 31)) * 0x9e3779b97f4a7c15ull;
    const unsigned long long key = ((x ^ (x >> 32)) * 0xd1b54a32d192ed03ull) | 1ull;
    return key * ((unsigned long long)c.x * 0x85ebca6bu + (unsigned long long)c.y * 0xc2b2ae35u + (unsigned long long)c.z * 0x27d4eb2fu + (unsigned long long)c.w * 0x165667b1u);
}
// Hashes are added in two halves, each modulo 2^32.
__device__ __forceinline__ void add_hash(uint2& sum, unsigned long long h) {
    sum.x += (uint32_t)h;
    sum.y += (uint32_t)(h >> 32);
}
__device__ __forceinline__ uint2 warp_sum(uint2 h) { return make_uint2(__reduce_add_sync(0xffffffffu, h.x), __reduce_add_sync(0xffffffffu, h.y)); }
constexpr int kHashClasses = 16;  // the most warps that share a row group

__global__ void __launch_bounds__(256)
k_vlut_layout(const uint32_t* __restrict__ codes, int n_out, int kb, int units, int64_t tiles, const uint2* __restrict__ table, uint4* __restrict__ out) {
    const int64_t tile = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
    if (tile >= tiles) return;
    const int lane = threadIdx.x & 31;
    const int64_t group = tile / units;
    const int unit = (int)(tile - group * units);
    const TileWords w = tile_words(codes, n_out, kb, group, unit, table);
    out[tile * 64 + lane] = w.lo;
    out[tile * 64 + 32 + lane] = w.hi;
    uint2 h = make_uint2(0u, 0u);
    add_hash(h, hash_codes(group_codes<false>(codes, n_out, kb, group, unit), unit));
    h = warp_sum(h);
    if (lane < 2) atomicAdd(reinterpret_cast<uint32_t*>(out + tiles * 64) + 2 * (group * kHashClasses + unit % kHashClasses) + lane, lane ? h.y : h.x);
}

// ---------------------------------------------------------------------------------------------
struct Product {
    const uint4* w;
    const uint2* hash;
    const uint32_t* codes;  // null: the caller vouches for the layout
    int wide_codes;
    const uint2* table;
    const float* beta;
    int per_row;          // one scale covers whole rows: rows_per_scale of them
    int rows_per_scale;
    e8::TileDiv td;       // blocks kernel: block index -> scale
    int n_out, kb, units, T;
    const void* x;
    int64_t ldx, ldy;
    const float* bias;
    float clip;
    int kw_log2;
    Targets out;
};

// Whether this warp's parts of the codes are others than those the layout was made from.
template <bool WIDE, int BATCH>
__device__ __forceinline__ bool codes_changed(const Product& a, int64_t group, int first, int kw) {
    uint2 sum = make_uint2(0u, 0u);
    if ((threadIdx.x & 31) == 0)
        for (int k = first; k < kHashClasses; k += kw) {
            const uint2 h = __ldg(a.hash + group * kHashClasses + k);
            sum.x -= h.x;
            sum.y -= h.y;
        }
    for (int u = first; u < a.units; u += BATCH * kw) {
        uint4 c[BATCH];
#pragma unroll
        for (int k = 0; k < BATCH; ++k) c[k] = u + k * kw < a.units ? group_codes<WIDE>(a.codes, a.n_out, a.kb, group, u + k * kw) : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
        for (int k = 0; k < BATCH; ++k) add_hash(sum, hash_codes(c[k], u + k * kw));
    }
    sum = warp_sum(sum);
    return (sum.x | sum.y) != 0u;
}

// One result from weights that are scaled and clamped first, by a whole warp.  The kernel multiplies unscaled, so its sums can
// overflow where the product does not, and it takes a clamp apart into two products, which turns an infinite activation or a
// scale of zero into 0 * inf: a result that is not finite is taken from here instead.
template <int P>
__device__ __noinline__ float scaled_product(const Product& a, int row, int t) {
    const int lane = threadIdx.x & 31, r = row & 15;
    const uint8_t* tile = reinterpret_cast<const uint8_t*>(a.w) + (int64_t)(row >> 4) * a.units * 1024 + (r & 7) * 64 + (r >> 3) * 2;
    float sum = 0.0f;
    for (int first = 0; first < a.kb; first += 32) {
        const int blk = first + lane;
        if (blk < a.kb) {
            const int64_t at = (int64_t)row * a.kb + blk;
            uint32_t bytes[4];  // coordinates 2 c, 2 c + 1
            if (a.codes) {
                const uint2 b = code_bytes_of(a.table, __ldg(a.codes + at));
                bytes[0] = b.x; bytes[1] = b.x >> 16; bytes[2] = b.y; bytes[3] = b.y >> 16;
            } else {
#pragma unroll
                for (int c = 0; c < 4; ++c)
                    bytes[c] = __ldg(reinterpret_cast<const uint16_t*>(tile + (int64_t)(blk >> 3) * 1024 + ((blk >> 2) & 1) * 512 + c * 16 + (blk & 3) * 4));
            }
            const float scale = a.beta ? __ldg(a.beta + (a.per_row ? row / a.rows_per_scale : e8::tile_of(a.td, at))) : 1.0f;
            const char* x = reinterpret_cast<const char*>(a.x) + ((int64_t)t * a.ldx + blk * 8) * (P == 1 ? 2 : 4);
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                float w = __fdiv_rn(0.5f * (float)((int)((bytes[i >> 1] >> (8 * (i & 1))) & 0xffu) - kByteBias), scale);
                if (a.clip > 0.0f) w = fminf(fmaxf(w, -a.clip), a.clip);
                sum = __fmaf_rn(w, P == 1 ? __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(x)[i]) : reinterpret_cast<const float*>(x)[i], sum);
            }
        }
        if (__any_sync(0xffffffffu, sum != sum)) return NAN;  // and nothing makes it a number again
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    return sum;
}

// Adds the KW partial tiles of every row group of this CTA in a fixed order and stores the results.
template <int NT, int P, int WARPS>
__device__ __forceinline__ void reduce_and_store(const float (*part)[16][8 * NT + 1], const Product& a, int t0) {
    const int rw = WARPS >> a.kw_log2, kw = 1 << a.kw_log2;
    for (int e = threadIdx.x; e < rw * 16 * 8 * NT; e += WARPS * 32) {  // the bound is a multiple of 32: whole warps
        const int r = e & 15, t = (e >> 4) & (8 * NT - 1), group = (e >> 4) / (8 * NT);  // consecutive threads: consecutive rows of one token
        const int row = (blockIdx.x * rw + group) * 16 + r;
        const bool mine = row < a.n_out && t0 + t < a.T;
        float v = part[group << a.kw_log2][r][t];
        for (int w = 1; w < kw; ++w) v += part[(group << a.kw_log2) + w][r][t];
        for (uint32_t todo = __ballot_sync(0xffffffffu, mine && !(fabsf(v) < INFINITY)); todo; todo &= todo - 1) {  // rare
            const int src = __ffs(todo) - 1;
            const float again = scaled_product<P>(a, __shfl_sync(0xffffffffu, row, src), __shfl_sync(0xffffffffu, t0 + t, src));
            if ((int)(threadIdx.x & 31) == src) v = again;
        }
        if (mine) store_result(a.out, (int64_t)(t0 + t) * a.ldy + row, v + (a.bias ? __ldg(a.bias + row) : 0.0f));
    }
}

// How a weight is scaled: once per row; once per block with the scales of a row in order (rows of whole units, read as
// vectors); once per block through the tile index.
constexpr int kPerRow = 0, kPerBlock = 1, kPerTile = 2;

// Shared memory of one warp: activations of a unit as bf16 [buffer][plane][token][8 blocks of 16 bytes], the block index
// exclusive-ored with the token so that the eight rows of an ldmatrix fall into different banks, and the scales of a unit
// [4 blocks][16 rows][4].
template <int NT, int P, int SCALE>
struct WarpSmem {
    static constexpr int kBuffers = P == 1 ? 2 : 1, kPlane = 8 * NT * 128;
    uint8_t x[kBuffers * P * kPlane];
    float scale[SCALE == kPerRow ? 4 : 128];
};

__device__ __forceinline__ void copy16_async(uint32_t dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
// Four 8 x 8 b16 matrices; lane l gives the address of row l % 8 of matrix l / 8.
__device__ __forceinline__ void load_matrices(uint32_t addr, uint32_t (&r)[4]) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}

// CTAs per SM of bf16 tokens: what the loop over the layout needs; the loop over the codes spills instead.
template <int NT, int P, int WARPS>
constexpr int kProductCtas = P == 3 ? (NT == 1 ? 2 : 1) : (WARPS == 16 ? 2 : (NT == 1 ? 4 : 2));

template <int NT, int P, bool CLIP, int SCALE, int WARPS>
__global__ void __launch_bounds__(WARPS * 32, kProductCtas<NT, P, WARPS>)
k_product(const __grid_constant__ Product a) {
    typedef WarpSmem<NT, P, SCALE> Smem;
    extern __shared__ __align__(128) uint8_t smem[];
    grid_wait();
    grid_trigger();
    const int thread = behind_wait((int)threadIdx.x), warp = thread >> 5, lane = thread & 31, g = lane >> 2, c = lane & 3;
    Smem& mem = reinterpret_cast<Smem*>(smem)[warp];
    float(*part)[16][8 * NT + 1] = reinterpret_cast<float(*)[16][8 * NT + 1]>(smem + WARPS * sizeof(Smem));
    const int kw = 1 << a.kw_log2, rw = WARPS >> a.kw_log2, first = warp & (kw - 1), t0 = blockIdx.y * (8 * NT);
    const int group = blockIdx.x * rw + (warp >> a.kw_log2);
    const int tokens = a.T - t0 < 8 * NT ? a.T - t0 : 8 * NT;
    float acc[NT][4], sign_acc[NT][4], lost[NT][4];  // lost: what rounding took from acc, float32 tokens only
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[n][i] = sign_acc[n][i] = lost[n][i] = 0.0f;
    float row_scale[2] = {0.5f, 0.5f};
    bool changed = false;
    // This warp's units; DECODE: with words from the codes instead of the layout.
    auto run_units = [&](auto from_codes) {
        constexpr bool DECODE = decltype(from_codes)::value;
        const uint4* wp = a.w + ((int64_t)group * a.units + first) * 64 + lane;
        uint4 next[2];
        if (!DECODE && first < a.units) { next[0] = __ldcs(wp); next[1] = __ldcs(wp + 32); }

        // Activations of unit u.  bf16: asynchronous 16-byte copies, eight lanes per token; float32: through registers (8
        // floats per lane and step), split into three planes.  Tokens beyond T are not written (their columns of the result
        // are not stored), blocks beyond K are zero.
        constexpr int STEPS = 2 * NT;  // four tokens per step
        float4 held[STEPS][2];  // unused for bf16
        const uint32_t x_base = (uint32_t)__cvta_generic_to_shared(mem.x);
        const int st = lane >> 3, sb = lane & 7;  // token of the step, block of the unit
        const uint8_t* xp = reinterpret_cast<const uint8_t*>(a.x) + ((int64_t)(t0 + st) * a.ldx + (int64_t)first * 64 + sb * 8) * (P == 1 ? 2 : 4);
        auto request = [&](int u, int buffer) {  // xp points at unit u
#pragma unroll
            for (int i = 0; i < STEPS; ++i) {
                const int t = 4 * i + st;
                const uint8_t* src = xp + (int64_t)(4 * i) * a.ldx * (P == 1 ? 2 : 4);
                if constexpr (P == 1) {
                    const uint32_t off = (uint32_t)(buffer * Smem::kPlane + t * 128 + ((sb ^ (t & 7)) << 4));
                    if (t < tokens) {
                        if (u * 8 + sb < a.kb) copy16_async(x_base + off, src);
                        else *reinterpret_cast<uint4*>(mem.x + off) = make_uint4(0u, 0u, 0u, 0u);
                    }
                } else {
                    held[i][0] = held[i][1] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                    if (t < tokens && u * 8 + sb < a.kb) {
                        held[i][0] = __ldg(reinterpret_cast<const float4*>(src));
                        held[i][1] = __ldg(reinterpret_cast<const float4*>(src) + 1);
                    }
                }
            }
            if (P == 1) asm volatile("cp.async.commit_group;" ::: "memory");
            xp += (int64_t)(64 * (P == 1 ? 2 : 4)) << a.kw_log2;
        };
        // The scales of unit u: lane l holds four blocks of row l / 2.
        float4 next_scale = make_float4(1.0f, 1.0f, 1.0f, 1.0f);
        const int srow = group * 16 + (lane >> 1) < a.n_out ? group * 16 + (lane >> 1) : a.n_out - 1;
        int64_t sat = (int64_t)srow * a.kb + (int64_t)first * 8 + 4 * (lane & 1);
        auto request_scales = [&](int u) {
            if (SCALE == kPerBlock) {
                next_scale = __ldcs(reinterpret_cast<const float4*>(a.beta + sat));
            } else if (SCALE == kPerTile) {
                float v[4];
#pragma unroll
                for (int k = 0; k < 4; ++k) v[k] = u * 8 + 4 * (lane & 1) + k < a.kb ? __ldg(a.beta + e8::tile_of(a.td, sat + k)) : 1.0f;
                next_scale = make_float4(v[0], v[1], v[2], v[3]);
            }
            sat += 8 * kw;
        };

        if (first < a.units) {
            request(first, 0);
            if (SCALE != kPerRow) request_scales(first);
        }
        if (SCALE == kPerRow && a.beta) {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int row = group * 16 + g + 8 * h;
                row_scale[h] = 0.5f * reciprocal<P == 3>(__ldg(a.beta + (row < a.n_out ? row : a.n_out - 1) / a.rows_per_scale));
            }
        }
        bool bind = CLIP && SCALE == kPerRow && __any_sync(0xffffffffu, kMaxTwice * fmaxf(fabsf(row_scale[0]), fabsf(row_scale[1])) > a.clip);
        int buffer = 0;
        for (int u = first; u < a.units; u += kw) {
            if (DECODE) {
                const TileWords t = tile_words(a.codes, a.n_out, a.kb, group, u, a.table);
                next[0] = t.lo;
                next[1] = t.hi;
            }
            const uint32_t w[8] = {next[0].x, next[0].y, next[0].z, next[0].w, next[1].x, next[1].y, next[1].z, next[1].w};
            const bool more = u + kw < a.units;
            wp += 64 * kw;
            if (!DECODE && more) { next[0] = __ldcs(wp); next[1] = __ldcs(wp + 32); }
            if constexpr (P == 3) {
#pragma unroll
                for (int i = 0; i < STEPS; ++i) {
                    const int t = 4 * i + st;
                    const float4 lo = held[i][0], hi = held[i][1];
                    uint32_t q[4][3];
                    split3(lo.x, lo.y, q[0]); split3(lo.z, lo.w, q[1]); split3(hi.x, hi.y, q[2]); split3(hi.z, hi.w, q[3]);
                    if (t < tokens) {
#pragma unroll
                        for (int p = 0; p < P; ++p)
                            *reinterpret_cast<uint4*>(mem.x + p * Smem::kPlane + t * 128 + ((sb ^ (t & 7)) << 4)) = make_uint4(q[0][p], q[1][p], q[2][p], q[3][p]);
                    }
                }
            }
            if (SCALE != kPerRow) {
                const float4 r = make_float4(reciprocal<P == 3>(2.0f * next_scale.x), reciprocal<P == 3>(2.0f * next_scale.y), reciprocal<P == 3>(2.0f * next_scale.z), reciprocal<P == 3>(2.0f * next_scale.w));
                *reinterpret_cast<float4*>(mem.scale + (lane & 1) * 64 + (lane >> 1) * 4) = r;
                if (CLIP) bind = __any_sync(0xffffffffu, kMaxTwice * fmaxf(fmaxf(fabsf(r.x), fabsf(r.y)), fmaxf(fabsf(r.z), fabsf(r.w))) > a.clip);
                if (more) request_scales(u + kw);
            }
            if (more) request(u + kw, buffer ^ 1);
            if (P == 1) {
                if (more) asm volatile("cp.async.wait_group 1;" ::: "memory");
                else asm volatile("cp.async.wait_group 0;" ::: "memory");
            }
            __syncwarp();
            // float32 tokens: the products of the lower planes are summed apart and a unit's blocks before they join the others',
            // for the tensor cores truncate where they add a small term to a large one and a long chain of additions rounds more
            float d[NT][4], ds[NT][4], low[NT][4], low_s[NT][4], unit_acc[NT][4];
            float(&into)[NT][4] = P == 3 ? unit_acc : acc;
#pragma unroll
            for (int n = 0; n < NT; ++n)
#pragma unroll
                for (int i = 0; i < 4; ++i) unit_acc[n][i] = 0.0f;
#pragma unroll
            for (int half = 0; half < 2; ++half) {  // blocks 4 half .. + 3
                float scale[2][4];
                if (SCALE != kPerRow) {
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const float4 v = *reinterpret_cast<const float4*>(mem.scale + half * 64 + (g + 8 * h) * 4);
                        scale[h][0] = v.x; scale[h][1] = v.y; scale[h][2] = v.z; scale[h][3] = v.w;
                    }
                }
                uint32_t b[NT][P][4];  // coordinates 2c, 2c + 1 of the four blocks, token 8 n + g
#pragma unroll
                for (int n = 0; n < NT; ++n)
#pragma unroll
                    for (int p = 0; p < P; ++p)
                        load_matrices(x_base + (uint32_t)((P == 1 ? buffer : p) * Smem::kPlane + (8 * n + (lane & 7)) * 128 + (((4 * half + (lane >> 3)) ^ (lane & 7)) << 4)), b[n][p]);
#pragma unroll
                for (int k = 0; k < 4; k += 2) {
                    const int b0 = 4 * half + k;
                    uint32_t t[4] = {twice_pair<false>(w[b0]), twice_pair<true>(w[b0]), twice_pair<false>(w[b0 + 1]), twice_pair<true>(w[b0 + 1])};
                    uint32_t sign[4];
                    if (CLIP && bind) {
#pragma unroll
                        for (int i = 0; i < 4; ++i)
                            sign[i] = clamp_signs(t[i], clamp_limit(a.clip, SCALE == kPerRow ? row_scale[i & 1] : scale[i & 1][k + (i >> 1)]));
                    }
#pragma unroll
                    for (int n = 0; n < NT; ++n) {
                        if (SCALE == kPerRow) {
#pragma unroll
                            for (int p = 0; p < P; ++p) {
                                float(&dp)[4] = p == 0 ? d[n] : low[n];
                                float(&dsp)[4] = p == 0 ? ds[n] : low_s[n];
                                if (b0 == 0 && p < 2) mma_16816<true>(dp, t, b[n][p][k], b[n][p][k + 1]);
                                else mma_16816<false>(dp, t, b[n][p][k], b[n][p][k + 1]);
                                if (CLIP && bind) {
                                    if (b0 == 0 && p < 2) mma_16816<true>(dsp, sign, b[n][p][k], b[n][p][k + 1]);
                                    else mma_16816<false>(dsp, sign, b[n][p][k], b[n][p][k + 1]);
                                }
                            }
                        } else {
#pragma unroll
                            for (int q = 0; q < 2; ++q) {
                                const uint32_t tq[2] = {t[2 * q], t[2 * q + 1]};
                                mma_1688<true>(d[n], tq, b[n][0][k + q]);
                                if constexpr (P == 3) {
                                    mma_1688<true>(low[n], tq, b[n][1][k + q]);
                                    mma_1688<false>(low[n], tq, b[n][2][k + q]);
#pragma unroll
                                    for (int i = 0; i < 4; ++i) d[n][i] += low[n][i];
                                }
#pragma unroll
                                for (int h = 0; h < 2; ++h) {  // in pairs: the two tokens of a row share its scale
                                    const float f = scale[h][k + q];
                                    e8::split2(e8::fma2(e8::pair2(d[n][2 * h], d[n][2 * h + 1]), e8::pair2(f, f), e8::pair2(into[n][2 * h], into[n][2 * h + 1])),
                                               into[n][2 * h], into[n][2 * h + 1]);
                                }
                                if (CLIP && bind) {
                                    const uint32_t sq[2] = {sign[2 * q], sign[2 * q + 1]};
                                    mma_1688<true>(ds[n], sq, b[n][0][k + q]);
                                    if constexpr (P == 3) {
                                        mma_1688<true>(low_s[n], sq, b[n][1][k + q]);
                                        mma_1688<false>(low_s[n], sq, b[n][2][k + q]);
#pragma unroll
                                        for (int i = 0; i < 4; ++i) ds[n][i] += low_s[n][i];
                                    }
#pragma unroll
                                    for (int i = 0; i < 4; ++i) into[n][i] = __fmaf_rn(ds[n][i], copysignf(a.clip, scale[i >> 1][k + q]), into[n][i]);
                                }
                            }
                        }
                    }
                }
            }
            if (SCALE == kPerRow) {
                // float32 additions between units: at most four chained tensor-core accumulations per term
#pragma unroll
                for (int n = 0; n < NT; ++n)
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        if (P == 3) add_exactly(acc[n][i], lost[n][i], d[n][i] + low[n][i]);
                        else acc[n][i] += d[n][i];
                        if (CLIP && bind) sign_acc[n][i] += P == 3 ? ds[n][i] + low_s[n][i] : ds[n][i];
                    }
            } else if (P == 3) {
#pragma unroll
                for (int n = 0; n < NT; ++n)
#pragma unroll
                    for (int i = 0; i < 4; ++i) add_exactly(acc[n][i], lost[n][i], unit_acc[n][i]);
            }
            __syncwarp();  // the next unit overwrites what this one read
            buffer ^= 1;
        }
    };
    if (group * 16 < a.n_out) {
        if (a.codes) changed = a.wide_codes ? codes_changed<true, NT == 1 ? 4 : 8>(a, group, first, kw) : codes_changed<false, NT == 1 ? 4 : 8>(a, group, first, kw);
        run_units(std::false_type());
    }
    // accumulator layout: [0], [1] = (row g, tokens 2c, 2c + 1); [2], [3] = (row g + 8, same tokens)
    auto put_part = [&]() {
#pragma unroll
        for (int n = 0; n < NT; ++n)
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                float v = acc[n][i];
                if (P == 3 && lost[n][i] == lost[n][i]) v += lost[n][i];
                if (SCALE == kPerRow) {
                    v *= row_scale[i >> 1];
                    if (CLIP) v = __fmaf_rn(sign_acc[n][i], copysignf(a.clip, row_scale[i >> 1]), v);
                }
                part[warp][g + 8 * (i >> 1)][8 * n + 2 * c + (i & 1)] = v;
                acc[n][i] = sign_acc[n][i] = lost[n][i] = 0.0f;
            }
    };
    put_part();
    if (__syncthreads_or(changed)) {
        if (group * 16 < a.n_out) run_units(std::true_type());
        put_part();
        __syncthreads();
    }
    reduce_and_store<NT, P, WARPS>(part, a, t0);
}

// Whether one scale covers whole rows.
bool scale_per_row(const float* beta, int64_t blocks_per_tile, int kb) { return !beta || kb == 0 || blocks_per_tile % kb == 0; }

template <int NT, int P, bool CLIP, int SCALE, int WARPS>
int launch_as(const Product& a, cudaStream_t st) {
    const int groups = (a.n_out + 15) / 16, rw = WARPS >> a.kw_log2;
    const dim3 grid((groups + rw - 1) / rw, (a.T + 8 * NT - 1) / (8 * NT));
    if (grid.y > 65535) return fail(COSET_E_UNSUPPORTED, "T too large for the few-token product");
    constexpr int smem = WARPS * (int)(sizeof(WarpSmem<NT, P, SCALE>) + 16 * (8 * NT + 1) * sizeof(float));
    if (smem > 48 * 1024)
        if (int e = check_cuda(cudaFuncSetAttribute(k_product<NT, P, CLIP, SCALE, WARPS>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem), "cudaFuncSetAttribute")) return e;
    return launch_dependent("e8_vlut_product", k_product<NT, P, CLIP, SCALE, WARPS>, grid, WARPS * 32, smem, st, a);
}

template <int NT, int P, bool CLIP>
int launch_product(Product a, int scale, cudaStream_t st) {
    // Warps per row group, from K alone: a warp should have at least two units (its next loads overlap the arithmetic),
    // and up to 16 warps share a row group of a long K (8 where a thread needs more registers).
    constexpr int most = NT == 1 && P == 1 ? 4 : 3;
    while (a.kw_log2 < most && (4 << a.kw_log2) <= a.units) ++a.kw_log2;
#define PRODUCT_AS(SCALE)                                                                          \
    if constexpr (most == 4)                                                                       \
        if (a.kw_log2 == 4) return launch_as<NT, P, CLIP, SCALE, 16>(a, st);                       \
    return launch_as<NT, P, CLIP, SCALE, 8>(a, st)
    if (scale == kPerRow) { PRODUCT_AS(kPerRow); }
    if (scale == kPerBlock) { PRODUCT_AS(kPerBlock); }
    PRODUCT_AS(kPerTile);
#undef PRODUCT_AS
}

template <int P>
int launch_tokens(const Product& a, int scale, cudaStream_t st) {
    if (a.T > 8) return a.clip > 0.0f ? launch_product<2, P, true>(a, scale, st) : launch_product<2, P, false>(a, scale, st);
    return a.clip > 0.0f ? launch_product<1, P, true>(a, scale, st) : launch_product<1, P, false>(a, scale, st);
}

}  // namespace

extern "C" int64_t coset_e8_vlut_layout_bytes(int n_out, int n_in) {
    if (n_out < 0 || n_in < 0) return 0;
    return (((int64_t)n_out + 15) / 16) * (((int64_t)n_in + 63) / 64) * 1024 + (((int64_t)n_out + 15) / 16) * kHashClasses * 8;
}

extern "C" int coset_e8_vlut_layout(const void* codes, int n_out, int n_in, void* layout, void* stream) {
    if (n_out < 0 || n_in < 0 || (n_in % 8) != 0) return fail(COSET_E_BADARG, "bad shape (n_in must be a multiple of 8)");
    if (n_out == 0 || n_in == 0) return 0;
    if (!codes || !layout) return fail(COSET_E_BADARG, "null pointer");
    if (!aligned(codes, 4) || !aligned(layout, 16)) return fail(COSET_E_ALIGN, "codes must be 4-byte and the layout 16-byte aligned");
    cudaStream_t st = (cudaStream_t)stream;
    const uint2* table = residual_table_q4(st);
    if (!table) return COSET_E_STATE;
    const int kb = n_in / 8, units = (kb + 7) / 8;
    const int64_t tiles = (((int64_t)n_out + 15) / 16) * units;
    const unsigned grid = (unsigned)((tiles + 7) / 8);
    const int64_t groups = tiles / units;
    if (int e = check_cuda(cudaMemsetAsync((uint8_t*)layout + tiles * 1024, 0, groups * kHashClasses * 8, st), "e8_vlut_layout")) return e;
    k_vlut_layout<<<grid, 256, 0, st>>>((const uint32_t*)codes, n_out, kb, units, tiles, table, (uint4*)layout);
    return check_launch("e8_vlut_layout");
}

static int vlut_product(const void* codes, const void* layout, const float* beta, int64_t blocks_per_tile, int n_out, int n_in, const void* x, int x_dtype,
                        int64_t ldx, int T, const float* bias, void* const* y_targets, int n_targets, int y_dtype, int64_t ldy, float clip, void* stream) {
    if (n_out < 0 || n_in < 0 || T < 0 || (n_in % 8) != 0) return fail(COSET_E_BADARG, "bad shape (n_in must be a multiple of 8)");
    if (n_targets < 1 || n_targets > kMaxTargets || !y_targets) return fail(COSET_E_BADARG, "need 1..16 result buffers");
    if (n_out == 0 || T == 0) return 0;
    if (!layout || !x) return fail(COSET_E_BADARG, "null pointer");
    if ((x_dtype != COSET_DTYPE_F32 && x_dtype != COSET_DTYPE_BF16) || (y_dtype != COSET_DTYPE_F32 && y_dtype != COSET_DTYPE_BF16))
        return fail(COSET_E_BADARG, "unknown dtype");
    if (ldx < n_in || ldy < n_out) return fail(COSET_E_BADARG, "leading dimension too small");
    if (!aligned(x, 16) || ((ldx * (x_dtype == COSET_DTYPE_F32 ? 4 : 2)) % 16) != 0 || !aligned(layout, 16))
        return fail(COSET_E_ALIGN, "the layout and the rows of x must be 16-byte aligned");
    if (!aligned(codes, 4)) return fail(COSET_E_ALIGN, "codes must be 4-byte aligned");
    if (beta && blocks_per_tile < 1) return fail(COSET_E_BADARG, "blocks_per_tile must be >= 1");
    if (!(clip == clip)) return fail(COSET_E_BADARG, "clip is not a number");
    const int kb = n_in / 8;
    Product a = {};
    a.units = (kb + 7) / 8;
    a.w = (const uint4*)layout;
    a.hash = (const uint2*)((const uint8_t*)layout + (((int64_t)n_out + 15) / 16) * a.units * 1024);
    a.codes = (const uint32_t*)codes;
    a.wide_codes = aligned(codes, 16);
    if (codes && !(a.table = residual_table_q4((cudaStream_t)stream))) return COSET_E_STATE;
    a.beta = beta;
    a.n_out = n_out; a.kb = kb; a.T = T;
    a.x = x; a.ldx = ldx; a.ldy = ldy; a.bias = bias; a.clip = clip > 0.0f && clip < INFINITY ? clip : 0.0f;  // an infinite clamp is none
    for (int k = 0; k < n_targets; ++k) {
        if (!y_targets[k]) return fail(COSET_E_BADARG, "result buffer %d is null", k);
        a.out.y[k] = y_targets[k];
    }
    a.out.n = n_targets;
    a.out.bf16 = y_dtype == COSET_DTYPE_BF16 ? 1 : 0;
    const bool rows = scale_per_row(beta, blocks_per_tile, kb), one = blocks_per_tile == 1 && (kb % 8) == 0 && aligned(beta, 16);
    a.per_row = rows;
    a.rows_per_scale = rows && beta && kb > 0 ? (int)(blocks_per_tile / kb < n_out ? blocks_per_tile / kb : n_out) : 1;
    if (!rows) a.td = e8::make_tile_div(blocks_per_tile, (int64_t)n_out * kb);
    cudaStream_t st = (cudaStream_t)stream;
    const int scale_kind = rows ? kPerRow : (one ? kPerBlock : kPerTile);
    return x_dtype == COSET_DTYPE_BF16 ? launch_tokens<1>(a, scale_kind, st) : launch_tokens<3>(a, scale_kind, st);
}

extern "C" int coset_e8_vlut_product(const void* layout, const float* beta, int64_t blocks_per_tile, int n_out, int n_in, const void* x, int x_dtype,
                                     int64_t ldx, int T, const float* bias, void* const* y_targets, int n_targets, int y_dtype, int64_t ldy,
                                     float clip, void* stream) {
    return vlut_product(nullptr, layout, beta, blocks_per_tile, n_out, n_in, x, x_dtype, ldx, T, bias, y_targets, n_targets, y_dtype, ldy, clip, stream);
}

extern "C" int coset_e8_vlut_product_checked(const void* codes, const void* layout, const float* beta, int64_t blocks_per_tile, int n_out, int n_in,
                                             const void* x, int x_dtype, int64_t ldx, int T, const float* bias, void* const* y_targets, int n_targets,
                                             int y_dtype, int64_t ldy, float clip, void* stream) {
    if (!codes && n_out > 0 && T > 0 && n_in > 0) return fail(COSET_E_BADARG, "null pointer");
    return vlut_product(codes, layout, beta, blocks_per_tile, n_out, n_in, x, x_dtype, ldx, T, bias, y_targets, n_targets, y_dtype, ldy, clip, stream);
}
