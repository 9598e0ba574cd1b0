// Backward pass of the HNLQLinearQAT weight path (straight-through estimator).
//
// Forward (coset/core/layers.py:429-463):  U = e8_quantize(W * beta) / beta,  Wq = clamp(U, +-clip)
// is coset_e8_quantize with COSET_SCALE_MUL_TILE; it also emits the packed codes, so the backward
// pass re-creates U from 4 B/block instead of re-reading a saved 32 B/block tensor.
//
// Backward, as torch autograd evaluates the reference graph (clamp -> div -> STE -> mul,
// coset/core/layers.py:62-95 for the STE):
//   g_c      = g * 1[-clip <= U <= clip]
//   t        = g_c / beta                       (div backward w.r.t. the numerator)
//   dW       = t * beta                         (mul backward)
//   dbeta    = sum_tile  t * W - g_c * Q / beta^2  =  sum_tile t * (W - U),   Q = beta * U
#include <cooperative_groups.h>
#include <cuda_bf16.h>

#include "common.cuh"
#include "e8_fast.cuh"
#include "e8_io.cuh"
#include "e8_literal.cuh"

using namespace coset;

namespace {

constexpr int kThreads = 256;

// One block's contribution; returns the block's dbeta partial.
template <int DTG, bool Q4>
__device__ __forceinline__ float bwd_block(const void* __restrict__ g, const float* __restrict__ w,
                                           const void* __restrict__ codes, const uint2* __restrict__ table, float beta,
                                           float clip, int q, int64_t b, float* __restrict__ dw) {
    float gv[8], wv[8], qv[8], uv[8], out[8];
    e8::Row8<DTG>::load(g, b, gv);
    e8::Row8<0>::load(w, b, wv);
    if (Q4) {
        float v2[8];
        e8::decode_q4m2_twice(__ldg(reinterpret_cast<const uint32_t*>(codes) + b), table, v2);
        e8::scale_twice<2>(v2, beta, uv);
    } else {
        uint32_t words[2];
        if (q <= 4) {
            const uint16_t* c = reinterpret_cast<const uint16_t*>(codes) + b * 2;
            words[0] = c[0]; words[1] = c[1];
        } else {
            const uint32_t* c = reinterpret_cast<const uint32_t*>(codes) + b * 2;
            words[0] = c[0]; words[1] = c[1];
        }
        float qf = (float)q, wgt = 1.0f;
#pragma unroll
        for (int i = 0; i < 8; ++i) qv[i] = 0.0f;
        for (int m = 0; m < 2; ++m) {
            int d[8];
            float r[8];
            if (q <= 4) e8::unpack_level<2>(words[m], d); else e8::unpack_level<4>(words[m], d);
            e8::level_residual(d, qf, r);
#pragma unroll
            for (int i = 0; i < 8; ++i) qv[i] = __fadd_rn(qv[i], __fmul_rn(wgt, r[i]));
            wgt = __fmul_rn(wgt, qf);
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) uv[i] = __fdiv_rn(qv[i], beta);
    }
    float acc = 0.0f;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        float u = uv[i];
        bool pass = (clip > 0.0f) ? (u >= -clip && u <= clip) : (u == u);
        float gc = pass ? gv[i] : 0.0f;
        float t = __fdiv_rn(gc, beta);
        out[i] = __fmul_rn(t, beta);
        acc += t * (wv[i] - u);
    }
    e8::Row8<0>::store(dw, b, out);
    return acc;
}

__device__ __forceinline__ float sigmoidf_exact(float t) { return __fdiv_rn(1.0f, __fadd_rn(1.0f, expf(-t))); }

// The gradient of a scale, or of the theta that it came from: d theta = (d beta * range) * (1 - s) * s, the product torch
// autograd forms for mul followed by sigmoid.
struct ThetaRule {
    const float* theta;   // null: the gradient of beta itself is wanted
    const float* brange;
};
__device__ __forceinline__ float scale_gradient(float dbeta, const ThetaRule& r, int64_t tile) {
    if (!r.theta) return dbeta;
    const float s = sigmoidf_exact(__ldg(r.theta + tile));
    return __fmul_rn(__fmul_rn(__fmul_rn(dbeta, __ldg(r.brange + tile)), __fsub_rn(1.0f, s)), s);
}

// blocks_per_tile == 1: one thread per block, dbeta written directly.
template <int DTG, bool Q4>
__global__ void __launch_bounds__(kThreads)
k_bwd_block_tiles(const void* __restrict__ g, const float* __restrict__ w, const void* __restrict__ codes,
                  const uint2* __restrict__ table, const float* __restrict__ beta, float clip, int q, int64_t n,
                  float* __restrict__ dw, float* __restrict__ dbeta, ThetaRule rule) {
    int64_t b = (int64_t)blockIdx.x * kThreads + threadIdx.x;
    if (b >= n) return;
    float bt = __ldg(beta + b);
    float acc = bwd_block<DTG, Q4>(g, w, codes, table, bt, clip, q, b, dw);
    if (dbeta) dbeta[b] = scale_gradient(acc, rule, b);
}

// blocks_per_tile > 1 (one scale per weight row): one warp per tile, lanes stride over the
// tile's blocks (coalesced 1 KiB per step), shuffle reduction, no scratch memory.
template <int DTG, bool Q4>
__global__ void __launch_bounds__(kThreads)
k_bwd_row_tiles(const void* __restrict__ g, const float* __restrict__ w, const void* __restrict__ codes,
                const uint2* __restrict__ table, const float* __restrict__ beta, float clip, int q, int64_t n,
                int64_t bpt, int64_t tiles, float* __restrict__ dw, float* __restrict__ dbeta, ThetaRule rule) {
    int64_t tile = ((int64_t)blockIdx.x * kThreads + threadIdx.x) >> 5;
    int lane = threadIdx.x & 31;
    if (tile >= tiles) return;
    float bt = __ldg(beta + tile);
    int64_t lo = tile * bpt, hi = lo + bpt;
    if (hi > n) hi = n;
    float acc = 0.0f;
    for (int64_t b = lo + lane; b < hi; b += 32) acc += bwd_block<DTG, Q4>(g, w, codes, table, bt, clip, q, b, dw);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (lane == 0 && dbeta) dbeta[tile] = scale_gradient(acc, rule, tile);
}

// Per-tile scale of the layer (coset/core/layers.py:415-417):
//   beta = beta_min + sigmoid(theta) * (beta_max - beta_min),   sigmoid(t) = 1 / (1 + exp(-t))
// and, in the same launch, the bias rounded to bf16 for a bf16 product (n_bias = 0: none).
__global__ void __launch_bounds__(kThreads)
k_layer_beta(const float* __restrict__ theta, const float* __restrict__ bmin, const float* __restrict__ brange, int64_t tiles,
             float* __restrict__ beta, const float* __restrict__ bias, int64_t n_bias, __nv_bfloat16* __restrict__ bias16) {
    int64_t i = (int64_t)blockIdx.x * kThreads + threadIdx.x;
    if (i < n_bias) bias16[i] = __float2bfloat16_rn(__ldg(bias + i));
    if (i >= tiles) return;
    beta[i] = __fadd_rn(__ldg(bmin + i), __fmul_rn(sigmoidf_exact(__ldg(theta + i)), __ldg(brange + i)));
}

// Column sums of a row-major [rows, cols] matrix: the gradient of the bias, the sum of the gradient of the output over the
// tokens.  Bound: one read of the matrix.  A CTA of 256 threads owns one 128-byte column strip (8 lanes of 16 bytes) and
// every kColSplits-th group of 32 rows; the CTAs of a strip form a cluster, whose first CTA adds their partial sums
// through distributed shared memory in a fixed order, so no scratch memory, no atomics and no second launch.  Sums are
// float32; of float32 elements they keep what rounding takes from them, and all partial sums do, so that the error is that of
// the last rounding (2.6e-8 against 64 bits; plain chains gave 1.1e-7, torch's reduction 8e-8; price 9.8 -> 12.2 us for [8192, 1024]).
// WIDE = false: one element per lane, where the rows are not 16-byte aligned.
// Measured against torch's reduction: [4096, 3072] bf16 18.2 -> 5.1 us (4.9 TB/s), [128, 768] float32 4.5 -> 2.9.
constexpr int kColSplits = 8, kColLanes = 8, kColRows = kThreads / kColLanes;

template <int DT, bool WIDE>
__global__ void __launch_bounds__(kThreads)
k_column_sum(const void* __restrict__ x, int64_t rows, int64_t cols, void* __restrict__ out, int out_bf16) {
    constexpr int E = WIDE ? (DT == 0 ? 4 : 8) : 1;  // elements per lane
    __shared__ float part[kColRows][kColLanes * E + 1], part_lost[DT == 0 ? kColRows : 1][kColLanes * E + 1];
    __shared__ float total[kColLanes * E], total_lost[kColLanes * E];
    cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
    const int lane = threadIdx.x % kColLanes, row = threadIdx.x / kColLanes, split = blockIdx.x % kColSplits;
    const int64_t strip = blockIdx.x / kColSplits, col = (strip * kColLanes + lane) * E;
    float acc[E], lost[E];
#pragma unroll
    for (int e = 0; e < E; ++e) acc[e] = lost[e] = 0.0f;
    if (col < cols) {
#pragma unroll 8
        for (int64_t r = (int64_t)split * kColRows + row; r < rows; r += kColSplits * kColRows) {
            if constexpr (!WIDE) {
                const int64_t at = r * cols + col;
                if (DT == 0) add_exactly(acc[0], lost[0], __ldcs((const float*)x + at));
                else acc[0] += __bfloat162float(((const __nv_bfloat16*)x)[at]);
            } else if constexpr (DT == 0) {
                const float4 v = __ldcs(reinterpret_cast<const float4*>((const float*)x + r * cols + col));
                add_exactly(acc[0], lost[0], v.x); add_exactly(acc[1], lost[1], v.y);
                add_exactly(acc[2], lost[2], v.z); add_exactly(acc[3], lost[3], v.w);
            } else {
                const uint4 v = __ldcs(reinterpret_cast<const uint4*>((const __nv_bfloat16*)x + r * cols + col));
                const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    acc[2 * e] += __uint_as_float(w[e] << 16);
                    acc[2 * e + 1] += __uint_as_float(w[e] & 0xffff0000u);
                }
            }
        }
    }
#pragma unroll
    for (int e = 0; e < E; ++e) {
        part[row][lane * E + e] = acc[e];
        if (DT == 0) part_lost[row][lane * E + e] = lost[e];
    }
    __syncthreads();
    if (threadIdx.x < kColLanes * E) {
        float s = 0.0f, l = 0.0f;
#pragma unroll
        for (int r = 0; r < kColRows; ++r) {
            add_exactly(s, l, part[r][threadIdx.x]);
            if (DT == 0) l += part_lost[r][threadIdx.x];
        }
        total[threadIdx.x] = s;
        total_lost[threadIdx.x] = l;
    }
    cluster.sync();
    if (split == 0 && threadIdx.x < kColLanes * E) {
        const int64_t c = strip * kColLanes * E + threadIdx.x;
        float s = 0.0f, l = 0.0f;
#pragma unroll
        for (int k = 0; k < kColSplits; ++k) {
            add_exactly(s, l, cluster.map_shared_rank(total, k)[threadIdx.x]);
            l += cluster.map_shared_rank(total_lost, k)[threadIdx.x];
        }
        if (l == l) s += l;  // not a number beside an infinite sum
        if (c < cols) {
            if (out_bf16) reinterpret_cast<__nv_bfloat16*>(out)[c] = __float2bfloat16_rn(s);
            else reinterpret_cast<float*>(out)[c] = s;
        }
    }
    cluster.sync();  // no CTA leaves while its sums are read
}

}  // namespace

extern "C" int coset_layer_beta_bias(const float* theta, const float* beta_min, const float* beta_range, int64_t n_tiles,
                                     float* beta, const float* bias, int64_t n_bias, void* bias_bf16, void* stream) {
    if (n_tiles < 0 || n_bias < 0) return fail(COSET_E_BADARG, "n_tiles or n_bias is negative");
    if (n_tiles == 0 && n_bias == 0) return 0;
    if (n_tiles > 0 && (!theta || !beta_min || !beta_range || !beta)) return fail(COSET_E_BADARG, "null pointer");
    if (n_bias > 0 && (!bias || !bias_bf16)) return fail(COSET_E_BADARG, "null pointer");
    const int64_t n = n_tiles > n_bias ? n_tiles : n_bias;
    k_layer_beta<<<(unsigned)((n + kThreads - 1) / kThreads), kThreads, 0, (cudaStream_t)stream>>>(
        theta, beta_min, beta_range, n_tiles, beta, bias, n_bias, (__nv_bfloat16*)bias_bf16);
    return check_launch("layer_beta");
}

extern "C" int coset_layer_beta(const float* theta, const float* beta_min, const float* beta_range, int64_t n_tiles,
                                float* beta, void* stream) {
    return coset_layer_beta_bias(theta, beta_min, beta_range, n_tiles, beta, nullptr, 0, nullptr, stream);
}

extern "C" int coset_column_sum(const void* x, int x_dtype, int64_t rows, int64_t cols, void* out, int out_dtype, void* stream) {
    if (rows < 0 || cols < 0) return fail(COSET_E_BADARG, "negative size");
    if ((x_dtype != COSET_DTYPE_F32 && x_dtype != COSET_DTYPE_BF16) || (out_dtype != COSET_DTYPE_F32 && out_dtype != COSET_DTYPE_BF16))
        return fail(COSET_E_BADARG, "unknown dtype");
    if (cols == 0) return 0;
    if (!out || (rows > 0 && !x)) return fail(COSET_E_BADARG, "null pointer");
    const int elem = x_dtype == COSET_DTYPE_F32 ? 4 : 2;
    if (!aligned(x, elem)) return fail(COSET_E_ALIGN, "x is not aligned to its elements");
    const bool wide = aligned(x, 16) && (cols * elem) % 16 == 0;
    const int64_t per_strip = kColLanes * (wide ? 16 / elem : 1), strips = (cols + per_strip - 1) / per_strip;
    if (strips > 0x7fffffff / kColSplits) return fail(COSET_E_UNSUPPORTED, "too many columns");
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = kColSplits;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.gridDim = dim3((unsigned)(strips * kColSplits));
    cfg.blockDim = dim3(kThreads);
    cfg.stream = (cudaStream_t)stream;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    const int bf16 = out_dtype == COSET_DTYPE_BF16 ? 1 : 0;
    cudaError_t e;
    if (x_dtype == COSET_DTYPE_F32) e = wide ? cudaLaunchKernelEx(&cfg, k_column_sum<0, true>, x, rows, cols, out, bf16) : cudaLaunchKernelEx(&cfg, k_column_sum<0, false>, x, rows, cols, out, bf16);
    else e = wide ? cudaLaunchKernelEx(&cfg, k_column_sum<1, true>, x, rows, cols, out, bf16) : cudaLaunchKernelEx(&cfg, k_column_sum<1, false>, x, rows, cols, out, bf16);
    if (int rc = check_cuda(e, "column_sum")) return rc;
    return check_launch("column_sum");
}

extern "C" int coset_e8_layer_fake_quant_fwd(const float* w, const float* theta, const float* beta_min, const float* beta_range,
                                             int64_t n_blocks, int64_t blocks_per_tile, int q, float clip, void* out,
                                             int out_dtype, void* codes, float* beta, void* stream) {
    if (n_blocks < 0 || blocks_per_tile < 1) return fail(COSET_E_BADARG, "bad n_blocks / blocks_per_tile");
    const int64_t tiles = (n_blocks + blocks_per_tile - 1) / blocks_per_tile;
    if (int e = coset_layer_beta(theta, beta_min, beta_range, tiles, beta, stream)) return e;
    return coset_e8_quantize(w, COSET_DTYPE_F32, beta, COSET_SCALE_MUL_TILE, n_blocks, blocks_per_tile, q, 2, clip, out,
                             out_dtype, codes, stream);
}

static int fake_quant_bwd(const void* grad_out, int grad_dtype, const float* w, const void* codes, const float* beta, int64_t n_blocks,
                          int64_t blocks_per_tile, int q, float clip, float* grad_w, float* grad_beta, ThetaRule rule, void* stream) {
    if (n_blocks < 0 || blocks_per_tile < 1) return fail(COSET_E_BADARG, "bad n_blocks / blocks_per_tile");
    if (n_blocks == 0) return 0;
    if (!grad_out || !w || !codes || !beta || !grad_w) return fail(COSET_E_BADARG, "null pointer");
    if (grad_dtype != COSET_DTYPE_F32 && grad_dtype != COSET_DTYPE_BF16) return fail(COSET_E_BADARG, "unknown grad_dtype");
    if (q < 2 || q > 16) return fail(COSET_E_UNSUPPORTED, "unsupported q=%d", q);
    if (!aligned(grad_out, 16) || !aligned(w, 16) || !aligned(grad_w, 16) || !aligned(codes, 4))
        return fail(COSET_E_ALIGN, "grad_out, w, grad_w must be 16-byte and codes 4-byte aligned");
    if (n_blocks > ((int64_t)1 << 36)) return fail(COSET_E_BADARG, "n_blocks too large");
    cudaStream_t st = (cudaStream_t)stream;
    const uint2* table = nullptr;
    if (q == 4) {
        table = residual_table_q4(st);
        if (!table) return COSET_E_STATE;
    }
#define LAUNCH_BWD(DTG, Q4)                                                                                       \
    do {                                                                                                          \
        if (blocks_per_tile == 1) {                                                                               \
            unsigned grid = (unsigned)((n_blocks + kThreads - 1) / kThreads);                                     \
            k_bwd_block_tiles<DTG, Q4><<<grid, kThreads, 0, st>>>(grad_out, w, codes, table, beta, clip, q,       \
                                                                  n_blocks, grad_w, grad_beta, rule);             \
        } else {                                                                                                  \
            int64_t tiles = (n_blocks + blocks_per_tile - 1) / blocks_per_tile;                                   \
            unsigned grid = (unsigned)((tiles * 32 + kThreads - 1) / kThreads);                                   \
            k_bwd_row_tiles<DTG, Q4><<<grid, kThreads, 0, st>>>(grad_out, w, codes, table, beta, clip, q,         \
                                                                n_blocks, blocks_per_tile, tiles, grad_w,         \
                                                                grad_beta, rule);                                 \
        }                                                                                                         \
    } while (0)
    if (grad_dtype == COSET_DTYPE_F32) {
        if (q == 4) LAUNCH_BWD(0, true); else LAUNCH_BWD(0, false);
    } else {
        if (q == 4) LAUNCH_BWD(1, true); else LAUNCH_BWD(1, false);
    }
#undef LAUNCH_BWD
    return check_launch("e8_fake_quant_bwd");
}

extern "C" int coset_e8_fake_quant_bwd(const void* grad_out, int grad_dtype, const float* w, const void* codes,
                                       const float* beta, int64_t n_blocks, int64_t blocks_per_tile, int q,
                                       float clip, float* grad_w, float* grad_beta, void* stream) {
    return fake_quant_bwd(grad_out, grad_dtype, w, codes, beta, n_blocks, blocks_per_tile, q, clip, grad_w, grad_beta, ThetaRule{nullptr, nullptr}, stream);
}

extern "C" int coset_e8_layer_fake_quant_bwd(const void* grad_out, int grad_dtype, const float* w, const void* codes,
                                             const float* beta, const float* theta, const float* beta_range, int64_t n_blocks,
                                             int64_t blocks_per_tile, int q, float clip, float* grad_w, float* grad_theta,
                                             void* stream) {
    if (grad_theta && n_blocks > 0 && (!theta || !beta_range)) return fail(COSET_E_BADARG, "null pointer");
    return fake_quant_bwd(grad_out, grad_dtype, w, codes, beta, n_blocks, blocks_per_tile, q, clip, grad_w, grad_theta,
                          ThetaRule{theta, beta_range}, stream);
}
