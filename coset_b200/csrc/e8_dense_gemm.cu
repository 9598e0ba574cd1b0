// Dense products of medium size in bf16, float32 sums, one rounding of the result:
//     y[T, N] = x[T, K] W[N, K]^T + bias (float32)    a layer's kept dense weight with some tens to some thousand tokens
//     dx[T, K] = g[T, N] W[N, K]                       and the two products of a training layer's backward pass: the same kernel, with one
//     dw[N, K] = g[T, N]^T x[T, K]                     or both operands read along the other dimension (MN-major tiles)
//
// Between 17 and 2047 tokens a 4096 x 4096 layer has 32 MB of weights to stream and 0.6 to 69 GFLOP to do: the tiles must be large
// in features (so that the tokens are not read over and over) and there must be enough of them for 148 SMs.  So a pair of CTAs
// owns 256 features (tcgen05.mma.cta_group::2, M = 256: features are the rows, tokens the N of the instruction, 32 to 256 of them, so
// that no tensor work is done for tokens that are not there), and where feature and token tiles leave SMs idle, K is split
// over the 2 or 4 pairs of one cluster.  The pairs then add their sums through distributed shared memory in the order of K: every pair
// owns a part of the tokens, receives the others' sums for it and stores it.  No scratch memory, no second launch, same bits in
// every run.  The bias joins the float32 sums.
//
// Roles of the warps and the barriers of a pair are those of k_gemm_pair (e8_decode_gemm.cu); every wait is bounded in time.  What bounds
// a small product is latency: 2.3 thousand cycles until the first load, 1.2 until it arrives, 105 ns per K step of 64 with 32 or 64 tokens (the issue
// of its four instructions and one wait; stages of two steps below 160 tokens share the wait), 2 to 7 thousand cycles for the sums.  The kernel is
// launched as a programmatic dependent, which hides about 2 us of that behind the kernel before it.
// Two CTAs fit an SM (ten warps, at most 112 KB of stages) where there are more tiles than SMs.
// Measured on the device, 4096 x 4096 (graph replays, three weights in turn), this kernel / torch's product with its cast of the bias / without a bias: 64 tokens
// 11.3 / 10.8 / 8.7 us, 256 tokens 14.5 / 13.1 / 10.9, 1024 tokens 26.9 / 26.6 / 25.1.  It costs the host one launch, and the host bounds such a call: the
// layer's with 256 tokens 21.6 -> 14.6 us where weights alternate, 19.3 -> 11.7 on one weight, 14.8 -> 11.6 without a bias.  The products of a training
// step of a [3072, 768] layer with 4096 tokens: 26.3 + 17.0 + 17.3 us against 18.4 + 16.0 + 14.7 for torch's, but the host bounds the step: 146 -> 118 us.
#include <cuda.h>
#include <cuda_bf16.h>
#include <math.h>

#include "common.cuh"
#include "umma.cuh"

using namespace coset;
using namespace coset::umma;

namespace {

constexpr int kRows = 128;           // weight rows of one CTA
constexpr int kMaxStages = 8;
constexpr int kEpilogueWarps = 8, kTmaWarp = 8, kMmaWarp = 9;
constexpr int kThreads = 10 * 32;
constexpr int kAlignment = 1024;         // of the stages, which the base of the shared memory need not have
constexpr int kSmemBudget = 227 * 1024 - kAlignment;
constexpr int kSmemOfTwo = 112 * 1024;   // two CTAs on an SM (228 KB, 1 KB of which each CTA takes)
constexpr int kMostSize = INT32_MAX - 512;
constexpr int kBarrierBytes = 16 * kMaxStages + 16;
constexpr int kScratchRow = 40;       // 32 features and a pad, in values
constexpr int kScratchBytes = kEpilogueWarps * 32 * kScratchRow * 2;

struct Plan {
    int tokens;  // N of the instruction: tokens of one pair, a multiple of 32 up to 256
    int split;   // pairs that share K: 1, 2 or 4
    int stages;
    int sub;     // 64-wide K steps of a stage
};

struct Shape {
    int N, K, T;
    Plan plan;
    const float* bias;
    int round_bias;   // to bf16 before it is added, as torch does
    __nv_bfloat16* y;
    int64_t ldy;
    int vector_rows;  // rows of y are made of 16-byte chunks
    int* status;
    int late;         // the pair of each cluster that takes its first wait for run out, -1: none (see coset_e8_dense_linear_late)
};

// what a pair receives of the others' sums: apart from the stages, which a slower pair may still be using when a faster one sends
__host__ __device__ constexpr int sums_bytes(int tokens, int split) { return (split - 1) * (tokens / split) * kRows * 4; }
__host__ __device__ constexpr int stage_bytes(int tokens, int sub) { return sub * (kRows + tokens / 2) * BK * 2; }

// Columns (tokens) of this CTA's accumulator that other pairs own, W at a time, into their reduction buffers [slot][token][row]; where a wait gave
// up no numbers, so that the sums of no pair are taken for whole.
template <int W>
__device__ __forceinline__ void send_columns(const Shape& s, bool ok, uint32_t tmem, uint32_t base, int pair, int half, int row, int group) {
    const int own = s.plan.tokens / s.plan.split;
    for (int c = group * W; c < s.plan.tokens; c += (kEpilogueWarps / 4) * W) {
        const int to = c / own;  // W divides own
        if (to == pair) continue;
        uint32_t r[W];
        tmem_ld(tmem + (uint32_t)c, r);
        const int slot = pair < to ? pair : pair - 1;
        const uint32_t dst = peer_smem(base, (uint32_t)(2 * to + half)) + (uint32_t)(((slot * own + c - to * own) * kRows + row) * 4);
#pragma unroll
        for (int j = 0; j < W; ++j) asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(dst + (uint32_t)(j * kRows * 4)), "r"(ok ? r[j] : 0x7fffffffu) : "memory");
    }
}
// The columns this pair owns: summed with what the others sent, plus bias, rounded and stored.  A lane holds one feature and W tokens;
// a scratch of the warp turns them into rows of 32 features, so that four lanes store the 64 bytes of a token.
template <int W>
__device__ __forceinline__ void store_columns(const Shape& s, bool ok, uint32_t tmem, const float* sums, __nv_bfloat16* scratch, int pair, int row, int group, int feature0,
                                              int token0) {
    const int own = s.plan.tokens / s.plan.split, lane = threadIdx.x & 31;
    float bias = !ok ? NAN : s.bias && feature0 + lane < s.N ? __ldg(behind_wait(s.bias) + feature0 + lane) : 0.0f;  // a wait gave up: no number
    if (s.round_bias) bias = __bfloat162float(__float2bfloat16_rn(bias));
    for (int c = group * W; c < own; c += (kEpilogueWarps / 4) * W) {
        const int t = token0 + pair * own + c;
        if (t >= s.T || feature0 >= s.N) break;
        uint32_t r[W];
        tmem_ld(tmem + (uint32_t)(pair * own + c), r);
        float v[W];
#pragma unroll
        for (int j = 0; j < W; ++j) v[j] = 0.0f;
        for (int p = 0; p < s.plan.split; ++p) {  // in the order of K
            if (p == pair) {
#pragma unroll
                for (int j = 0; j < W; ++j) v[j] += __uint_as_float(r[j]);
            } else {
                const float* from = sums + ((p < pair ? p : p - 1) * own + c) * kRows + row;
#pragma unroll
                for (int j = 0; j < W; ++j) v[j] += from[j * kRows];
            }
        }
#pragma unroll
        for (int j = 0; j < W; ++j) scratch[j * kScratchRow + lane] = __float2bfloat16_rn(v[j] + bias);
        __syncwarp();
        const int count = s.T - t < W ? s.T - t : W;
        if (s.vector_rows) {
            const int chunk = lane & 3;
            __nv_bfloat16* y = s.y + (int64_t)(t + (lane >> 2)) * s.ldy + feature0 + 8 * chunk;
            if (feature0 + 8 * chunk < s.N) {
#pragma unroll
                for (int j = 0; j < W; j += 8, y += 8 * s.ldy)
                    if (j + (lane >> 2) < count) *reinterpret_cast<uint4*>(y) = *reinterpret_cast<const uint4*>(scratch + (j + (lane >> 2)) * kScratchRow + 8 * chunk);
            }
        } else if (feature0 + lane < s.N) {
            for (int j = 0; j < count; ++j) s.y[(int64_t)(t + j) * s.ldy + feature0 + lane] = scratch[j * kScratchRow + lane];
        }
        __syncwarp();
    }
}

// One K step of 64 of an operand's `rows` rows from `row0` on into `dst`.
template <bool MN>
__device__ __forceinline__ void load_operand(uint32_t dst, const CUtensorMap* map, int rows, int row0, int k0, uint32_t bar) {
    if (!MN) tma_load_pair(dst, map, k0, row0, bar);
    else
        for (int r = 0; r < rows; r += 64) tma_load_pair(dst + (uint32_t)(r * BK * 2), map, row0 + r, k0, bar);
}

// W_MN, X_MN: the operand lies in memory with K as its slow dimension.
template <int kSub, bool W_MN, bool X_MN>
__global__ void __launch_bounds__(kThreads, 2)
k_linear_pair(const __grid_constant__ CUtensorMap x_map, const __grid_constant__ CUtensorMap w_map, const __grid_constant__ Shape s) {
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw = smem_u32(smem_raw);
    const uint32_t base = (raw + 1023u) & ~1023u;  // the same offset in all CTAs of the cluster
    uint8_t* gen = smem_raw + (base - raw);
    const int bytes = stage_bytes(s.plan.tokens, kSub), stages = s.plan.stages;
    const uint32_t bar_base = base + (uint32_t)(stages * bytes);
    const uint32_t full_base = bar_base + 8 * kMaxStages, done_bar = bar_base + 16 * kMaxStages;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(gen + stages * bytes + 16 * kMaxStages + 8);

    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const uint32_t crank = __shfl_sync(0xffffffffu, cluster_rank(), 0);
    const int half = (int)(crank & 1u), pair = (int)(crank >> 1);
    const bool leader = half == 0;
    const uint16_t both = (uint16_t)(3u << (crank & ~1u));
    const uint32_t leader_full = peer_smem(base, crank & ~1u) + (full_base - base);
    const int row0 = (int)(blockIdx.x / (2 * s.plan.split)) * 2 * kRows + half * kRows;  // this CTA's features
    const int token0 = (int)blockIdx.y * s.plan.tokens;                                  // this pair's tokens
    uint32_t columns = 32;
    while ((int)columns < s.plan.tokens) columns *= 2;

    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(columns) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    if (tid == kTmaWarp * 32) {
        asm volatile("prefetch.tensormap [%0];" ::"l"(&w_map) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(&x_map) : "memory");
        for (int i = 0; i < stages; ++i) {
            mbar_init(bar_base + 8 * i, 1);   // empty: one commit
            mbar_init(full_base + 8 * i, 1);  // full (used in the leader): its arrive + both CTAs' bytes
        }
        mbar_init(done_bar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    cluster_sync();  // the partner's barriers exist before anything arrives on them
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = __shfl_sync(0xffffffffu, *tmem_slot, 0);
    bool ok = true;
    grid_wait();
    grid_trigger();

    const int steps = (s.K + BK - 1) / BK, split_log2 = s.plan.split >> 1;  // 1, 2, 4
    const int first = steps * pair >> split_log2, last = steps * (pair + 1) >> split_log2;
    const uint32_t x_at = kSub * kRows * BK * 2, x_bytes = (uint32_t)(s.plan.tokens * BK);
    if (warp == kTmaWarp) {
        int stage = 0;
        uint32_t phase = 1;  // of the round before
        for (int k = first, n = 0; k < last; k += kSub, ++n) {
            if (n >= stages && !mbar_wait_warp(bar_base + 8 * stage, phase)) { ok = false; break; }
            if (elect_one()) {  // rows beyond N or T and columns beyond K arrive as zeros
                const uint32_t at = base + (uint32_t)(stage * bytes), bar = leader_full + 8 * stage;
                const int subs = last - k < kSub ? last - k : kSub;
                if (leader) mbar_arrive_expect_tx(full_base + 8 * stage, (uint32_t)(2 * subs) * (kRows * BK * 2 + x_bytes));
#pragma unroll
                for (int i = 0; i < kSub; ++i)
                    if (i < subs) {
                        load_operand<W_MN>(at + i * (kRows * BK * 2), &w_map, kRows, row0, (k + i) * BK, bar);
                        load_operand<X_MN>(at + x_at + i * x_bytes, &x_map, s.plan.tokens / 2, token0 + half * (s.plan.tokens / 2), (k + i) * BK, bar);
                    }
            }
            __syncwarp();
            if (++stage == stages) { stage = 0; phase ^= 1u; }
        }
    } else if (warp == kMmaWarp && leader) {
        // the descriptors of all tiles differ in the 14-bit address field alone (units of 16 bytes)
        const uint64_t w0 = W_MN ? umma_desc_mn(base) : umma_desc(base), x0 = X_MN ? umma_desc_mn(base) : umma_desc(base);
        const uint32_t w_hi = (uint32_t)(w0 >> 32), w_lo = (uint32_t)w0, x_hi = (uint32_t)(x0 >> 32), x_lo = (uint32_t)x0;
        constexpr uint32_t kWStep = W_MN ? 128 : 2, kXStep = X_MN ? 128 : 2;  // 16 of K: two groups of eight rows, or 32 bytes inside the swizzle row
        // kind::f16: float32 sums, bf16 x bf16, M = 256 over the pair
        const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((W_MN ? 1u : 0u) << 15) | ((X_MN ? 1u : 0u) << 16) | ((uint32_t)(s.plan.tokens >> 3) << 17) | ((uint32_t)(256 >> 4) << 24);
        int stage = 0;
        uint32_t phase = 0;
        for (int k = first; k < last; k += kSub) {
            if (pair == s.late || !mbar_wait_warp(full_base + 8 * stage, phase)) { ok = false; break; }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            if (elect_one()) {
                const uint32_t a_lo = w_lo + (uint32_t)(stage * (bytes >> 4)), b_lo = x_lo + (uint32_t)(stage * (bytes >> 4)) + (x_at >> 4);
#pragma unroll
                for (int i = 0; i < kSub; ++i)
                    if (i == 0 || k + i < last) {
#pragma unroll
                        for (int j = 0; j < BK / 16; ++j)
                            umma_f16_pair(tmem, make_desc(a_lo + (uint32_t)(i * (kRows * BK * 2 >> 4)) + (uint32_t)j * kWStep, w_hi),
                                          make_desc(b_lo + (uint32_t)i * (x_bytes >> 4) + (uint32_t)j * kXStep, x_hi), idesc, i + j > 0 || k > first ? 1u : 0u);
                    }
                umma_commit_pair(bar_base + 8 * stage, both);
                if (k + kSub >= last) umma_commit_pair(done_bar, both);
            }
            __syncwarp();
            if (++stage == stages) { stage = 0; phase ^= 1u; }
        }
    }
    __syncwarp();
    if (!ok && s.status) atomicExch(s.status, 1);
    ok = __all_sync(0xffffffffu, mbar_wait_cluster<32>(done_bar, 0u) && ok);  // always: the products must have retired before tensor memory is read or freed
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");

    const int quarter = warp & 3, group = warp >> 2, row = quarter * 32 + lane;  // a warp reads lanes 32 (warp % 4) .. + 31
    const uint32_t lanes = tmem + ((uint32_t)(quarter * 32) << 16);
    const int own = s.plan.tokens / s.plan.split;
    if (s.plan.split > 1) {
        if (warp < kEpilogueWarps) {
            if (own >= 64) send_columns<16>(s, ok, lanes, bar_base + kBarrierBytes, pair, half, row, group);
            else send_columns<8>(s, ok, lanes, bar_base + kBarrierBytes, pair, half, row, group);
        }
        cluster_sync();  // ... and the sums have arrived
    }
    if (warp < kEpilogueWarps) {
        const float* sums = reinterpret_cast<const float*>(gen + stages * bytes + kBarrierBytes);
        __nv_bfloat16* scratch = reinterpret_cast<__nv_bfloat16*>(gen) + warp * 32 * kScratchRow;
        const int feature0 = row0 + quarter * 32;
        if (own >= 128) store_columns<32>(s, ok, lanes, sums, scratch, pair, row, group, feature0, token0);
        else if (own >= 64) store_columns<16>(s, ok, lanes, sums, scratch, pair, row, group, feature0, token0);
        else store_columns<8>(s, ok, lanes, sums, scratch, pair, row, group, feature0, token0);
    }
    if (!ok) {
        if (s.status) atomicExch(s.status, 1);
        for (int i = 0; i < 64; ++i) __nanosleep(1000);  // a wait gave up: leave copies still in flight time to land
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    cluster_sync();  // neither CTA frees tensor memory or leaves while the pair's work could still touch it
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(columns) : "memory");
}

// Stages: what fits, no more than there is work for, and room for the epilogue's scratch.
Plan with_stages(int tokens, int split, int steps, bool two = false) {
    Plan p = {tokens, split, 1, tokens <= 128 ? 2 : 1};
    const int bytes = stage_bytes(tokens, p.sub), need = ((steps + split - 1) / split + p.sub - 1) / p.sub, least = (kScratchBytes + bytes - 1) / bytes;
    p.stages = ((two ? kSmemOfTwo : kSmemBudget) - kBarrierBytes - sums_bytes(tokens, split)) / bytes;
    if (p.stages > kMaxStages) p.stages = kMaxStages;
    if (p.stages > need) p.stages = need;
    if (p.stages < least) p.stages = least;
    return p;
}

// Clusters of 2 * split CTAs that the device runs at once.  148 SMs hold 74 pairs, but the GPCs' sizes leave fewer places for larger
// clusters (14 of eight CTAs: 16 took two waves).
int clusters_at_once(int split) { return split == 1 ? sm_count() / 2 : split == 2 ? sm_count() * 35 / 148 : sm_count() * 13 / 148; }

// The plan of the least estimated time in ns.  Measured over 41 products from [17, 4096] x [4096, 4096] to [4096, 2048] x [2048, 2048] in all three
// forms: a K step of 64 takes 110 ns with 16 pairs at work and 155 with 74 (the loads), or 1.4 ns a token (the tensor cores, from 110
// tokens on); the exchange of the sums 1.7 us with 32 tokens and two pairs and 4.4 with 256; every further round of clusters 2 to 4 us where a CTA has
// an SM to itself, and half of that where two share one and each one's loads and stores run under the other's products ([4096, 2048] x [2048, 2048]
// 30.3 -> 26.8 us).  The plan taken was within 3 % of the best one on average, 15 % at worst.
Plan make_plan(int N, int K, int T, int unit) {  // unit: tokens come in multiples of it
    const int steps = (K + BK - 1) / BK;
    Plan best = with_stages(unit, 1, steps);
    double least = 0.0;
    for (int tokens = unit; tokens <= 256 && tokens < T + unit; tokens += unit)
        for (int split = 1; split <= 4 && split <= steps; split *= 2) {
            const int64_t clusters = (int64_t)((N + 2 * kRows - 1) / (2 * kRows)) * ((T + tokens - 1) / tokens);
            const int64_t at_once = clusters_at_once(split), rounds = (clusters + at_once - 1) / at_once, pairs = clusters * split < 74 ? clusters * split : 74;
            const bool two = rounds > 1 && split == 1;
            const double loads = 100.0 + 0.75 * (double)pairs, products = 1.4 * tokens, step = loads > products ? loads : products;
            const double exchange = split == 1 ? 0.0 : split == 2 ? 1300.0 + 12.0 * tokens : 1800.0 + 16.0 * tokens;
            const double time = exchange + (double)rounds * ((steps + split - 1) / split) * step + (double)(rounds - 1) * (two ? 2200.0 : 4300.0);
            if (least == 0.0 || time < least) {
                least = time;
                best = with_stages(tokens, split, steps, two);
            }
        }
    return best;
}

template <int kSub, bool W_MN, bool X_MN>
int launch_linear(const CUtensorMap& x_map, const CUtensorMap& w_map, const Shape& s, cudaStream_t st) {
    const int smem = kAlignment + s.plan.stages * stage_bytes(s.plan.tokens, kSub) + kBarrierBytes + sums_bytes(s.plan.tokens, s.plan.split);
    const auto kernel = k_linear_pair<kSub, W_MN, X_MN>;
    // The bound belongs to the kernel, not to the call: what any plan may ask for, so that no thread lowers it between another's two calls.
    if (int e = check_cuda(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kAlignment + kSmemBudget), "cudaFuncSetAttribute")) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)((s.N + 2 * kRows - 1) / (2 * kRows) * 2 * s.plan.split), (unsigned)((s.T + s.plan.tokens - 1) / s.plan.tokens));
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = (size_t)smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)(2 * s.plan.split);
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    return check_cuda(cudaLaunchKernelEx(&cfg, kernel, x_map, w_map, s), "dense product");
}

template <bool W_MN, bool X_MN>
int dense_product(const void* w, int64_t ldw, const void* x, int64_t ldx, int N, int T, int K, const float* bias, int round_bias, void* y, int64_t ldy,
                  int* status, void* stream, const Plan* given = nullptr, int late = -1) {
    if (N < 0 || T < 0 || K < 0) return fail(COSET_E_BADARG, "negative size");
    if (N > kMostSize || T > kMostSize || K > kMostSize) return fail(COSET_E_UNSUPPORTED, "sizes are counted in 32 bits, with room for a tile");
    if (N == 0 || T == 0) return 0;
    if (K == 0) return fail(COSET_E_BADARG, "nothing to sum over");
    if (!w || !x || !y) return fail(COSET_E_BADARG, "null pointer");
    if (ldw < (W_MN ? N : K) || ldx < (X_MN ? T : K) || ldw % 8 != 0 || ldx % 8 != 0 || ldy < N)
        return fail(COSET_E_BADARG, "leading dimensions: at least a row, and multiples of 8 for the operands");
    if (!aligned(x, 16) || !aligned(w, 16)) return fail(COSET_E_ALIGN, "the operands must be 16-byte aligned");
    Shape s = {N, K, T, given ? *given : make_plan(N, K, T, X_MN ? 128 : 32), bias, round_bias, (__nv_bfloat16*)y, ldy, aligned(y, 16) && ldy % 8 == 0 && N % 8 == 0, status, late};
    if ((T + s.plan.tokens - 1) / s.plan.tokens > 65535) return fail(COSET_E_UNSUPPORTED, "too many columns");
    CUtensorMap x_map, w_map;
    if (int e = X_MN ? make_bf16_map(&x_map, x, T, K, ldx, BK) : make_bf16_map(&x_map, x, K, T, ldx, s.plan.tokens / 2)) return e;
    if (int e = W_MN ? make_bf16_map(&w_map, w, N, K, ldw, BK) : make_bf16_map(&w_map, w, K, N, ldw, kRows)) return e;
    return s.plan.sub == 2 ? launch_linear<2, W_MN, X_MN>(x_map, w_map, s, (cudaStream_t)stream) : launch_linear<1, W_MN, X_MN>(x_map, w_map, s, (cudaStream_t)stream);
}

}  // namespace

extern "C" int coset_e8_dense_linear(const void* w_bf16, int n_out, int n_in, const void* x_bf16, int64_t ldx, int T, const float* bias, int round_bias,
                                     void* y, int64_t ldy, int* status, void* stream) {
    if (n_in % 8 != 0) return fail(COSET_E_BADARG, "bad shape (n_in must be a multiple of 8)");
    return dense_product<false, false>(w_bf16, n_in, x_bf16, ldx, n_out, T, n_in, bias, round_bias, y, ldy, status, stream);
}

extern "C" int coset_e8_dense_linear_late(const void* w_bf16, int n_out, int n_in, const void* x_bf16, int T, void* y, int tokens, int split, int late, int* status, void* stream) {
    const int steps = (n_in + BK - 1) / BK;
    if (n_in <= 0 || n_in % 8 != 0 || tokens < 32 || tokens > 256 || tokens % 32 != 0 || (split != 1 && split != 2 && split != 4) || split > steps)
        return fail(COSET_E_BADARG, "no such plan");
    const Plan plan = with_stages(tokens, split, steps);
    return dense_product<false, false>(w_bf16, n_in, x_bf16, n_in, n_out, T, n_in, nullptr, 0, y, n_out, status, stream, &plan, late);
}

extern "C" int coset_dense_input_grad(const void* g_bf16, const void* w_bf16, int T, int n_out, int n_in, void* dx, int* status, void* stream) {
    return dense_product<true, false>(w_bf16, n_in, g_bf16, n_out, n_in, T, n_out, nullptr, 0, dx, n_in, status, stream);
}

extern "C" int coset_dense_weight_grad(const void* g_bf16, const void* x_bf16, int T, int n_out, int n_in, void* dw, int* status, void* stream) {
    return dense_product<true, true>(x_bf16, n_in, g_bf16, n_out, n_in, n_out, T, nullptr, 0, dw, n_in, status, stream);
}
