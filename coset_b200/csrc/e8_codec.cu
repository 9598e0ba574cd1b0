// E8 HNLQ codec kernels and their C-ABI entry points: projection, encode, decode, fused
// round trip (quantise), packed <-> float32 digit views, and the q=4 residual table.
//
// One thread owns one 8-vector ("block"): 32 B in (two 128-bit loads, a warp reads 1 KiB
// contiguously), all state in registers, 4 B packed code out.  The kernels are HBM-bound by
// design; algorithmic bytes per block (q=4, M=2, float32): encode 32+4 (+4 per-block scale),
// decode 4+32 (+4), round trip 32+32 (+4).
#include <stdarg.h>

#include <mutex>

#include "common.cuh"
#include "e8_fast.cuh"
#include "e8_fast2.cuh"
#include "e8_io.cuh"
#include "e8_literal.cuh"

namespace coset {

static thread_local char g_err[512] = "";

int fail(int code, const char* fmt, ...) {
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(g_err, sizeof(g_err), fmt, ap);
    va_end(ap);
    return code;
}
int check_cuda(cudaError_t e, const char* what) {
    if (e == cudaSuccess) return 0;
    return fail((int)e, "%s: %s", what, cudaGetErrorString(e));
}
int check_launch(const char* what) { return check_cuda(cudaGetLastError(), what); }

int sm_count() {
    static int cached[64] = {0};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 148;
    if (cached[dev] == 0) {
        int n = 0;
        if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 148;
        cached[dev] = n;
    }
    return cached[dev];
}

}  // namespace coset

using namespace coset;

namespace {

constexpr int kThreads = 256;

// one divisor as a kernel argument instead of a device pointer (the digit entry points)
constexpr int kScaleDivValue = 3;

template <int MODE>
__device__ __forceinline__ float scale_in(float v, float s) {
    if (MODE == COSET_SCALE_DIV_SCALAR || MODE == kScaleDivValue) return __fdiv_rn(v, s);
    if (MODE == COSET_SCALE_MUL_TILE) return __fmul_rn(v, s);
    return v;
}
template <int MODE>
__device__ __forceinline__ float scale_out(float v, float s) {
    if (MODE == COSET_SCALE_DIV_SCALAR) return __fmul_rn(v, s);
    if (MODE == COSET_SCALE_MUL_TILE) return __fdiv_rn(v, s);
    return v;
}
// a row times its scale, in pairs
template <int MODE>
__device__ __forceinline__ void scale_row(float (&v)[8], float s) {
    if (MODE == COSET_SCALE_MUL_TILE) {
#pragma unroll
        for (int i = 0; i < 4; ++i) e8::split2(e8::mul2(e8::pair2(v[2 * i], v[2 * i + 1]), e8::pair2(s, s)), v[2 * i], v[2 * i + 1]);
    } else {
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] = scale_in<MODE>(v[i], s);
    }
}
template <int MODE>
__device__ __forceinline__ float load_scale(const float* scale, const e8::TileDiv& td, int64_t block) {
    if (MODE == COSET_SCALE_DIV_SCALAR) return __ldg(scale);
    if (MODE == COSET_SCALE_MUL_TILE) {
        // per-block scales are streamed once; per-row scales are reused by the whole row
        return td.divisor == 1 ? __ldcs(scale + block) : __ldg(scale + e8::tile_of(td, block));
    }
    return 1.0f;
}

__device__ __forceinline__ float clampf(float v, float clip) {
    // torch.clamp: NaN stays NaN
    if (clip > 0.0f) v = (v < -clip) ? -clip : ((v > clip) ? clip : v);
    return v;
}

// ---------------------------------------------------------------- projection
__global__ void __launch_bounds__(kThreads) k_projection(const float* __restrict__ x, int64_t n, float* __restrict__ y) {
    int64_t b = (int64_t)blockIdx.x * kThreads + threadIdx.x;
    if (b >= n) return;
    float v[8], o[8];
    e8::Row8<0>::load(x, b, v);
    e8::projection(v, o);
    e8::Row8<0>::store(y, b, o);
}

// ---------------------------------------------------------------- generic (any 2<=q<=16, M<=8)
// e8_encode, coset/core/e8/codecs.py:63-83: x_l starts as the scaled input and is divided by q
// after every level (cumulative IEEE divisions, no re-quantisation).
template <int BPD>
__device__ __forceinline__ void encode_levels_generic(float (&xl)[8], int q, int M, uint32_t* words) {
    float qf = (float)q;
    for (int m = 0; m < M; ++m) {
        float y[8];
        int d[8];
        bool half = e8::projection(xl, y);
        e8::encode_coords(y, half, q, d);
        words[m] = e8::pack_level<BPD>(d);
#pragma unroll
        for (int i = 0; i < 8; ++i) xl[i] = __fdiv_rn(xl[i], qf);
    }
}

// E8Decoder._full_decode, coset/core/e8/codecs.py:159-172 (before the final scale).
template <int BPD>
__device__ __forceinline__ void decode_levels_generic(const uint32_t* words, int q, int M, float (&xh)[8]) {
    float qf = (float)q, w = 1.0f;
#pragma unroll
    for (int i = 0; i < 8; ++i) xh[i] = 0.0f;
    for (int m = 0; m < M; ++m) {
        int d[8];
        float r[8];
        e8::unpack_level<BPD>(words[m], d);
        e8::level_residual(d, qf, r);
#pragma unroll
        for (int i = 0; i < 8; ++i) xh[i] = __fadd_rn(xh[i], __fmul_rn(w, r[i]));
        w = __fmul_rn(w, qf);
    }
}

template <int BPD>
struct LevelWord;
template <>
struct LevelWord<2> { typedef uint16_t type; };
template <>
struct LevelWord<4> { typedef uint32_t type; };

template <int DT, int MODE, int BPD>
__global__ void __launch_bounds__(kThreads)
k_encode_generic(const void* __restrict__ x, const float* __restrict__ scale, e8::TileDiv td, int64_t n, int q,
                 int M, void* __restrict__ codes) {
    int64_t b = (int64_t)blockIdx.x * kThreads + threadIdx.x;
    if (b >= n) return;
    float v[8];
    e8::Row8<DT>::load(x, b, v);
    float s = load_scale<MODE>(scale, td, b);
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = scale_in<MODE>(v[i], s);
    uint32_t words[8];
    encode_levels_generic<BPD>(v, q, M, words);
    typename LevelWord<BPD>::type* out = reinterpret_cast<typename LevelWord<BPD>::type*>(codes) + b * M;
    for (int m = 0; m < M; ++m) out[m] = (typename LevelWord<BPD>::type)words[m];
}

template <int DT, int MODE, int BPD>
__global__ void __launch_bounds__(kThreads)
k_decode_generic(const void* __restrict__ codes, const float* __restrict__ scale, e8::TileDiv td, int64_t n, int q,
                 int M, void* __restrict__ out) {
    int64_t b = (int64_t)blockIdx.x * kThreads + threadIdx.x;
    if (b >= n) return;
    const typename LevelWord<BPD>::type* in = reinterpret_cast<const typename LevelWord<BPD>::type*>(codes) + b * M;
    uint32_t words[8];
    for (int m = 0; m < M; ++m) words[m] = in[m];
    float xh[8];
    decode_levels_generic<BPD>(words, q, M, xh);
    float s = load_scale<MODE>(scale, td, b);
#pragma unroll
    for (int i = 0; i < 8; ++i) xh[i] = scale_out<MODE>(xh[i], s);
    e8::Row8<DT>::store(out, b, xh);
}

template <int DTI, int DTO, int MODE, int BPD>
__global__ void __launch_bounds__(kThreads)
k_quantize_generic(const void* __restrict__ x, const float* __restrict__ scale, e8::TileDiv td, int64_t n, int q,
                   int M, float clip, void* __restrict__ out, void* __restrict__ codes) {
    int64_t b = (int64_t)blockIdx.x * kThreads + threadIdx.x;
    if (b >= n) return;
    float v[8];
    e8::Row8<DTI>::load(x, b, v);
    float s = load_scale<MODE>(scale, td, b);
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = scale_in<MODE>(v[i], s);
    uint32_t words[8];
    encode_levels_generic<BPD>(v, q, M, words);
    if (codes) {
        typename LevelWord<BPD>::type* co = reinterpret_cast<typename LevelWord<BPD>::type*>(codes) + b * M;
        for (int m = 0; m < M; ++m) co[m] = (typename LevelWord<BPD>::type)words[m];
    }
    float xh[8];
    decode_levels_generic<BPD>(words, q, M, xh);
#pragma unroll
    for (int i = 0; i < 8; ++i) xh[i] = clampf(scale_out<MODE>(xh[i], s), clip);
    e8::Row8<DTO>::store(out, b, xh);
}

// ---------------------------------------------------------------- q = 4, M = 2 (one uint32 per block)
template <int DT, int MODE, bool LITERAL>
__global__ void __launch_bounds__(kThreads, 6)
k_encode_q4m2(const void* __restrict__ x, const float* __restrict__ scale, e8::TileDiv td, int64_t n,
              uint32_t* __restrict__ codes) {
    int64_t b = (int64_t)blockIdx.x * kThreads + threadIdx.x;
    if (b >= n) return;
    float v[8];
    e8::Row8<DT>::load(x, b, v);
    float s = load_scale<MODE>(scale, td, b);
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = scale_in<MODE>(v[i], s);
    __stcs(codes + b, e8::encode_q4m2<LITERAL>(v));
}

// Queued encoder: the fused round trip and the digits of q=4, M=2 (codes alone: k_encode_q4m2_listed below).
//
// Warps are persistent; one loop iteration of a warp covers ROWS * 32 consecutive blocks,
// one row per lane and sub-step.  Every lane runs the cheapest tier (level_fast2_q4: one rounding
// pass, both cosets from it, digits on the FP32 pipe) behind one pre-test, max|x| <= 1.96 and
// sum|x| <= 7.96, which makes the top level the origin and bounds every quantity of that tier.
// Whatever the tier cannot prove -- a block near a rounding tie, a block whose top level is not the
// origin, a non-finite block -- is NOT handled in place (that would idle the other 31 lanes for
// hundreds of instructions): the lane appends the block's index to a per-warp queue in shared memory
// (a shared-memory atomic hands out the slot, so no warp-wide vote sits on the common path).  Once
// per iteration the warp looks at the queue length; with 32 or more entries (and at the end) it
// drains 32 of them with all lanes busy: every lane reads the row of its entry again -- one memory
// round trip per 32 deferred blocks -- and encodes it from scratch with the always-valid tiers.
// This also serves an overloaded quantiser, where most blocks need the top level: the queue then
// fills every iteration and is drained by full warps.
constexpr int kEncWarps = kThreads / 32;

// Rows per lane and iteration of the encoders: three keep the loads of the later rows behind the arithmetic of the
// earlier ones (four at 85 registers and 3 CTAs per SM were 5 % slower); one where three would leave resident CTAs of the
// chip without work (digits of 65536 blocks 6.7 -> 5.5 us, a [768, 768] layer's weights 7.1 -> 5.8).  The grid gives every
// warp an iteration, with at most kEncCtasPerSm CTAs per SM for three rows and the four resident ones for one.
constexpr int kEncCtasPerSm = 12;
inline unsigned encoder_grid(int64_t n_blocks, int* rows) {
    const int64_t sms = sm_count(), need3 = (n_blocks + 3 * kThreads - 1) / (3 * kThreads), need1 = (n_blocks + kThreads - 1) / kThreads;
    *rows = need3 >= 4 * sms ? 3 : 1;
    const int64_t need = *rows == 3 ? need3 : need1, cap = (*rows == 3 ? kEncCtasPerSm : 4) * sms;
    return (unsigned)(need < cap ? (need < 1 ? 1 : need) : cap);
}

// KIND = kRecon: the fused round trip -- every finished code is decoded through the residual table, unscaled,
// clamped and written as [n, 8] of type DTO; the packed code is stored only if `codes` is not null (e8_quantize /
// the layer's weight path).  KIND = kDigits: the code is written as the reference's float32 digits [n, 2, 8].
// `value` is the divisor of MODE == kScaleDivValue and the clamp otherwise.
constexpr int kRecon = 0, kDigits = 1;

__device__ __forceinline__ void store_digits(float* __restrict__ digits, int64_t row, uint32_t word) {
    int d[8];
    float f[8];
    e8::unpack_level<2>(word, d);
#pragma unroll
    for (int i = 0; i < 8; ++i) f[i] = (float)d[i];
    e8::Row8<0>::store(digits, row, f);
}

template <int DT, int MODE, int KIND, int DTO, int ROWS>
__global__ void __launch_bounds__(kThreads, 4)
k_encode_q4m2_queued(const void* __restrict__ x, const float* __restrict__ scale, e8::TileDiv td, int64_t n,
                     uint32_t* __restrict__ codes, const uint2* __restrict__ table, void* __restrict__ out, float value) {
    constexpr int kQueueSlots = 32 * (ROWS + 1);  // < 32 left after a drain + at most 32 per sub-step
    __shared__ uint32_t q_index[kEncWarps][2][kQueueSlots];  // block index lo / hi
    __shared__ int q_count[kEncWarps];
    if ((threadIdx.x & 31) == 0) q_count[threadIdx.x >> 5] = 0;
    __syncwarp();
    grid_wait();
    grid_trigger();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    auto emit = [&](int64_t b, uint32_t code, float s) {
        if constexpr (KIND == kDigits) {
            store_digits((float*)out, 2 * b, code & 0xffffu);
            store_digits((float*)out, 2 * b + 1, code >> 16);
        } else {
            if (codes) __stcs(codes + b, code);
            float v2[8], xh[8];
            e8::decode_q4m2_twice(code, table, v2);
            e8::scale_twice<MODE>(v2, s, xh);
#pragma unroll
            for (int i = 0; i < 8; ++i) xh[i] = clampf(xh[i], value);
            e8::Row8<DTO>::store(out, b, xh);
        }
    };
    auto scale_of = [&](int64_t b) { return MODE == kScaleDivValue ? value : load_scale<MODE>(scale, td, b); };
    int count = 0;  // warp-uniform copy of q_count[warp] as of the last look

    // Completes the last min(count, 32) queued blocks with all lanes busy.
    auto drain = [&]() {
        const int take = count < 32 ? count : 32;
        if (lane < take) {
            const int e = count - take + lane;
            const int64_t b = (int64_t)(((uint64_t)q_index[warp][1][e] << 32) | q_index[warp][0][e]);
            float v[8];
            e8::Row8<DT>::load(x, b, v);
            const float s = scale_of(b);
#pragma unroll
            for (int i = 0; i < 8; ++i) v[i] = scale_in<MODE>(v[i], s);
            emit(b, e8::finish_block_q4(v, 0u, 0), s);
        }
        count -= take;
        __syncwarp();
        if (lane == 0) q_count[warp] = count;
        __syncwarp();
    };

    const int64_t span = 32 * ROWS;
    const int64_t stride = (int64_t)gridDim.x * kEncWarps * span;
    for (int64_t base = ((int64_t)blockIdx.x * kEncWarps + warp) * span; base < n; base += stride) {
        bool defer[ROWS];
        bool any_defer = false;
        {
            // All rows are requested first; the tier then runs row after row in straight-line code, so
            // the loads of the later rows overlap the arithmetic of the earlier ones.  The rows are not
            // kept beyond this scope.
            float v[ROWS][8];
            float sc[ROWS];
#pragma unroll
            for (int j = 0; j < ROWS; ++j) {
                const int64_t b = base + j * 32 + lane;
                sc[j] = 1.0f;
                if (b < n) {
                    e8::Row8<DT>::load(x, b, v[j]);
                    sc[j] = scale_of(b);
                } else {
#pragma unroll
                    for (int i = 0; i < 8; ++i) v[j][i] = 0.0f;
                }
            }
#pragma unroll
            for (int j = 0; j < ROWS; ++j) {
                const int64_t b = base + j * 32 + lane;
                float s1 = 0.0f;
                scale_row<MODE>(v[j], sc[j]);
#pragma unroll
                for (int i = 0; i < 8; ++i) s1 += fabsf(v[j][i]);
                // max |x_i| as a tree of three-input maxima; a NaN is dropped by fmaxf but poisons s1
                const float m0 = fmaxf(fmaxf(fabsf(v[j][0]), fabsf(v[j][1])), fabsf(v[j][2]));
                const float m1 = fmaxf(fmaxf(fabsf(v[j][3]), fabsf(v[j][4])), fabsf(v[j][5]));
                const float amax = fmaxf(fmaxf(m0, m1), fmaxf(fabsf(v[j][6]), fabsf(v[j][7])));
                const bool pre = amax <= 1.96f && s1 <= 7.96f;       // top level is the origin, tier applicable
                const bool origin = amax <= 0.49f && s1 <= 1.99f;    // this level is the origin too: code 0
                uint32_t code;
                const bool proven = e8::level_fast2_q4(v[j], code);
                const bool done = origin || (pre && proven);
                defer[j] = b < n && !done;
                if (b < n && done) emit(b, origin ? 0u : code, sc[j]);
                any_defer = any_defer || defer[j];
            }
        }
        if (any_defer) {  // rare: one branch per iteration keeps the queue code off the common path
#pragma unroll
            for (int j = 0; j < ROWS; ++j) {
                if (defer[j]) {
                    const int64_t b = base + j * 32 + lane;
                    const int pos = atomicAdd(&q_count[warp], 1);
                    q_index[warp][0][pos] = (uint32_t)b;
                    q_index[warp][1][pos] = (uint32_t)((uint64_t)b >> 32);
                }
            }
        }
        __syncwarp();
        count = *reinterpret_cast<volatile int*>(&q_count[warp]);
        while (count >= 32) drain();
    }
    while (count > 0) drain();
}

// ---------------------------------------------------------------- encode-only production path
// The codes-only encoder.  Any state carried across the loop in registers (a queue length, a vote per iteration, a second
// loop) costs 10-25 % of its time through register pressure at the 64-register budget, so the loop carries none: a lane
// whose block the cheapest tier cannot prove puts the block's index on a list of its CTA in shared memory, in a rare
// branch, and after its loop the CTA finishes the listed blocks with all lanes busy, while other CTAs of the SM are still
// in their loops.  A CTA with more such blocks than its list holds (an overloaded quantiser) stores a marker code instead
// (top level word non-zero, which the cheapest tier never produces) and sweeps its own codes for the marker.
// Measured against a list in global memory that a second launch finished: a lane then waited for the return of a global
// atomic (27 % of the warps of the benchmark data did) and the second launch took 10 us at any size.
constexpr uint32_t kDeferredMark = 0x80000000u;
constexpr int kListCap = 1024;  // the benchmark data defers 1 % of the 19000 blocks of a CTA

// One level by the tiers that accept every block.  amax, s1: max and sum of |x_i|.
__device__ __forceinline__ uint32_t level_exact_q4(const float (&x)[8], float amax, float s1) {
    return e8::level_slow_q4(x, s1 == s1 && s1 - s1 == 0.0f ? amax : __int_as_float(0x7fc00000));
}
// One level of a deferred block: the cheapest tier when it applies, then the exact-rounding tier, then the
// literal search.
__device__ __forceinline__ uint32_t level_any_q4(const float (&x)[8], float amax, float s1, const uint4* rows) {
    uint32_t digits;
    if (amax <= 1.96f && s1 <= 7.96f && e8::level_fast2_q4(x, digits, rows)) return digits;
    return level_exact_q4(x, amax, s1);
}

// SAT: every scaled coordinate is first clamped to +-kSaturate, which keeps the two-level code from wrapping around (the top level
// stays the origin); only deferred blocks can exceed the bound, so the clamp costs nothing on the common path.
constexpr float kSaturate = 3.9f;  // 8 * 3.9 / 4 < 7.96 and 3.9 / 4 < 1.96: level 1 of a clamped block is the origin

// How a block's scale is found: any MODE by the general rule, one block per scale, or by a division that fits 32 bits.
constexpr int kAnyScale = 0, kBlockScale = 1, kTileScale = 2;

// kRing > 0: rows on their way to shared memory per thread (cp.async), so that the loop waits for no load and holds one row in
// registers.  What bounds the loop is then the issue of instructions (82 % of the cycles, ALU pipe 63 %, FMA pipe 39 % over 2^24 blocks; with three rows
// per iteration in registers 77, 72 and 33 % over 2^25), hence offsets of 32 bits (n < 2^27 blocks, the caller cuts longer calls), a form
// for each kind of scale, and the signs at the flip coordinates read from the row by index.  The two halves of a float32 row lie in the
// order of bit 2 of the thread, so that eight lanes meet eight groups of banks; they come through L1, whose lines both halves share.
// Measured against the form with registers: 2^25 float32 blocks with a scale each 298 -> 271 us, with one scale for 96 blocks 317 -> 290,
// bf16 342 -> 291; 13.7 M blocks with one scale 136 -> 120; 10^6 bf16 blocks 18.9 -> 13.7.  Three rows under way were 2 % slower, five
// CTAs per SM (48 registers) 3-4 %.
// kRing = 0: straight from global memory, for calls in which a thread has a block or two (65536 blocks 4.2 us, through the ring 4.9).
constexpr int kRowsUnderWay = 2;

__device__ __forceinline__ void copy_async_if(bool go, uint32_t dst, const void* src) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %0, 0;\n\t@p cp.async.ca.shared.global [%1], [%2], 16;\n\t}" ::"r"((uint32_t)go), "r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void copy_async_if(bool go, uint32_t dst, uint32_t dst_next, const void* src) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %0, 0;\n\t@p cp.async.ca.shared.global [%1], [%3], 16;\n\t@p cp.async.ca.shared.global [%2], [%3 + 16], 16;\n\t}"
                 ::"r"((uint32_t)go), "r"(dst), "r"(dst_next), "l"(src) : "memory");
}
__device__ __forceinline__ void copy_word_async_if(bool go, uint32_t dst, const void* src) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %0, 0;\n\t@p cp.async.ca.shared.global [%1], [%2], 4;\n\t}" ::"r"((uint32_t)go), "r"(dst), "l"(src) : "memory");
}

// n < 2^27; scale: of block 0, which is block `skip` of its tile (kTileScale).
template <int DT, int MODE, bool SAT, int SCALES, int kRing>
__global__ void __launch_bounds__(kThreads, 4)
k_encode_q4m2_listed(const void* __restrict__ x, const float* __restrict__ scale, e8::TileDiv td, uint32_t skip, uint32_t n, uint32_t* codes) {
    constexpr int kRowBytes = DT == 0 ? 32 : 16, kSlots = kRing > 0 ? kRing : 1;
    __shared__ __align__(16) uint8_t ring[kSlots][kThreads][kRowBytes];
    __shared__ float ring_scale[SCALES == kBlockScale ? kSlots : 1][kThreads];
    __shared__ uint4 flip_rows[8];
    __shared__ uint32_t list[kListCap];
    __shared__ uint32_t listed;
    static_assert(sizeof(ring) >= kEncWarps * 64 * sizeof(uint32_t), "the sweep's queue fits the idle ring");
    if (threadIdx.x < 8) flip_rows[threadIdx.x] = e8::kFlipRows[threadIdx.x];
    if (threadIdx.x == 0) listed = 0u;
    __syncthreads();
    grid_wait();
    grid_trigger();
    const uint32_t stride = gridDim.x * kThreads, first = blockIdx.x * kThreads + threadIdx.x;
    auto scale_of = [&](uint32_t b) -> float {
        if (SCALES == kBlockScale) return __ldcs(scale + b);
        if (SCALES == kTileScale) return __ldg(scale + (__umulhi(skip + b, td.mul) >> td.shr));
        return load_scale<MODE>(scale, td, b);
    };
    // The code of a block by the cheapest tier, or a place on the list; `between` runs once the block has been read.
    auto encode = [&](uint32_t b, const float (&v)[8], auto fetch, auto between) {
        float s1 = 0.0f;
#pragma unroll
        for (int i = 0; i < 8; ++i) s1 += fabsf(v[i]);
        // max |x_i| as a tree of three-input maxima; a NaN is dropped by fmaxf but poisons s1
        const float m0 = fmaxf(fmaxf(fabsf(v[0]), fabsf(v[1])), fabsf(v[2]));
        const float m1 = fmaxf(fmaxf(fabsf(v[3]), fabsf(v[4])), fabsf(v[5]));
        const float amax = fmaxf(fmaxf(m0, m1), fmaxf(fabsf(v[6]), fabsf(v[7])));
        const bool pre = amax <= 1.96f && s1 <= 7.96f;     // top level is the origin, tier applicable
        const bool origin = amax <= 0.49f && s1 <= 1.99f;  // this level is the origin too: code 0
        uint32_t code;
        const bool proven = e8::level_fast2_q4(v, code, flip_rows, fetch);
        between();
        if (b < n) {
            if (origin || (pre && proven)) {
                __stcs(reinterpret_cast<uint32_t*>(reinterpret_cast<uint8_t*>(codes) + (uint64_t)(b * 4u)), origin ? 0u : code);
            } else {  // rare
                const uint32_t pos = atomicAdd(&listed, 1u);
                if (pos < (uint32_t)kListCap) list[pos] = b;
                else codes[b] = kDeferredMark;
            }
        }
    };
    if constexpr (kRing > 0) {
        const uint32_t row_at = (uint32_t)__cvta_generic_to_shared(&ring[0][threadIdx.x][0]), scale_at = (uint32_t)__cvta_generic_to_shared(&ring_scale[0][threadIdx.x]);
        const uint32_t flip = DT == 0 ? (threadIdx.x & 4u) * 4u : 0u;  // 16: the halves change places
        auto request = [&](uint32_t b, int slot) {
            const uint8_t* src = reinterpret_cast<const uint8_t*>(x) + (uint64_t)(b * (uint32_t)kRowBytes);
            const uint32_t dst = row_at + (uint32_t)(slot * kThreads * kRowBytes);
            if (DT == 0) copy_async_if(b < n, dst + flip, dst + (flip ^ 16u), src);
            else copy_async_if(b < n, dst, src);
            if (SCALES == kBlockScale) copy_word_async_if(b < n, scale_at + (uint32_t)(slot * kThreads * 4), reinterpret_cast<const uint8_t*>(scale) + (uint64_t)(b * 4u));
            asm volatile("cp.async.commit_group;" ::: "memory");
        };
#pragma unroll
        for (int k = 0; k < kRing; ++k) request(first + k * stride, k);
        for (uint32_t base = first; base < n; base += kRing * stride) {
#pragma unroll
            for (int k = 0; k < kRing; ++k) {
                const uint32_t b = base + k * stride;
                const float direct = SCALES != kBlockScale && b < n ? scale_of(b) : 1.0f;
                asm volatile("cp.async.wait_group %0;" ::"n"(kRing - 1) : "memory");
                const uint8_t* row = &ring[k][threadIdx.x][0];
                float v[8];
                if (DT == 0) {
                    const float4 lo = *reinterpret_cast<const float4*>(row + flip), hi = *reinterpret_cast<const float4*>(row + (flip ^ 16u));
                    v[0] = lo.x; v[1] = lo.y; v[2] = lo.z; v[3] = lo.w; v[4] = hi.x; v[5] = hi.y; v[6] = hi.z; v[7] = hi.w;
                } else {
                    const uint4 r = *reinterpret_cast<const uint4*>(row);
                    const uint32_t w[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        v[2 * i] = __uint_as_float(w[i] << 16);
                        v[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
                    }
                }
                const float sc = SCALES == kBlockScale ? ring_scale[k][threadIdx.x] : direct;
                scale_row<MODE>(v, sc);
                const auto coordinate = [&](uint32_t i) {
                    const float r = DT == 0 ? *reinterpret_cast<const float*>(row + ((i * 4u) ^ flip))
                                            : __uint_as_float((uint32_t)*reinterpret_cast<const uint16_t*>(row + i * 2u) << 16);
                    return scale_in<MODE>(r, sc);
                };
                encode(b, v, coordinate, [&]() { request(b + kRing * stride, k); });
            }
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
    } else {
        for (uint32_t b = first; b < n; b += stride) {
            float v[8];
            e8::Row8<DT>::load(x, b, v);
            scale_row<MODE>(v, scale_of(b));
            encode(b, v, e8::NoFetch(), []() {});
        }
    }
    auto finish = [&](uint32_t b) {
        float v[8];
        e8::Row8<DT>::load(x, b, v);
        const float s = scale_of(b);
        float amax = 0.0f, s1 = 0.0f;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            v[i] = scale_in<MODE>(v[i], s);
            if (SAT) v[i] = fminf(fmaxf(v[i], -kSaturate), kSaturate);  // a NaN becomes -kSaturate: finite, harmless
            amax = fmaxf(amax, fabsf(v[i]));
            s1 += fabsf(v[i]);
        }
        uint32_t code = 0u;
#pragma unroll 1
        for (int m = 0; m < 2; ++m) {
            const bool origin = amax <= 0.49f && s1 <= 1.99f;
            // the cheapest tier has refused level 0 as it is
            if (!origin) code |= (m > 0 ? level_any_q4(v, amax, s1, flip_rows) : level_exact_q4(v, amax, s1)) << (16 * m);
#pragma unroll
            for (int i = 0; i < 8; ++i) v[i] = __fmul_rn(v[i], 0.25f);
            amax *= 0.25f;
            s1 *= 0.25f;
        }
        __stcs(codes + b, code);
    };
    __syncthreads();  // the list is complete and the markers of this CTA are visible to it
    const uint32_t total = listed;
    if (total > (uint32_t)kListCap) {
        // every warp reads the codes that it wrote, 32 marked blocks at a time.  A listed block whose old content happens to
        // be the marker is finished twice, with the same result; the sweep is over before the list is worked off, whose
        // results may equal the marker.
        int count = 0;
        const int lane = threadIdx.x & 31;
        uint32_t* queue = reinterpret_cast<uint32_t*>(&ring[0][0][0]) + (threadIdx.x >> 5) * 64;
        auto drain = [&](int take) {
            if (lane < take) finish(queue[count - take + lane]);
            count -= take;
            __syncwarp();
        };
        for (uint32_t base = first - lane; base < n; base += stride) {
            const uint32_t b = base + lane;
            const bool marked = b < n && codes[b] == kDeferredMark;
            const uint32_t bal = __ballot_sync(0xffffffffu, marked);
            if (bal) {
                if (marked) queue[count + __popc(bal & ((1u << lane) - 1u))] = b;
                count += __popc(bal);
                __syncwarp();
                if (count >= 32) drain(32);
            }
        }
        if (count > 0) drain(count);
        __syncthreads();
    }
    for (uint32_t e = threadIdx.x; e < total && e < (uint32_t)kListCap; e += kThreads) finish(list[e]);
}

// Four blocks per thread (kThreads apart, so every access stays coalesced): all codes are
// loaded before the first table lookup, which multiplies the gathers in flight per thread
// (measured per 2^25 blocks: 2 per thread 0.236 ms, 4 per thread 0.231 ms, 8 per thread 0.231 ms).
constexpr int kDecPerThread = 4;
// TABLE is `uint2` (8-byte entries) or `uint32_t` (packed 4-byte entries, used for float32 output,
// where the kernel is bound by the gathers and not by instruction issue).
template <int DT, int MODE, typename TABLE>
__global__ void __launch_bounds__(kThreads)
k_decode_q4m2(const uint32_t* __restrict__ codes, const float* __restrict__ scale, e8::TileDiv td, int64_t n,
              const TABLE* __restrict__ table, void* __restrict__ out) {
    grid_wait();
    grid_trigger();
    const int64_t base = (int64_t)blockIdx.x * (kThreads * kDecPerThread) + behind_wait((int)threadIdx.x);
    if (MODE == COSET_SCALE_DIV_SCALAR) scale = behind_wait(scale);
    uint32_t code[kDecPerThread];
    float s[kDecPerThread];
#pragma unroll
    for (int j = 0; j < kDecPerThread; ++j) {
        int64_t b = base + j * kThreads;
        code[j] = b < n ? __ldcs(codes + b) : 0u;
        s[j] = b < n ? load_scale<MODE>(scale, td, b) : 1.0f;
    }
#pragma unroll
    for (int j = 0; j < kDecPerThread; ++j) {
        int64_t b = base + j * kThreads;
        if (b < n) {
            float v2[8], xh[8];
            e8::decode_q4m2_twice(code[j], table, v2);
            e8::scale_twice<MODE>(v2, s[j], xh);
            e8::Row8<DT>::store(out, b, xh);
        }
    }
}

// Many blocks: the residual table in its compact form in shared memory, one CTA of 1024 threads per SM (see e8::compact_residues).
//
// What bounds the kernel above is the gathers, 27 cycles per warp for 32 lines of L1 and L2, the more so in bf16, whose rows are half as long.
// A gather from shared memory costs the conflicts of 32 banks, both levels of a code share the arithmetic on 2-bit fields, and everything on
// eight coordinates is done in pairs.  The table is loaded before grid_wait: it is there for good, and the kernel before still drains.
// Rows requested ahead per thread: two float32 rows, next to each other across the CTA; four bf16 rows, far apart.  Measured, from the kernel above
// (one scale per block): float32 400000 blocks 8.1 -> 6.2 us, 10^6 13.9 -> 9.8, 4 M 35.6 -> 28.4, 2^25 222 -> 217, but 200000 4.2 -> 4.4; bf16 10^6 6.9 -> 6.7 (one scale
// for 96 blocks 7.7 -> 6.7, 2^25 160 -> 143), but 700000 4.8 -> 5.4.  Four float32 rows far apart took 267 us for 2^25, two bf16 rows 167.
constexpr int kSharedThreads = 1024;
template <int DT>
constexpr int kSharedRows = DT == 0 ? 2 : 4;
inline int64_t shared_decoder_from(int out_dtype) { return (out_dtype == COSET_DTYPE_F32 ? 2 : 6) * (int64_t)sm_count() * kSharedThreads; }
constexpr int kSharedTableBytes = 65536 * 2;

template <int MODE>
__device__ __forceinline__ void scale_twice_pairs(const float (&v2)[8], float s, float (&out)[8]) {
    const float a = fabsf(s);
    if (MODE == COSET_SCALE_MUL_TILE && a > 1e-18f && a < 1e18f) {  // scale_twice, in pairs
        const float s2 = __fmul_rn(s, 2.0f), r = __frcp_rn(s2);
        const e8::F2 rr = e8::pair2(r, r), ss = e8::pair2(-s2, -s2);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const e8::F2 v = e8::pair2(v2[2 * i], v2[2 * i + 1]), q = e8::mul2(v, rr);
            e8::split2(e8::fma2(e8::fma2(q, ss, v), rr, q), out[2 * i], out[2 * i + 1]);
        }
    } else {
        e8::scale_twice<MODE>(v2, s, out);
    }
}

template <int DT, int MODE, int SCALES>
__global__ void __launch_bounds__(kSharedThreads, 1)
k_decode_q4m2_shared(const uint32_t* __restrict__ codes, const float* __restrict__ scale, e8::TileDiv td, uint32_t skip, uint32_t n, const uint16_t* __restrict__ compact,
                     const uint2* __restrict__ table, void* __restrict__ out) {
    extern __shared__ __align__(16) uint16_t lut[];
#pragma unroll
    for (int k = 0; k < kSharedTableBytes / 16 / kSharedThreads; ++k)
        reinterpret_cast<uint4*>(lut)[k * kSharedThreads + threadIdx.x] = __ldg(reinterpret_cast<const uint4*>(compact) + k * kSharedThreads + threadIdx.x);
    grid_wait();
    grid_trigger();
    constexpr int kRows = kSharedRows<DT>;
    const uint32_t round = gridDim.x * kSharedThreads * kRows, stride = DT == 0 ? (uint32_t)kSharedThreads : gridDim.x * kSharedThreads;
    const uint32_t first = blockIdx.x * kSharedThreads * (DT == 0 ? kRows : 1) + (uint32_t)behind_wait((int)threadIdx.x);
    const float one = MODE == COSET_SCALE_DIV_SCALAR ? __ldg(behind_wait(scale)) : 1.0f;
    uint32_t next[kRows];
    float next_scale[kRows];
    auto request = [&](uint32_t b, int j) {
        next[j] = 0u;
        next_scale[j] = one;
        if (b < n) {
            next[j] = __ldcs(reinterpret_cast<const uint32_t*>(reinterpret_cast<const uint8_t*>(codes) + (uint64_t)(b * 4u)));
            if (SCALES == kBlockScale) next_scale[j] = __ldcs(reinterpret_cast<const float*>(reinterpret_cast<const uint8_t*>(scale) + (uint64_t)(b * 4u)));
            if (SCALES == kTileScale) next_scale[j] = __ldg(scale + (__umulhi(skip + b, td.mul) >> td.shr));
        }
    };
#pragma unroll
    for (int j = 0; j < kRows; ++j) request(first + j * stride, j);
    __syncthreads();
    for (uint32_t base = first; base < n; base += round) {
#pragma unroll
        for (int j = 0; j < kRows; ++j) {
            const uint32_t b = base + j * stride;
            const uint32_t code = next[j];
            const float s = next_scale[j];
            request(b + round, j);
            if (b >= n) continue;
            const uint32_t e = (uint32_t)lut[code & 0xffffu] | ((uint32_t)lut[code >> 16] << 16), r = e8::compact_residues(code);
            float v2[8], xh[8];
            if (e8::compact_marked(e) == 0u) {
                // nibbles 4 m + s: coordinates 0, 2, 4, 6 and 1, 3, 5, 7 of level 0, and of level 1 in the upper half
                const uint32_t even = ((e & 0x33333333u) << 2) | (r & 0x33333333u), odd = (e & 0xccccccccu) | ((r >> 2) & 0x33333333u);
                auto levels = [](uint32_t t) { return t + 4u * (t >> 16); };  // bytes 0 and 1
                const uint32_t t04 = levels(even & 0x0f0f0f0fu), t26 = levels((even >> 4) & 0x0f0f0f0fu);
                const uint32_t t15 = levels(odd & 0x0f0f0f0fu), t37 = levels((odd >> 4) & 0x0f0f0f0fu);
                const float off = -(12582912.0f + 5.0f * e8::kCompactBias), off7 = -(12582912.0f + 5.0f * e8::kCompactBias7);
                const e8::F2 o = e8::pair2(off, off);
                e8::split2(e8::add2(e8::pair2(e8::biased_byte_to_float<0>(t04), e8::biased_byte_to_float<0>(t15)), o), v2[0], v2[1]);
                e8::split2(e8::add2(e8::pair2(e8::biased_byte_to_float<0>(t26), e8::biased_byte_to_float<0>(t37)), o), v2[2], v2[3]);
                e8::split2(e8::add2(e8::pair2(e8::biased_byte_to_float<1>(t04), e8::biased_byte_to_float<1>(t15)), o), v2[4], v2[5]);
                e8::split2(e8::add2(e8::pair2(e8::biased_byte_to_float<1>(t26), e8::biased_byte_to_float<1>(t37)), e8::pair2(off, off7)), v2[6], v2[7]);
            } else {
                e8::decode_q4m2_twice(code, table, v2);
            }
            scale_twice_pairs<MODE>(v2, s, xh);
            e8::Row8<DT>::store(reinterpret_cast<uint8_t*>(out) + (uint64_t)(b * (DT == 0 ? 32u : 16u)), 0, xh);
        }
    }
}

// Residual table of the q=4 decoder, produced by the literal float32 decoder itself:
// entry[w] = 2 * (G b - 4 Q(G b / 4)) + 7 for the 16-bit level word w, as 8 unsigned bytes.
__global__ void k_build_table_q4(uint2* __restrict__ table, uint32_t* __restrict__ packed, uint16_t* __restrict__ compact, int* __restrict__ bad) {
    int w = blockIdx.x * blockDim.x + threadIdx.x;
    if (w >= 65536) return;
    int d[8];
    float r[8];
    e8::unpack_level<2>((uint32_t)w, d);
    e8::level_residual(d, 4.0f, r);
    uint32_t lo = 0, hi = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        lo |= ((uint32_t)((__float2int_rn(__fmul_rn(r[i], 2.0f)) + e8::kTableBias) & 0xff)) << (8 * i);
        hi |= ((uint32_t)((__float2int_rn(__fmul_rn(r[i + 4], 2.0f)) + e8::kTableBias) & 0xff)) << (8 * i);
    }
    table[w] = make_uint2(lo, hi);
    // packed entry (layout at e8::biased_bytes_q4m2); `bad` counts residuals that do not fit it
    int t[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) t[i] = __float2int_rn(__fmul_rn(r[i], 2.0f));
    const int p = t[0] & 1;
    uint32_t e = (uint32_t)p << 31;
    bool ok = true;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int nib = (t[i] - p + (i < 7 ? e8::kNibbleBias : e8::kNibbleBias7)) >> 1;
        ok = ok && ((t[i] & 1) == p) && nib >= 0 && nib <= (i < 7 ? 15 : 7);
        e |= ((uint32_t)nib & 0xfu) << (4 * i);
    }
    packed[w] = e;
    // compact entry (layout at e8::compact_residues)
    const uint32_t res = e8::compact_residues((uint32_t)w);
    uint32_t fields = 0;
    bool marked = false;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int diff = t[i] + (i < 7 ? e8::kCompactBias : e8::kCompactBias7) - (int)((res >> (2 * i)) & 3u);
        const int m = diff >> 2;
        ok = ok && (diff & 3) == 0 && m >= 0 && m <= (i < 7 ? 4 : 2);
        marked = marked || m == 4;
        fields |= (uint32_t)(m & 3) << (2 * i);
    }
    compact[w] = (uint16_t)(marked ? fields | 0xc000u : fields);
    if (!ok) atomicAdd(bad, 1);
}

// ---------------------------------------------------------------- digit views
template <int BPD>
__global__ void __launch_bounds__(kThreads)
k_unpack_f32(const void* __restrict__ codes, int64_t n_words, float* __restrict__ digits) {
    int64_t i = (int64_t)blockIdx.x * kThreads + threadIdx.x;  // one level word per thread
    if (i >= n_words) return;
    uint32_t w = reinterpret_cast<const typename LevelWord<BPD>::type*>(codes)[i];
    int d[8];
    float f[8];
    e8::unpack_level<BPD>(w, d);
#pragma unroll
    for (int j = 0; j < 8; ++j) f[j] = (float)d[j];
    e8::Row8<0>::store(digits, i, f);
}

template <int BPD>
__global__ void __launch_bounds__(kThreads)
k_pack_f32(const float* __restrict__ digits, int64_t n_words, int q, void* __restrict__ codes) {
    int64_t i = (int64_t)blockIdx.x * kThreads + threadIdx.x;
    if (i >= n_words) return;
    float f[8];
    int d[8];
    e8::Row8<0>::load(digits, i, f);
#pragma unroll
    for (int j = 0; j < 8; ++j) d[j] = e8::floored_mod(__float2int_rn(f[j]), q);
    reinterpret_cast<typename LevelWord<BPD>::type*>(codes)[i] = (typename LevelWord<BPD>::type)e8::pack_level<BPD>(d);
}

// Digits of any (q, M) from the literal search, and values from digits: what coset_e8_encode / _decode do with packed
// codes in between, without the packed array (4 launches and 72 bytes per block less for q = 4, M = 2).
__global__ void __launch_bounds__(kThreads)
k_encode_digits_generic(const float* __restrict__ x, float beta, int64_t n, int q, int M, float* __restrict__ digits) {
    grid_wait();
    grid_trigger();
    const int64_t b = (int64_t)blockIdx.x * kThreads + behind_wait((int)threadIdx.x);
    if (b >= n) return;
    float xl[8];
    e8::Row8<0>::load(x, b, xl);
#pragma unroll
    for (int i = 0; i < 8; ++i) xl[i] = __fdiv_rn(xl[i], beta);
    const float qf = (float)q;
    for (int m = 0; m < M; ++m) {
        float y[8], f[8];
        int d[8];
        const bool half = e8::projection(xl, y);
        e8::encode_coords(y, half, q, d);
#pragma unroll
        for (int i = 0; i < 8; ++i) f[i] = (float)d[i];
        e8::Row8<0>::store(digits, b * M + m, f);
#pragma unroll
        for (int i = 0; i < 8; ++i) xl[i] = __fdiv_rn(xl[i], qf);
    }
}

// Q4: the residual of a level comes from the table; the sum over the levels is exact in float32 (multiples of 1/2
// below 2^18), so its order does not matter.
template <bool Q4>
__global__ void __launch_bounds__(kThreads)
k_decode_digits(const float* __restrict__ digits, float beta, int64_t n, int q, int M, const uint2* __restrict__ table, float* __restrict__ out) {
    grid_wait();
    grid_trigger();
    const int64_t b = (int64_t)blockIdx.x * kThreads + behind_wait((int)threadIdx.x);
    if (b >= n) return;
    float xh[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) xh[i] = 0.0f;
    const float qf = (float)q;
    float w = 1.0f;
    for (int m = 0; m < M; ++m) {
        float f[8], r[8];
        int d[8];
        e8::Row8<0>::load(digits, b * M + m, f);
        if (Q4) {
#pragma unroll
            for (int j = 0; j < 8; ++j) d[j] = __float2int_rn(f[j]) & 3;
            const uint2 t = __ldg(table + e8::pack_level<2>(d));
            const uint32_t tw[2] = {t.x, t.y};
#pragma unroll
            for (int j = 0; j < 8; ++j) r[j] = 0.5f * (float)((int)((tw[j >> 2] >> (8 * (j & 3))) & 0xffu) - e8::kTableBias);
        } else {
#pragma unroll
            for (int j = 0; j < 8; ++j) d[j] = e8::floored_mod(__float2int_rn(f[j]), q);
            e8::level_residual(d, qf, r);
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) xh[i] = __fadd_rn(xh[i], __fmul_rn(w, r[i]));
        w = __fmul_rn(w, qf);
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) xh[i] = __fmul_rn(xh[i], beta);
    e8::Row8<0>::store(out, b, xh);
}

inline unsigned grid_for(int64_t n) { return (unsigned)((n + kThreads - 1) / kThreads); }

int check_common(const void* a, const void* b, int64_t n_blocks, int q, int M) {
    if (n_blocks < 0) return fail(COSET_E_BADARG, "n_blocks is negative");
    if (n_blocks > 0 && (!a || !b)) return fail(COSET_E_BADARG, "null data pointer");
    if (q < 2 || q > 16 || M < 1 || M > 8) return fail(COSET_E_UNSUPPORTED, "unsupported q=%d M=%d (need 2<=q<=16, 1<=M<=8)", q, M);
    if ((int64_t)grid_for(n_blocks) != (n_blocks + kThreads - 1) / kThreads || n_blocks > ((int64_t)1 << 38))
        return fail(COSET_E_BADARG, "n_blocks too large");
    return 0;
}
int check_scale(const float* scale, int mode, int64_t bpt) {
    if (mode < 0 || mode > 2) return fail(COSET_E_BADARG, "unknown scale_mode %d", mode);
    if (mode != COSET_SCALE_NONE && !scale) return fail(COSET_E_BADARG, "scale is null");
    if (mode == COSET_SCALE_MUL_TILE && bpt < 1) return fail(COSET_E_BADARG, "blocks_per_tile must be >= 1");
    return 0;
}

}  // namespace

namespace coset {

const uint2* residual_table_q4(cudaStream_t stream) {
    static std::mutex mu;
    static uint2* tables[64] = {nullptr};
    int dev = 0;
    if (check_cuda(cudaGetDevice(&dev), "cudaGetDevice")) return nullptr;
    if (dev < 0 || dev >= 64) { fail(COSET_E_STATE, "device index %d out of range", dev); return nullptr; }
    std::lock_guard<std::mutex> lock(mu);
    if (!tables[dev]) {
        uint2* t = nullptr;  // 65536 x 8 B, then 65536 x 4 B packed, 65536 x 2 B compact, the builder's self-check word
        if (check_cuda(cudaMalloc(&t, 65536 * (sizeof(uint2) + sizeof(uint32_t) + sizeof(uint16_t)) + 16), "cudaMalloc(residual table)")) return nullptr;
        uint32_t* packed = reinterpret_cast<uint32_t*>(t + 65536);
        uint16_t* compact = reinterpret_cast<uint16_t*>(packed + 65536);
        int* bad = reinterpret_cast<int*>(compact + 65536);
        int bad_host = -1;
        // Built on the caller's stream: every later use on any stream must see it complete, so
        // the one-time build synchronises that stream.
        bool failed = check_cuda(cudaMemsetAsync(bad, 0, sizeof(int), stream), "table build") != 0;
        if (!failed) {
            k_build_table_q4<<<65536 / 256, 256, 0, stream>>>(t, packed, compact, bad);
            failed = check_launch("k_build_table_q4") ||
                     check_cuda(cudaMemcpyAsync(&bad_host, bad, sizeof(int), cudaMemcpyDeviceToHost, stream), "table build") ||
                     check_cuda(cudaStreamSynchronize(stream), "table build");
        }
        if (!failed && bad_host != 0) {
            fail(COSET_E_STATE, "residual table: %d entries do not fit the packed layouts", bad_host);
            failed = true;
        }
        if (failed) {
            cudaFree(t);
            return nullptr;
        }
        tables[dev] = t;
    }
    return tables[dev];
}

const uint32_t* residual_table_q4_packed(cudaStream_t stream) {
    const uint2* t = residual_table_q4(stream);
    return t ? reinterpret_cast<const uint32_t*>(t + 65536) : nullptr;
}

const uint16_t* residual_table_q4_compact(cudaStream_t stream) {
    const uint32_t* p = residual_table_q4_packed(stream);
    return p ? reinterpret_cast<const uint16_t*>(p + 65536) : nullptr;
}

}  // namespace coset

namespace {

// A call in parts whose offsets fit 32 bits: fn(first block, blocks, scale of the first block, division of kTileScale, its place in its tile).
template <int MODE, typename Fn>
int in_parts(const float* scale, const e8::TileDiv& td, int64_t n, Fn fn) {
    constexpr int64_t kMost = 1 << 26, kLongTile = 1 << 30;
    const int64_t tile = MODE == COSET_SCALE_MUL_TILE ? td.divisor : 1;
    for (int64_t at = 0; at < n;) {
        int64_t count = n - at < kMost ? n - at : kMost, skip = at % tile;
        const float* s = scale;
        e8::TileDiv part = {};
        if (MODE == COSET_SCALE_MUL_TILE) {
            s += at / tile;
            if (tile > kLongTile) {  // the part ends with its tile: the quotient of the empty division is 0
                count = count < tile - skip ? count : tile - skip;
                skip = 0;
            } else if (tile > 1) {
                part = e8::make_tile_div(tile, kLongTile + kMost);
            }
        }
        if (int rc = fn(at, count, s, part, (uint32_t)skip)) return rc;
        at += count;
    }
    return 0;
}

template <int DT, int MODE, bool SAT>
int launch_encode_q4m2(const void* x, const float* scale, e8::TileDiv td, int64_t n, uint32_t* codes, cudaStream_t st) {
    const int64_t resident = 4 * (int64_t)sm_count();
    if (n < 3 * resident * kThreads) {  // a thread has at most three blocks
        const int64_t need = (n + kThreads - 1) / kThreads;
        return launch_dependent("e8_encode", k_encode_q4m2_listed<DT, MODE, SAT, kAnyScale, 0>, (unsigned)(need < resident ? need : resident), kThreads, 0, st,
                                x, scale, td, 0u, (uint32_t)n, codes);
    }
    return in_parts<MODE>(scale, td, n, [&](int64_t at, int64_t count, const float* s, e8::TileDiv part, uint32_t skip) {
        // Up to 32 blocks per thread of the resident CTAs, these alone, each with one pass over its list; beyond, three CTAs follow one another, so that
        // the lists of the first are worked off while others are in their loops (4.2 M blocks 47 us against 52, 13.7 M 124 against 120).
        const int64_t need = (count + kThreads - 1) / kThreads, cap = need <= 32 * resident ? resident : 3 * resident;
        const unsigned grid = (unsigned)(need < cap ? need : cap);
        const void* xs = (const uint8_t*)x + at * (DT == 0 ? 32 : 16);
        auto go = [&](auto kernel) { return launch_dependent("e8_encode", kernel, grid, kThreads, 0, st, xs, s, part, skip, (uint32_t)count, codes + at); };
        if constexpr (MODE != COSET_SCALE_MUL_TILE) return go(k_encode_q4m2_listed<DT, MODE, SAT, kAnyScale, kRowsUnderWay>);
        else return td.divisor == 1 ? go(k_encode_q4m2_listed<DT, MODE, SAT, kBlockScale, kRowsUnderWay>) : go(k_encode_q4m2_listed<DT, MODE, SAT, kTileScale, kRowsUnderWay>);
    });
}

// The decoder with the table in shared memory.
template <int DT, int MODE>
int launch_decode_shared(const uint32_t* codes, const float* scale, e8::TileDiv td, int64_t n, const uint16_t* compact, const uint2* table, void* out, cudaStream_t st) {
    return in_parts<MODE>(scale, td, n, [&](int64_t at, int64_t count, const float* s, e8::TileDiv part, uint32_t skip) {
        auto go = [&](auto kernel) {
            if (int e = check_cuda(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSharedTableBytes), "cudaFuncSetAttribute")) return e;
            return launch_dependent("e8_decode", kernel, (unsigned)sm_count(), kSharedThreads, kSharedTableBytes, st, codes + at, s, part, skip, (uint32_t)count, compact, table,
                                    (void*)((uint8_t*)out + at * (DT == 0 ? 32 : 16)));
        };
        if constexpr (MODE != COSET_SCALE_MUL_TILE) return go(k_decode_q4m2_shared<DT, MODE, kAnyScale>);
        else return td.divisor == 1 ? go(k_decode_q4m2_shared<DT, MODE, kBlockScale>) : go(k_decode_q4m2_shared<DT, MODE, kTileScale>);
    });
}

}  // namespace

#define DISPATCH_MODE(MODE_VAR, ...)                                   \
    switch (MODE_VAR) {                                                \
        case 0: { constexpr int MODE = 0; __VA_ARGS__; } break;         \
        case 1: { constexpr int MODE = 1; __VA_ARGS__; } break;         \
        default: { constexpr int MODE = 2; __VA_ARGS__; } break;        \
    }
#define DISPATCH_DT(DT_VAR, NAME, ...)                                 \
    if ((DT_VAR) == COSET_DTYPE_F32) { constexpr int NAME = 0; __VA_ARGS__; } else { constexpr int NAME = 1; __VA_ARGS__; }

extern "C" {

int coset_version(void) { return 100; }
const char* coset_last_error_string(void) { return coset::g_err; }

int coset_e8_code_bytes(int q, int M) {
    if (q < 2 || q > 16 || M < 1 || M > 8) return 0;
    return M * (q <= 4 ? 2 : 4);
}

int coset_e8_projection(const float* x, int64_t n_blocks, float* y, void* stream) {
    if (int e = check_common(x, y, n_blocks, 4, 2)) return e;
    if (n_blocks == 0) return 0;
    if (!aligned(x, 16) || !aligned(y, 16)) return fail(COSET_E_ALIGN, "x and y must be 16-byte aligned");
    k_projection<<<grid_for(n_blocks), kThreads, 0, (cudaStream_t)stream>>>(x, n_blocks, y);
    return check_launch("k_projection");
}

int coset_e8_encode(const void* x, int x_dtype, const float* scale, int scale_mode, int64_t n_blocks,
                    int64_t blocks_per_tile, int q, int M, int sem, void* codes, void* stream) {
    if (int e = check_common(x, codes, n_blocks, q, M)) return e;
    if (int e = check_scale(scale, scale_mode, blocks_per_tile)) return e;
    if (x_dtype != COSET_DTYPE_F32 && x_dtype != COSET_DTYPE_BF16) return fail(COSET_E_BADARG, "unknown x_dtype %d", x_dtype);
    if (sem != COSET_SEM_CORE && sem != COSET_SEM_CORE_LITERAL && sem != COSET_SEM_CORE_SATURATE)
        return fail(COSET_E_UNSUPPORTED, "semantics %d not available in this entry point", sem);
    if (sem == COSET_SEM_CORE_SATURATE && !(q == 4 && M == 2)) return fail(COSET_E_UNSUPPORTED, "saturating encode needs q=4, M=2");
    if (n_blocks == 0) return 0;
    if (!aligned(x, 16) || !aligned(codes, 4)) return fail(COSET_E_ALIGN, "x must be 16-byte and codes 4-byte aligned");
    cudaStream_t st = (cudaStream_t)stream;
    e8::TileDiv td = e8::make_tile_div(scale_mode == COSET_SCALE_MUL_TILE ? blocks_per_tile : 1, n_blocks);
    unsigned grid = grid_for(n_blocks);
    if (q == 4 && M == 2 && sem == COSET_SEM_CORE) {
        int rc = 0;
        DISPATCH_DT(x_dtype, DT, DISPATCH_MODE(scale_mode, (rc = launch_encode_q4m2<DT, MODE, false>(x, scale, td, n_blocks, (uint32_t*)codes, st))))
        return rc;
    } else if (q == 4 && M == 2 && sem == COSET_SEM_CORE_SATURATE) {
        int rc = 0;
        DISPATCH_DT(x_dtype, DT, DISPATCH_MODE(scale_mode, (rc = launch_encode_q4m2<DT, MODE, true>(x, scale, td, n_blocks, (uint32_t*)codes, st))))
        return rc;
    } else if (q == 4 && M == 2) {
        DISPATCH_DT(x_dtype, DT, DISPATCH_MODE(scale_mode, (k_encode_q4m2<DT, MODE, true><<<grid, kThreads, 0, st>>>(x, scale, td, n_blocks, (uint32_t*)codes))))
    } else if (q <= 4) {
        DISPATCH_DT(x_dtype, DT, DISPATCH_MODE(scale_mode, (k_encode_generic<DT, MODE, 2><<<grid, kThreads, 0, st>>>(x, scale, td, n_blocks, q, M, codes))))
    } else {
        DISPATCH_DT(x_dtype, DT, DISPATCH_MODE(scale_mode, (k_encode_generic<DT, MODE, 4><<<grid, kThreads, 0, st>>>(x, scale, td, n_blocks, q, M, codes))))
    }
    return check_launch("e8_encode");
}

int coset_e8_decode(const void* codes, const float* scale, int scale_mode, int64_t n_blocks, int64_t blocks_per_tile,
                    int q, int M, int sem, void* out, int out_dtype, void* stream) {
    if (int e = check_common(codes, out, n_blocks, q, M)) return e;
    if (int e = check_scale(scale, scale_mode, blocks_per_tile)) return e;
    if (out_dtype != COSET_DTYPE_F32 && out_dtype != COSET_DTYPE_BF16) return fail(COSET_E_BADARG, "unknown out_dtype %d", out_dtype);
    if (sem != COSET_SEM_CORE) return fail(COSET_E_UNSUPPORTED, "semantics %d not available in this entry point", sem);
    if (n_blocks == 0) return 0;
    if (!aligned(out, 16) || !aligned(codes, 4)) return fail(COSET_E_ALIGN, "out must be 16-byte and codes 4-byte aligned");
    cudaStream_t st = (cudaStream_t)stream;
    e8::TileDiv td = e8::make_tile_div(scale_mode == COSET_SCALE_MUL_TILE ? blocks_per_tile : 1, n_blocks);
    unsigned grid = grid_for(n_blocks);
    if (q == 4 && M == 2) {
        const uint2* table = residual_table_q4(st);
        const uint32_t* packed = residual_table_q4_packed(st);
        if (!table || !packed) return COSET_E_STATE;
        int rc = 0;
        if (n_blocks >= shared_decoder_from(out_dtype)) {
            const uint16_t* compact = residual_table_q4_compact(st);
            DISPATCH_DT(out_dtype, DT, DISPATCH_MODE(scale_mode, (rc = launch_decode_shared<DT, MODE>((const uint32_t*)codes, scale, td, n_blocks, compact, table, out, st))))
            return rc;
        }
        unsigned grid2 = (unsigned)((n_blocks + kThreads * kDecPerThread - 1) / (kThreads * kDecPerThread));
        if (out_dtype == COSET_DTYPE_F32) {
            DISPATCH_MODE(scale_mode, (rc = launch_dependent("e8_decode", k_decode_q4m2<0, MODE, uint32_t>, grid2, kThreads, 0, st, (const uint32_t*)codes, scale, td, n_blocks, packed, out)))
        } else {
            DISPATCH_MODE(scale_mode, (rc = launch_dependent("e8_decode", k_decode_q4m2<1, MODE, uint2>, grid2, kThreads, 0, st, (const uint32_t*)codes, scale, td, n_blocks, table, out)))
        }
        return rc;
    } else if (q <= 4) {
        DISPATCH_DT(out_dtype, DT, DISPATCH_MODE(scale_mode, (k_decode_generic<DT, MODE, 2><<<grid, kThreads, 0, st>>>(codes, scale, td, n_blocks, q, M, out))))
    } else {
        DISPATCH_DT(out_dtype, DT, DISPATCH_MODE(scale_mode, (k_decode_generic<DT, MODE, 4><<<grid, kThreads, 0, st>>>(codes, scale, td, n_blocks, q, M, out))))
    }
    return check_launch("e8_decode");
}

int coset_e8_quantize(const void* x, int x_dtype, const float* scale, int scale_mode, int64_t n_blocks,
                      int64_t blocks_per_tile, int q, int M, float clip, void* out, int out_dtype, void* codes_out,
                      void* stream) {
    if (int e = check_common(x, out, n_blocks, q, M)) return e;
    if (int e = check_scale(scale, scale_mode, blocks_per_tile)) return e;
    if ((x_dtype != 0 && x_dtype != 1) || (out_dtype != 0 && out_dtype != 1)) return fail(COSET_E_BADARG, "unknown dtype");
    if (n_blocks == 0) return 0;
    if (!aligned(x, 16) || !aligned(out, 16) || !aligned(codes_out, 4)) return fail(COSET_E_ALIGN, "x/out must be 16-byte and codes 4-byte aligned");
    cudaStream_t st = (cudaStream_t)stream;
    e8::TileDiv td = e8::make_tile_div(scale_mode == COSET_SCALE_MUL_TILE ? blocks_per_tile : 1, n_blocks);
    unsigned grid = grid_for(n_blocks);
    if (q == 4 && M == 2) {
        const uint2* table = residual_table_q4(st);
        if (!table) return COSET_E_STATE;
        int rows;
        const unsigned qgrid = encoder_grid(n_blocks, &rows);
        int rc = 0;
        DISPATCH_DT(x_dtype, DTI, DISPATCH_DT(out_dtype, DTO, DISPATCH_MODE(scale_mode, (rc = launch_dependent("e8_quantize", rows == 3 ? k_encode_q4m2_queued<DTI, MODE, kRecon, DTO, 3> : k_encode_q4m2_queued<DTI, MODE, kRecon, DTO, 1>, qgrid, kThreads, 0, st, x, scale, td, n_blocks, (uint32_t*)codes_out, table, out, clip)))))
        return rc;
    } else if (q <= 4) {
        DISPATCH_DT(x_dtype, DTI, DISPATCH_DT(out_dtype, DTO, DISPATCH_MODE(scale_mode, (k_quantize_generic<DTI, DTO, MODE, 2><<<grid, kThreads, 0, st>>>(x, scale, td, n_blocks, q, M, clip, out, codes_out)))))
    } else {
        DISPATCH_DT(x_dtype, DTI, DISPATCH_DT(out_dtype, DTO, DISPATCH_MODE(scale_mode, (k_quantize_generic<DTI, DTO, MODE, 4><<<grid, kThreads, 0, st>>>(x, scale, td, n_blocks, q, M, clip, out, codes_out)))))
    }
    return check_launch("e8_quantize");
}

int coset_e8_unpack_codes_f32(const void* codes, int64_t n_blocks, int q, int M, float* digits, void* stream) {
    if (int e = check_common(codes, digits, n_blocks, q, M)) return e;
    if (n_blocks == 0) return 0;
    if (!aligned(digits, 16)) return fail(COSET_E_ALIGN, "digits must be 16-byte aligned");
    int64_t nw = n_blocks * M;
    if (q <= 4) k_unpack_f32<2><<<grid_for(nw), kThreads, 0, (cudaStream_t)stream>>>(codes, nw, digits);
    else k_unpack_f32<4><<<grid_for(nw), kThreads, 0, (cudaStream_t)stream>>>(codes, nw, digits);
    return check_launch("e8_unpack_codes_f32");
}

int coset_e8_pack_codes_f32(const float* digits, int64_t n_blocks, int q, int M, void* codes, void* stream) {
    if (int e = check_common(digits, codes, n_blocks, q, M)) return e;
    if (n_blocks == 0) return 0;
    if (!aligned(digits, 16)) return fail(COSET_E_ALIGN, "digits must be 16-byte aligned");
    int64_t nw = n_blocks * M;
    if (q <= 4) k_pack_f32<2><<<grid_for(nw), kThreads, 0, (cudaStream_t)stream>>>(digits, nw, q, codes);
    else k_pack_f32<4><<<grid_for(nw), kThreads, 0, (cudaStream_t)stream>>>(digits, nw, q, codes);
    return check_launch("e8_pack_codes_f32");
}

int coset_e8_encode_digits_f32(const float* x, float beta, int64_t n_blocks, int q, int M, float* digits, void* stream) {
    if (int e = check_common(x, digits, n_blocks, q, M)) return e;
    if (n_blocks == 0) return 0;
    if (!aligned(x, 16) || !aligned(digits, 16)) return fail(COSET_E_ALIGN, "x and digits must be 16-byte aligned");
    cudaStream_t st = (cudaStream_t)stream;
    if (q == 4 && M == 2) {
        const e8::TileDiv td = e8::make_tile_div(1, n_blocks);
        int rows;
        const unsigned grid = encoder_grid(n_blocks, &rows);
        // two rows where the rule says three: with three, 104 bytes of registers spill (2^20 blocks 60 -> 54 us, both calls)
#define DIGITS_AS(MODE, ROWS) return launch_dependent("e8_encode_digits_f32", k_encode_q4m2_queued<0, MODE, kDigits, 0, ROWS>, grid, kThreads, 0, st, (const void*)x, (const float*)nullptr, td, n_blocks, (uint32_t*)nullptr, (const uint2*)nullptr, (void*)digits, beta)
        if (beta == 1.0f) {  // x / 1 is x
            if (rows == 3) DIGITS_AS(COSET_SCALE_NONE, 2);
            DIGITS_AS(COSET_SCALE_NONE, 1);
        }
        if (rows == 3) DIGITS_AS(kScaleDivValue, 2);
        DIGITS_AS(kScaleDivValue, 1);
#undef DIGITS_AS
    }
    return launch_dependent("e8_encode_digits_f32", k_encode_digits_generic, grid_for(n_blocks), kThreads, 0, st, x, beta, n_blocks, q, M, digits);
}

int coset_e8_decode_digits_f32(const float* digits, float beta, int64_t n_blocks, int q, int M, float* out, void* stream) {
    if (int e = check_common(digits, out, n_blocks, q, M)) return e;
    if (n_blocks == 0) return 0;
    if (!aligned(digits, 16) || !aligned(out, 16)) return fail(COSET_E_ALIGN, "digits and out must be 16-byte aligned");
    cudaStream_t st = (cudaStream_t)stream;
    if (q == 4) {
        const uint2* table = residual_table_q4(st);
        if (!table) return COSET_E_STATE;
        return launch_dependent("e8_decode_digits_f32", k_decode_digits<true>, grid_for(n_blocks), kThreads, 0, st, digits, beta, n_blocks, q, M, table, out);
    }
    return launch_dependent("e8_decode_digits_f32", k_decode_digits<false>, grid_for(n_blocks), kThreads, 0, st, digits, beta, n_blocks, q, M, (const uint2*)nullptr, out);
}

}  // extern "C"
