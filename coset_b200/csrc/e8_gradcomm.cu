// Decode-and-average for the E8-quantised gradient exchange.
//
// Every rank encodes its gradient with one shared scalar scale s (x * s, then q=4, M=2 codes),
// the packed codes are all-gathered into a [W, n_blocks] array in LOCAL memory, and this kernel
// reads the W code streams once and writes
//     out = ( sum_r x_hat_r ) / (s * W)
// The sum of reconstructions is exact (half-integers, accumulated as integers), the divisor
// d = RN(s * W) is formed once in float32 and the quotient is one IEEE division, so a CPU run of
// the same recipe is bit-identical.  No pointer to another GPU's memory is ever dereferenced.
//
// Bytes per block: W * 4 read + 32 written (float32 output).
#include "common.cuh"
#include "e8_fast.cuh"
#include "e8_io.cuh"

using namespace coset;

namespace {

constexpr int kThreads = 256;

// Code streams of the ranks when they are NOT gathered into local memory first: one pointer per
// rank into that rank's own buffer (peer memory, mapped into this process), read with plain loads
// over NVLink.  first = the rank whose stream is read first (each rank starts at a different peer).
constexpr int kMaxPeers = 16;
struct PeerStreams {
    const uint32_t* p[kMaxPeers];
    int first;
};

// One thread owns kPerThread consecutive blocks (1 or 4).  With 4 it requests a 16-byte vector of codes from
// every stream before the first table lookup and writes 128 contiguous bytes; measured on local memory that
// is no faster than one block per thread (0.336 against 0.320 ms for 8 streams of 13.7 M blocks: the kernel
// is bound by the table lookups), so 1 is used.
constexpr int kPerThread = 1;

__device__ __forceinline__ void accumulate_code(uint32_t code, const uint2* __restrict__ table, uint32_t (&acc)[4]) {
    const uint2 t0 = __ldg(table + (code & 0xffffu));
    uint2 t1 = make_uint2(0x07070707u, 0x07070707u);  // all-zero top-level word: zero residual, no lookup
    if (code >> 16) t1 = __ldg(table + (code >> 16));
    const uint32_t lo = t0.x + 4u * t1.x, hi = t0.y + 4u * t1.y;  // biased bytes, each <= 90
    acc[0] += lo & 0x00ff00ffu;
    acc[1] += (lo >> 8) & 0x00ff00ffu;
    acc[2] += hi & 0x00ff00ffu;
    acc[3] += (hi >> 8) & 0x00ff00ffu;
}

template <int DT>
__device__ __forceinline__ void store_mean(const uint32_t (&acc)[4], int world, float divisor, void* __restrict__ out, int64_t b) {
    // 16-bit lanes: acc[0] = coordinates (0,2), acc[1] = (1,3), acc[2] = (4,6), acc[3] = (5,7)
    const int bias = 5 * e8::kTableBias * world;  // every rank contributes 7 + 4*7 to each lane
    int v[8];
    v[0] = (int)(acc[0] & 0xffffu) - bias; v[2] = (int)(acc[0] >> 16) - bias;
    v[1] = (int)(acc[1] & 0xffffu) - bias; v[3] = (int)(acc[1] >> 16) - bias;
    v[4] = (int)(acc[2] & 0xffffu) - bias; v[6] = (int)(acc[2] >> 16) - bias;
    v[5] = (int)(acc[3] & 0xffffu) - bias; v[7] = (int)(acc[3] >> 16) - bias;
    float o[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const float sum = __fmul_rn((float)v[i], 0.5f);  // exact: |v| < 2^16
        o[i] = __fdiv_rn(sum, divisor);
    }
    e8::Row8<DT>::store(out, b, o);
}

template <int DT, bool PEERS>
__global__ void __launch_bounds__(kThreads)
k_decode_mean(const uint32_t* __restrict__ codes, PeerStreams peers, int world, int64_t n, int64_t stride, float divisor,
              const uint2* __restrict__ table, void* __restrict__ out, const int* __restrict__ status) {
    const int64_t b0 = ((int64_t)blockIdx.x * kThreads + threadIdx.x) * kPerThread;
    if (b0 >= n) return;
    // a bounded cross-rank wait before this launch gave up: the peers' streams are not known to be
    // complete, so nothing is read or written
    if (PEERS && status != nullptr && *reinterpret_cast<const volatile int*>(status) != 0) return;
    uint32_t acc[kPerThread][4];
#pragma unroll
    for (int j = 0; j < kPerThread; ++j) acc[j][0] = acc[j][1] = acc[j][2] = acc[j][3] = 0u;
    auto stream_ptr = [&](int r) -> const uint32_t* {
        if (PEERS) {
            int src = peers.first + r;
            if (src >= world) src -= world;
            return peers.p[src] + b0;
        }
        return codes + (int64_t)r * stride + b0;
    };
    // vector path when a stream's 16 bytes at b0 are aligned and inside the tensor; else (odd strides, the
    // tail of the tensor) four scalar loads
    const bool full = b0 + kPerThread <= n;
    for (int r0 = 0; r0 < world; r0 += 4) {
        uint32_t c4[4][kPerThread];
#pragma unroll
        for (int u = 0; u < 4; ++u) {  // up to four streams requested before the first table lookup
#pragma unroll
            for (int j = 0; j < kPerThread; ++j) c4[u][j] = 0u;
            if (r0 + u < world) {
                const uint32_t* p = stream_ptr(r0 + u);
                if (kPerThread == 4 && full && ((reinterpret_cast<uintptr_t>(p) & 15u) == 0)) {
                    const uint4 v = __ldcs(reinterpret_cast<const uint4*>(p));
                    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                    for (int j = 0; j < kPerThread; ++j) c4[u][j] = w[j & 3];
                } else {
#pragma unroll
                    for (int j = 0; j < kPerThread; ++j)
                        if (b0 + j < n) c4[u][j] = __ldcs(p + j);
                }
            }
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            if (r0 + u >= world) break;
#pragma unroll
            for (int j = 0; j < kPerThread; ++j) accumulate_code(c4[u][j], table, acc[j]);
        }
    }
#pragma unroll
    for (int j = 0; j < kPerThread; ++j)
        if (b0 + j < n) store_mean<DT>(acc[j], world, divisor, out, b0 + j);
}

// Up to 16 streams and enough blocks: the residual table sits in shared memory in its compact form and the decoding
// is done on 2-bit fields of two streams at a time.
//
// The kernel above is bound by its table gathers (27 cycles per warp gather; 0.332 ms for 8 streams of 13.7 M blocks
// against 0.134 ms of memory traffic).  Here one CTA of 1024 threads per SM holds the 128 KB table; a code costs one
// 2-byte shared-memory gather and about 14 instructions: the low words of two streams share one register, their
// entries another, and sums of up to four such pairs stay inside 4-bit lanes (4 x 3 = 12), of eight inside bytes.
// Streams beyond `world` are all-zero codes, whose residual is 0.  A block with a non-zero top-level word or a marked
// entry in any stream is summed by the general routine.  The quotient v / (2 d) is formed with one corrected
// multiplication (P. Markstein, IBM J. Res. Dev. 34, 1990): q0 = v r, q = q0 + r (v - 2 d q0) with r = RN(1 / 2 d) equals the IEEE quotient for every float32
// significand and every integer |v| <= 1024 (exhaustive check on the CPU), and |v| <= 16 * 55 here.
constexpr int kCompactThreads = 1024;
constexpr int kCompactMaxWorld = 16;
constexpr int kTableBytes = 65536 * 2;

template <int DT, bool PEERS, int PAIRS>
__global__ void __launch_bounds__(kCompactThreads, 1)
k_decode_mean_compact(const uint32_t* __restrict__ codes, PeerStreams peers, int world, int64_t n, int64_t stride, float twice_divisor,
                      float inverse, const uint16_t* __restrict__ compact, const uint2* __restrict__ table, void* __restrict__ out,
                      const int* __restrict__ status) {
    extern __shared__ uint16_t lut[];
#pragma unroll
    for (int k = 0; k < kTableBytes / 16 / kCompactThreads; ++k)
        reinterpret_cast<uint4*>(lut)[k * kCompactThreads + threadIdx.x] = __ldg(reinterpret_cast<const uint4*>(compact) + k * kCompactThreads + threadIdx.x);
    grid_wait();  // the table is there for good; the streams may come from the kernel before
    grid_trigger();
    if (PEERS && status != nullptr && *reinterpret_cast<const volatile int*>(status) != 0) return;  // see k_decode_mean
    const int64_t step = (int64_t)gridDim.x * kCompactThreads;
    uint32_t next[2 * PAIRS];
    auto fetch = [&](int64_t b) {
#pragma unroll
        for (int r = 0; r < 2 * PAIRS; ++r) {
            next[r] = 0u;
            if (r < world && b < n) {
                if (PEERS) {
                    int src = peers.first + r;
                    if (src >= world) src -= world;
                    next[r] = __ldcs(peers.p[src] + b);
                } else {
                    next[r] = __ldcs(codes + (int64_t)r * stride + b);
                }
            }
        }
    };
    int64_t b = (int64_t)blockIdx.x * kCompactThreads + behind_wait((int)threadIdx.x);
    fetch(b);
    __syncthreads();
    for (; b < n; b += step) {
        uint32_t code[2 * PAIRS];
#pragma unroll
        for (int r = 0; r < 2 * PAIRS; ++r) code[r] = next[r];
        fetch(b + step);
        uint32_t rest = 0u;                                  // non-zero: some stream needs the general routine
        uint32_t t04 = 0u, t26 = 0u, t15 = 0u, t37 = 0u;     // biased sums, one coordinate per byte: (0, 4), (2, 6), ...
#pragma unroll
        for (int p0 = 0; p0 < PAIRS; p0 += 4) {
            uint32_t me = 0u, mo = 0u, se = 0u, so = 0u;
#pragma unroll
            for (int p = p0; p < (p0 + 4 < PAIRS ? p0 + 4 : PAIRS); ++p) {
                const uint32_t w = __byte_perm(code[2 * p], code[2 * p + 1], 0x5410);
                const uint32_t e = (uint32_t)lut[code[2 * p] & 0xffffu] | ((uint32_t)lut[code[2 * p + 1] & 0xffffu] << 16);
                const uint32_t s = e8::compact_residues(w);
                rest |= ((code[2 * p] | code[2 * p + 1]) >> 16) | e8::compact_marked(e);
                me += e & 0x33333333u;
                mo += (e >> 2) & 0x33333333u;
                se += s & 0x33333333u;
                so += (s >> 2) & 0x33333333u;
            }
            auto widen = [](uint32_t m, uint32_t s) {  // 4 m + s per byte, both streams added into the low half
                const uint32_t t = 4u * (m & 0x0f0f0f0fu) + (s & 0x0f0f0f0fu);
                return (t & 0xffffu) + (t >> 16);
            };
            t04 += widen(me, se);
            t26 += widen(me >> 4, se >> 4);
            t15 += widen(mo, so);
            t37 += widen(mo >> 4, so >> 4);
        }
        if (rest == 0u) {
            const float off = 12582912.0f + (float)(2 * PAIRS * e8::kCompactBias), off7 = 12582912.0f + (float)(2 * PAIRS * e8::kCompactBias7);
            float v[8], o[8];
            v[0] = e8::biased_byte_to_float<0>(t04) - off; v[4] = e8::biased_byte_to_float<1>(t04) - off;
            v[2] = e8::biased_byte_to_float<0>(t26) - off; v[6] = e8::biased_byte_to_float<1>(t26) - off;
            v[1] = e8::biased_byte_to_float<0>(t15) - off; v[5] = e8::biased_byte_to_float<1>(t15) - off;
            v[3] = e8::biased_byte_to_float<0>(t37) - off; v[7] = e8::biased_byte_to_float<1>(t37) - off7;
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const float q0 = __fmul_rn(v[i], inverse);
                o[i] = __fmaf_rn(__fmaf_rn(-q0, twice_divisor, v[i]), inverse, q0);
            }
            e8::Row8<DT>::store(out, b, o);
        } else {
            uint32_t acc[4] = {0u, 0u, 0u, 0u};
#pragma unroll
            for (int r = 0; r < 2 * PAIRS; ++r) accumulate_code(code[r], table, acc);
            store_mean<DT>(acc, 2 * PAIRS, __fmul_rn(0.5f, twice_divisor), out, b);
        }
    }
}

// Where the compact kernel is used: it pays ~2 us for the table, so the tensor has to give every thread of the chip
// at least two blocks.
inline bool compact_applies(int world, int64_t n, float divisor) {
    const float a = divisor < 0.0f ? -divisor : divisor;
    return world <= kCompactMaxWorld && n >= 2 * (int64_t)sm_count() * kCompactThreads && a > 1e-18f && a < 1e18f;
}

template <int DT, bool PEERS>
int launch_decode_mean(const uint32_t* codes, const PeerStreams& peers, int world, int64_t n, int64_t stride, float divisor,
                       void* out, const int* status, cudaStream_t st) {
    const uint2* table = residual_table_q4(st);
    const uint16_t* compact = residual_table_q4_compact(st);
    if (!table || !compact) return COSET_E_STATE;
    if (compact_applies(world, n, divisor)) {
        const float twice = 2.0f * divisor, inverse = 1.0f / twice;
#define COMPACT_LAUNCH(PAIRS)                                                                                                       \
    do {                                                                                                                            \
        if (int e = check_cuda(cudaFuncSetAttribute(k_decode_mean_compact<DT, PEERS, PAIRS>, cudaFuncAttributeMaxDynamicSharedMemorySize, kTableBytes), "cudaFuncSetAttribute")) return e; \
        return launch_dependent("e8_decode_mean", k_decode_mean_compact<DT, PEERS, PAIRS>, sm_count(), kCompactThreads, kTableBytes, st, codes, peers, world, n, stride, twice, inverse, compact, table, out, status); \
    } while (0)
        if (world <= 2) COMPACT_LAUNCH(1);
        else if (world <= 4) COMPACT_LAUNCH(2);
        else if (world <= 8) COMPACT_LAUNCH(4);
        else COMPACT_LAUNCH(8);
#undef COMPACT_LAUNCH
    } else {
        const unsigned grid = (unsigned)((n + (int64_t)kThreads * kPerThread - 1) / ((int64_t)kThreads * kPerThread));
        k_decode_mean<DT, PEERS><<<grid, kThreads, 0, st>>>(codes, peers, world, n, stride, divisor, table, out, status);
    }
    return check_launch("e8_decode_mean");
}

}  // namespace

namespace {

// Cross-rank "everyone has arrived" with a bound.  flags[r] is rank r's own array of `world` words
// (peer / symmetric memory, mapped into this process); word s of it is written only by rank s.
// Thread t tells rank t that this rank has reached `epoch` (one release store over NVLink into
// flags[t][rank], after a system-scope fence that publishes everything this rank wrote before the
// launch) and then polls its own flags[rank][t] until rank t has said the same.  Epochs only grow, so
// the words are never cleared and a late reader of an old epoch passes at once.  The poll gives up
// after timeout_ns of the global timer: it records that in *status and returns, and the kernels that
// follow on the stream check *status before touching a peer's data.
struct PeerFlags {
    uint32_t* p[kMaxPeers];
};

__global__ void k_peer_signal_wait(PeerFlags flags, int world, int rank, uint32_t epoch, unsigned long long timeout_ns,
                                   int* __restrict__ status) {
    const int t = threadIdx.x;
    if (t >= world) return;
    __threadfence_system();
    asm volatile("st.release.sys.global.u32 [%0], %1;" ::"l"(flags.p[t] + rank), "r"(epoch) : "memory");
    const uint32_t* mine = flags.p[rank] + t;
    unsigned long long start;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(start));
    for (;;) {
        uint32_t v;
        asm volatile("ld.acquire.sys.global.u32 %0, [%1];" : "=r"(v) : "l"(mine) : "memory");
        if ((int32_t)(v - epoch) >= 0) break;
        unsigned long long now;
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(now));
        if (now - start > timeout_ns) {
            if (status != nullptr) atomicExch(status, 1 + t);  // 1 + the rank that did not arrive
            break;
        }
        __nanosleep(128);
    }
}

}  // namespace

extern "C" int coset_peer_signal_wait(void* const* rank_flags, int world, int rank, uint32_t epoch, int timeout_ms,
                                      int* status, void* stream) {
    if (world < 1 || world > kMaxPeers) return fail(COSET_E_BADARG, "world must be in 1..16");
    if (rank < 0 || rank >= world) return fail(COSET_E_BADARG, "rank outside the world");
    if (!rank_flags) return fail(COSET_E_BADARG, "null pointer");
    PeerFlags f = {};
    for (int r = 0; r < world; ++r) {
        if (!rank_flags[r] || !aligned(rank_flags[r], 4)) return fail(COSET_E_BADARG, "flag array %d is null or misaligned", r);
        f.p[r] = (uint32_t*)rank_flags[r];
    }
    const unsigned long long ns = (unsigned long long)(timeout_ms > 0 ? timeout_ms : 2000) * 1000000ull;
    k_peer_signal_wait<<<1, 32, 0, (cudaStream_t)stream>>>(f, world, rank, epoch, ns, status);
    return check_launch("peer_signal_wait");
}

extern "C" int coset_e8_decode_mean(const void* codes, int world, int64_t n_blocks, int64_t rank_stride_blocks,
                                    float scale, void* out, int out_dtype, void* stream) {
    if (world < 1 || world > 512) return fail(COSET_E_BADARG, "world must be in 1..512");
    if (n_blocks < 0 || rank_stride_blocks < n_blocks) return fail(COSET_E_BADARG, "bad n_blocks / rank stride");
    if (n_blocks == 0) return 0;
    if (!codes || !out) return fail(COSET_E_BADARG, "null pointer");
    if (out_dtype != COSET_DTYPE_F32 && out_dtype != COSET_DTYPE_BF16) return fail(COSET_E_BADARG, "unknown out_dtype");
    if (!aligned(codes, 4) || !aligned(out, 16)) return fail(COSET_E_ALIGN, "codes must be 4-byte and out 16-byte aligned");
    if (!(scale == scale) || scale == 0.0f) return fail(COSET_E_BADARG, "scale must be a non-zero number");
    const float divisor = scale * (float)world;  // one float32 rounding, reproduced by the CPU recipe
    const PeerStreams none = {};
    return (out_dtype == COSET_DTYPE_F32 ? launch_decode_mean<0, false> : launch_decode_mean<1, false>)(
        (const uint32_t*)codes, none, world, n_blocks, rank_stride_blocks, divisor, out, nullptr, (cudaStream_t)stream);
}

extern "C" int coset_e8_decode_mean_peers(const void* const* rank_codes, int world, int rank, int64_t n_blocks, float scale,
                                          void* out, int out_dtype, const int* status, void* stream) {
    if (world < 1 || world > kMaxPeers) return fail(COSET_E_BADARG, "world must be in 1..16 for the peer-memory form");
    if (rank < 0 || rank >= world) return fail(COSET_E_BADARG, "rank outside the world");
    if (n_blocks < 0) return fail(COSET_E_BADARG, "n_blocks is negative");
    if (n_blocks == 0) return 0;
    if (!rank_codes || !out) return fail(COSET_E_BADARG, "null pointer");
    if (out_dtype != COSET_DTYPE_F32 && out_dtype != COSET_DTYPE_BF16) return fail(COSET_E_BADARG, "unknown out_dtype");
    if (!aligned(out, 16)) return fail(COSET_E_ALIGN, "out must be 16-byte aligned");
    if (!(scale == scale) || scale == 0.0f) return fail(COSET_E_BADARG, "scale must be a non-zero number");
    PeerStreams peers = {};
    for (int r = 0; r < world; ++r) {
        if (!rank_codes[r] || !aligned(rank_codes[r], 4)) return fail(COSET_E_BADARG, "code stream %d is null or misaligned", r);
        peers.p[r] = (const uint32_t*)rank_codes[r];
    }
    peers.first = rank;
    const float divisor = scale * (float)world;
    return (out_dtype == COSET_DTYPE_F32 ? launch_decode_mean<0, true> : launch_decode_mean<1, true>)(
        nullptr, peers, world, n_blocks, 0, divisor, out, status, (cudaStream_t)stream);
}
