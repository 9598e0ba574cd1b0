// Dense float32 products of a training layer, small ones: y = x W^T + bias, dx = g W, dW = g^T x, full float32 multiply-adds.
//
// At 128 tokens and 768 features a library product is 15 us of host time and a kernel of 24 to 96 tiles on 148 SMs, for 75 million
// multiply-adds (2 us of the chip).  Here a CTA of 128 threads owns 32 x 64 results and a part of the sum: up to eight CTAs of a cluster
// share K where tiles are few, and add their sums in the order of K through distributed shared memory, every CTA a part of the rows.
// Chains of additions are 64 long and their sums are added apart, so from 32 tokens on the error against 64 bits is no larger than that of the library's
// products (1.0e-7 to 1.8e-7 over sums of 64 to 16384 products, the library's 1.0e-7 to 1.3e-6; chains of 128 had 2.1e-7, and 2.13e-7 against 2.02e-7 in
// the weight gradient of 2048 x 10 x 768; chains of 32 slow the forward product by a fifth).  For fewer tokens the library splits its sums finer (one token,
// 768 x 768: 1.24e-7 against 1.47e-7), and the training layer leaves them to it.
// What bounds a small one is latency (three to six steps of a load from L2 and 32 x 32 x 64 products each), a larger one the two 16-byte reads
// from shared memory per 16 multiply-adds: four rows by four columns per thread.  128 x 768 x 768, torch -> here: forward 17.0 -> 10.4 us, dx 14.6
// -> 10.4, dW 6.1 -> 7.7; 1024 x 512 x 512 19.6 -> 20.8, 15.5 -> 20.5, 19.3 -> 20.5.  Twice as many parts gained nothing; rows read 32 bytes per lane
// with K along the lanes' runs took 12.8 us.
#include "common.cuh"
#include "e8_fast2.cuh"

using namespace coset;

namespace {

constexpr int kM = 32, kN = 64, kK = 32, kThreads = 128;
constexpr int kMostParts = 8;
constexpr int kMostSize = INT32_MAX - 512;
constexpr int kFlush = 2;  // steps of a chain of additions

struct Operands {
    const float* a;  // C[m][n] = sum over k of A(m, k) B(n, k)
    const float* b;
    float* c;
    const float* bias;  // per column, or null
    int M, N, K;
    int parts_log2;
    int wide;  // rows of all operands are made of aligned 16-byte chunks
};

struct Tiles {
    float a[2][kK][kM];
    float b[2][kK][kN];
};
// Where column r of row k of a tile lies: 16-byte chunks exclusive-ored with k / 4, so that eight threads that write four k each of one
// row r meet eight groups of banks.
__device__ __forceinline__ int place(int k, int r) { return r ^ ((k >> 2 & 7) << 2); }

// Four consecutive floats p[0..3], zero where first + i >= limit or the row is not there.
__device__ __forceinline__ float4 load_four(const float* p, bool there, int first, int limit, bool wide) {
    if (wide && there && first + 4 <= limit) return __ldg(reinterpret_cast<const float4*>(p));
    float v[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) v[i] = there && first + i < limit ? __ldg(p + i) : 0.0f;
    return make_float4(v[0], v[1], v[2], v[3]);
}

// One operand's tile of R rows by kK on its way through registers, in fours along the dimension that is contiguous in memory.
template <bool K_MAJOR, int R>
struct Panel {
    static constexpr int kFours = R * kK / 4 / kThreads;
    float4 v[kFours];
    __device__ __forceinline__ void fetch(const float* base, int rows, int row0, int K, int k0, bool wide) {
#pragma unroll
        for (int i = 0; i < kFours; ++i) {
            const int at = i * kThreads + threadIdx.x;
            if (K_MAJOR) {
                const int r = row0 + at / (kK / 4), k = k0 + at % (kK / 4) * 4;
                v[i] = load_four(base + (int64_t)r * K + k, r < rows, k, K, wide);
            } else {
                const int k = k0 + at / (R / 4), r = row0 + at % (R / 4) * 4;
                v[i] = load_four(base + (int64_t)k * rows + r, k < K, r, rows, wide);
            }
        }
    }
    __device__ __forceinline__ void put(float (*tile)[R]) const {
#pragma unroll
        for (int i = 0; i < kFours; ++i) {
            const int at = i * kThreads + threadIdx.x;
            if (K_MAJOR) {
                const int r = at / (kK / 4), k = at % (kK / 4) * 4, p = place(k, r);
                tile[k][p] = v[i].x; tile[k + 1][p] = v[i].y; tile[k + 2][p] = v[i].z; tile[k + 3][p] = v[i].w;
            } else {
                const int k = at / (R / 4), r = at % (R / 4) * 4;
                *reinterpret_cast<float4*>(&tile[k][place(k, r)]) = v[i];
            }
        }
    }
};

__device__ __forceinline__ void sync_cluster() { asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ float4 load_from_rank(const float* here, uint32_t rank) {
    uint32_t addr;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(addr) : "r"((uint32_t)__cvta_generic_to_shared(here)), "r"(rank));
    float4 v;
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
    return v;
}

template <bool A_K, bool B_K>
__global__ void __launch_bounds__(kThreads)
k_f32_product(const __grid_constant__ Operands o) {
    __shared__ __align__(16) Tiles t;
    grid_wait();
    grid_trigger();
    const float *a = behind_wait(o.a), *b = behind_wait(o.b);
    const int parts = 1 << o.parts_log2, part = (int)(blockIdx.x & (parts - 1));
    const int n0 = (int)(blockIdx.x >> o.parts_log2) * kN, m0 = blockIdx.y * kM;
    const int steps = (o.K + kK - 1) / kK, first = (int)((int64_t)steps * part >> o.parts_log2), last = (int)((int64_t)steps * (part + 1) >> o.parts_log2);
    const int tn = threadIdx.x % 16 * 4, tm = threadIdx.x / 16 * 4;
    e8::F2 acc[4][2], total[4][2];
#pragma unroll
    for (int i = 0; i < 4; ++i) acc[i][0] = acc[i][1] = total[i][0] = total[i][1] = e8::pair2(0.0f, 0.0f);
    Panel<A_K, kM> pa;
    Panel<B_K, kN> pb;
    if (first < last) {
        pa.fetch(a, o.M, m0, o.K, first * kK, o.wide);
        pb.fetch(b, o.N, n0, o.K, first * kK, o.wide);
        pa.put(t.a[0]);
        pb.put(t.b[0]);
    }
    __syncthreads();
    for (int s = first; s < last; ++s) {
        const int buffer = (s - first) & 1;
        const bool more = s + 1 < last;
        if (more) {
            pa.fetch(a, o.M, m0, o.K, (s + 1) * kK, o.wide);
            pb.fetch(b, o.N, n0, o.K, (s + 1) * kK, o.wide);
        }
#pragma unroll
        for (int k = 0; k < kK; ++k) {
            const float4 x = *reinterpret_cast<const float4*>(&t.a[buffer][k][place(k, tm)]), w = *reinterpret_cast<const float4*>(&t.b[buffer][k][place(k, tn)]);
            const float xs[4] = {x.x, x.y, x.z, x.w};
            const e8::F2 lo = e8::pair2(w.x, w.y), hi = e8::pair2(w.z, w.w);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const e8::F2 xx = e8::pair2(xs[i], xs[i]);
                acc[i][0] = e8::fma2(xx, lo, acc[i][0]);
                acc[i][1] = e8::fma2(xx, hi, acc[i][1]);
            }
        }
        if (((s - first) & (kFlush - 1)) == kFlush - 1 || !more) {
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    total[i][j] = s - first < kFlush ? acc[i][j] : e8::add2(total[i][j], acc[i][j]);
                    acc[i][j] = e8::pair2(0.0f, 0.0f);
                }
        }
        if (more) {
            pa.put(t.a[buffer ^ 1]);
            pb.put(t.b[buffer ^ 1]);
        }
        __syncthreads();
    }
    float4 out[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        e8::split2(total[i][0], out[i].x, out[i].y);
        e8::split2(total[i][1], out[i].z, out[i].w);
    }
    auto store = [&](int row, int column, float4 v) {
        const int m = m0 + row, n = n0 + column;
        if (m >= o.M) return;
        float r[4] = {v.x, v.y, v.z, v.w};
        float* c = o.c + (int64_t)m * o.N + n;
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (o.bias && n + j < o.N) r[j] += __ldg(behind_wait(o.bias) + n + j);
        if (o.wide && n + 4 <= o.N) *reinterpret_cast<float4*>(c) = make_float4(r[0], r[1], r[2], r[3]);
        else {
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (n + j < o.N) c[j] = r[j];
        }
    };
    if (parts == 1) {
#pragma unroll
        for (int i = 0; i < 4; ++i) store(tm + i, tn, out[i]);
        return;
    }
    float* sums = reinterpret_cast<float*>(&t);  // [kM][kN], over the tiles that nobody reads any more
#pragma unroll
    for (int i = 0; i < 4; ++i) *reinterpret_cast<float4*>(sums + (tm + i) * kN + tn) = out[i];
    sync_cluster();
    const int rows = kM >> o.parts_log2;
    for (int e = threadIdx.x; e < rows * (kN / 4); e += kThreads) {
        const int row = part * rows + e / (kN / 4), column = e % (kN / 4) * 4;
        float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        for (int p = 0; p < parts; ++p) {
            const float4 q = load_from_rank(sums + row * kN + column, (uint32_t)p);
            v.x += q.x; v.y += q.y; v.z += q.z; v.w += q.w;
        }
        store(row, column, v);
    }
    sync_cluster();  // nobody leaves while its sums are read
}

template <bool A_K, bool B_K>
int f32_product(const float* a, const float* b, const float* bias, int M, int N, int K, float* c, void* stream) {
    if (M < 0 || N < 0 || K < 0) return fail(COSET_E_BADARG, "negative size");
    if (M > kMostSize || N > kMostSize || K > kMostSize) return fail(COSET_E_UNSUPPORTED, "sizes are counted in 32 bits, with room for a tile");
    if (M == 0 || N == 0) return 0;
    if (K == 0) return fail(COSET_E_BADARG, "nothing to sum over");
    if (!a || !b || !c) return fail(COSET_E_BADARG, "null pointer");
    if (!aligned(a, 4) || !aligned(b, 4) || !aligned(c, 4) || !aligned(bias, 4)) return fail(COSET_E_ALIGN, "pointers must be 4-byte aligned");
    const int64_t across = (N + kN - 1) / kN, down = (M + kM - 1) / kM, steps = (K + kK - 1) / kK;
    if (down > 65535) return fail(COSET_E_UNSUPPORTED, "too many rows");
    Operands o = {a, b, c, bias, M, N, K, 0, 0};
    // Parts of K: until every SM has two CTAs, with two steps left for each (the loads of one run under the products of the other).
    while ((1 << o.parts_log2) < kMostParts && (across * down << o.parts_log2) < 2 * (int64_t)sm_count() && steps >> (o.parts_log2 + 1) >= 2) ++o.parts_log2;
    o.wide = aligned(a, 16) && aligned(b, 16) && aligned(c, 16) && N % 4 == 0 && (A_K ? K : M) % 4 == 0 && (B_K ? K : N) % 4 == 0;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(across << o.parts_log2), (unsigned)down);
    cfg.blockDim = dim3(kThreads);
    cfg.stream = (cudaStream_t)stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 1u << o.parts_log2;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    return check_cuda(cudaLaunchKernelEx(&cfg, k_f32_product<A_K, B_K>, o), "float32 product");
}

}  // namespace

extern "C" int coset_f32_linear(const float* x, const float* w, const float* bias, int T, int n_out, int n_in, float* y, void* stream) {
    return f32_product<true, true>(x, w, bias, T, n_out, n_in, y, stream);
}
extern "C" int coset_f32_input_grad(const float* g, const float* w, int T, int n_out, int n_in, float* dx, void* stream) {
    return f32_product<true, false>(g, w, nullptr, T, n_in, n_out, dx, stream);
}
extern "C" int coset_f32_weight_grad(const float* g, const float* x, int T, int n_out, int n_in, float* dw, void* stream) {
    return f32_product<false, false>(g, x, nullptr, n_out, n_in, T, dw, stream);
}
