// The residual stream between two sublayers in one pass over each row: the previous sublayer's output (summed over
// its parts) is normalised and added, the new stream normalised for the next sublayer.  The stream and everything
// computed here is fp32; a CTA has one row at a time in registers, 8 elements per access.
//
// Bound by DRAM for prompts, by its chain of reductions for few rows: one barrier per sum.  What keeps rows in flight is the number of
// CTAs that the registers allow (rn_resident), and where CTAs walk rows a ring in shared memory (residual_norm_launch): the next row in
// registers instead, half as many CTAs, made eight parts of 4096 columns 211 us instead of 167.
#include <type_traits>

#include "../ktk_pipeline.cuh"
#include "../ktk_vec.cuh"
#include "ktk_layers.h"

namespace ktk {

constexpr int kRnThreads = 256;
constexpr int kRnMaxVec = 8;      // 8 x 8 elements per thread: rows of up to 16384 columns
// CTAs of full width that an SM's registers have to hold: where each takes a row, and of those that walk rows
__host__ __device__ constexpr int rn_resident(int nv) { return nv <= 1 ? 4 : nv <= 2 ? 3 : nv <= 4 ? 2 : 1; }
constexpr int kRnStages = 2;       // of a walker: one row at work, one on its way; more take the L1 that holds the weights

struct ResidualNormParams {
    const int64_t* tokens;
    const void* embed;
    int64_t vocab;
    float embed_scale;
    float* x;
    const void* y;
    int parts;
    const float *post_w, *post_b;
    float mult;
    const float *pre_w, *pre_b;
    void* h;
    float eps;
    int center, cols, stride;
    int64_t rows;
    int32_t* zero;
    int zero_n;
    int32_t* status;
};

// Sum over the CTA.  `part` has room for two sums, taken in turns: who writes one of them again has met everybody at the
// barrier of the other.
struct RowParts {
    float* part;
    int turn = 0;
    __device__ __forceinline__ void clear() {
        static_assert(kRnThreads == 256, "two vectors of four sums");
        // places of absent warps: nobody else writes them, and the first sum's barrier is in front of their first reading
        if (threadIdx.x < 2 * (kRnThreads / 32) && threadIdx.x % (kRnThreads / 32) >= blockDim.x / 32) part[threadIdx.x] = 0.0f;
    }
    __device__ __forceinline__ float sum(float v) {
        float* p = part + turn * (kRnThreads / 32);
        turn ^= 1;
        v = warp_sum_f(v);
        if ((threadIdx.x & 31) == 0) p[threadIdx.x >> 5] = v;
        __syncthreads();
        const float4 a = *reinterpret_cast<const float4*>(p), b = *reinterpret_cast<const float4*>(p + 4);
        return ((((((a.x + a.y) + a.z) + a.w) + b.x) + b.y) + b.z) + b.w;
    }
};

// v <- norm(v; w, b), in registers; elements past `cols` are zero before and after (their w and b are)
template <int NV>
__device__ __forceinline__ void norm_regs(float (&v)[NV][8], const float* w, const float* b, float eps, bool center,
                                          int cols, int nvec, RowParts& part) {
    float c = 0.0f;
    if (center) {
        float s = 0.0f;
#pragma unroll
        for (int i = 0; i < NV; ++i)
#pragma unroll
            for (int e = 0; e < 8; ++e) s += v[i][e];
        c = part.sum(s) / (float)cols;
    }
    float ss = 0.0f;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
        const int k = (threadIdx.x + i * blockDim.x) * 8;
#pragma unroll
        for (int e = 0; e < 8; ++e)
            if (k + e < cols) { const float d = v[i][e] - c; ss += d * d; }
    }
    const float inv = 1.0f / sqrtf(part.sum(ss) / (float)cols + eps);
#pragma unroll
    for (int i = 0; i < NV; ++i) {
        const int k = threadIdx.x + i * blockDim.x;
        if (k < nvec) {
            float wv[8], bv[8] = {0, 0, 0, 0, 0, 0, 0, 0};
            Vec8<float>::load(w + k * 8, wv);
            if (b != nullptr) Vec8<float>::load(b + k * 8, bv);
#pragma unroll
            for (int e = 0; e < 8; ++e) v[i][e] = k * 8 + e < cols ? (v[i][e] - c) * inv * wv[e] + bv[e] : 0.0f;
        }
    }
}

// The row's own part: x and y (its parts' sum) in registers, the new stream and its norm to memory.  TOKENS: the stream starts as
// embedding rows, scaled here.
template <typename T, int NV, bool TOKENS>
__device__ __forceinline__ void finish_row(const ResidualNormParams& p, int64_t r, float (&x)[NV][8], float (&y)[NV][8], int nvec,
                                           RowParts& part) {
    if (TOKENS) {
#pragma unroll
        for (int i = 0; i < NV; ++i)
#pragma unroll
            for (int e = 0; e < 8; ++e) x[i][e] *= p.embed_scale;
    }
    if (p.y != nullptr) {
        if (p.post_w != nullptr) norm_regs<NV>(y, p.post_w, p.post_b, p.eps, p.center != 0, p.cols, nvec, part);
#pragma unroll
        for (int i = 0; i < NV; ++i)
#pragma unroll
            for (int e = 0; e < 8; ++e) x[i][e] += p.mult * y[i][e];
    }
    if (TOKENS || p.y != nullptr) {
#pragma unroll
        for (int i = 0; i < NV; ++i) {
            const int k = threadIdx.x + i * blockDim.x;
            if (k < nvec) Vec8<float>::store(p.x + r * p.stride + k * 8, x[i]);
        }
    }
    if (p.h != nullptr) {
        if (p.pre_w != nullptr) norm_regs<NV>(x, p.pre_w, p.pre_b, p.eps, p.center != 0, p.cols, nvec, part);
#pragma unroll
        for (int i = 0; i < NV; ++i) {
            const int k = threadIdx.x + i * blockDim.x;
            if (k < nvec) Vec8<T>::store((T*)p.h + r * p.stride + k * 8, x[i]);
        }
    }
}

template <typename T, bool TOKENS> struct RowSource {
    using Stream = typename std::conditional<TOKENS, T, float>::type;
    const ResidualNormParams& p;
    // where row r of the stream lies; one thread of the CTA says so if its token is none of the vocabulary
    __device__ __forceinline__ const Stream* stream(int64_t r, bool tell) const {
        if (!TOKENS) return (const Stream*)p.x + r * p.stride;
        const int64_t t = p.tokens[r];
        if (t >= 0 && t < p.vocab) return (const Stream*)p.embed + t * p.stride;
        if (tell) report(p.status, KTK_STATUS_BAD_TABLE);
        return (const Stream*)p.embed;
    }
};

__device__ __forceinline__ void clear_counts(const ResidualNormParams& p) {
    if (p.zero != nullptr && blockIdx.x == 0)
        for (int i = threadIdx.x; i < p.zero_n; i += blockDim.x) p.zero[i] = 0;
}

// A CTA per row.  56 registers with NV = 1: two more would cost an SM a sixth of its CTAs of 192 threads (bf16, 8192 x 1536, the part
// normalised: 38.8 us, 40.9 with 58 registers, which is what r as a 64-bit index gives).
template <typename T, int NV, bool TOKENS>
__global__ void __launch_bounds__(kRnThreads, rn_resident(NV)) residual_norm_kernel(const ResidualNormParams p) {
    __shared__ __align__(16) float part_s[2 * (kRnThreads / 32)];
    RowParts part{part_s};
    part.clear();
    clear_counts(p);
    const int nvec = p.stride / 8;
    const unsigned r = blockIdx.x;
    const auto* from = RowSource<T, TOKENS>{p}.stream(r, threadIdx.x == 0);
    float x[NV][8], y[NV][8];
#pragma unroll
    for (int i = 0; i < NV; ++i) {
        const int k = threadIdx.x + i * blockDim.x;
#pragma unroll
        for (int e = 0; e < 8; ++e) x[i][e] = 0.0f;
        if (k < nvec) Vec8<typename RowSource<T, TOKENS>::Stream>::load(from + k * 8, x[i]);
    }
    if (p.y != nullptr) {
#pragma unroll
        for (int i = 0; i < NV; ++i) {
            const int k = threadIdx.x + i * blockDim.x;
#pragma unroll
            for (int e = 0; e < 8; ++e) y[i][e] = 0.0f;
            if (k >= nvec) continue;
            for (int j = 0; j < p.parts; ++j) {
                float t[8];
                Vec8<T>::load((const T*)p.y + (r * p.parts + j) * p.stride + k * 8, t);
#pragma unroll
                for (int e = 0; e < 8; ++e) y[i][e] += t[e];
            }
        }
    }
    finish_row<T, NV, TOKENS>(p, r, x, y, nvec, part);
}

// CTAs that walk rows c, c + gridDim.x, ...; a ring in shared memory keeps the next row on its way by bulk copies, a stage holding a row
// of the stream and its part.  8192 rows of 4096 bf16 columns inside a model 91 -> 72 us (402 MB).
template <typename T, bool TOKENS, int NV>
__global__ void __launch_bounds__(kRnThreads, rn_resident(NV)) residual_norm_walk_kernel(const ResidualNormParams p) {
    constexpr int stages = kRnStages;
    extern __shared__ __align__(128) uint8_t rn_ring[];
    __shared__ __align__(8) uint64_t full[kRnStages];
    __shared__ __align__(16) float part_s[2 * (kRnThreads / 32)];
    __shared__ int abort_flag;
    using Source = RowSource<T, TOKENS>;
    const Source source{p};
    RowParts part{part_s};
    part.clear();
    clear_counts(p);
    const int nvec = p.stride / 8, parts = p.y != nullptr ? p.parts : 0;
    const uint32_t x_bytes = (uint32_t)(p.stride * sizeof(typename Source::Stream)), y_bytes = (uint32_t)(parts * p.stride * sizeof(T));
    const uint32_t stage_bytes = x_bytes + y_bytes;
    const bool sums = (p.y != nullptr && p.post_w != nullptr) || (p.h != nullptr && p.pre_w != nullptr);
    if (threadIdx.x == 0) {
        for (int i = 0; i < stages; ++i) mbar_init(&full[i], 1);
        abort_flag = 0;
        mbar_init_fence();
    }
    __syncthreads();
    int issued = 0;                                          // rows asked for, by thread 0
    auto ask = [&](int64_t r) {
        if (r >= p.rows) return;
        const int s = issued++ % stages;
        uint8_t* at = rn_ring + s * stage_bytes;
        mbar_arrive_expect_tx(&full[s], stage_bytes);
        bulk_load(at, source.stream(r, true), x_bytes, &full[s]);
        if (y_bytes) bulk_load(at + x_bytes, (const T*)p.y + r * parts * p.stride, y_bytes, &full[s]);
    };
    const int64_t step = gridDim.x;
    if (threadIdx.x == 0)
        for (int i = 0; i < stages; ++i) ask(blockIdx.x + i * step);
    int s = 0;
    uint32_t parity = 0;
    int64_t r = blockIdx.x;
    for (int i = 0; r < p.rows; ++i, r += step) {
        // the vote keeps the warp together should a single lane give up: the sums below shuffle over all of it
        if (!__all_sync(0xffffffffu, mbar_wait(&full[s], parity, &abort_flag))) break;
        if (threadIdx.x == 0 && i > 0) {                     // everybody has read the row before: its sums had a barrier
            fence_proxy_async();
            ask(r + (stages - 1) * step);
        }
        const auto* xs = reinterpret_cast<const typename Source::Stream*>(rn_ring + s * stage_bytes);
        const T* ys = reinterpret_cast<const T*>(rn_ring + s * stage_bytes + x_bytes);
        float x[NV][8], y[NV][8];
#pragma unroll
        for (int v = 0; v < NV; ++v) {
            const int k = threadIdx.x + v * blockDim.x;
#pragma unroll
            for (int e = 0; e < 8; ++e) x[v][e] = y[v][e] = 0.0f;
            if (k >= nvec) continue;
            Vec8<typename Source::Stream>::load(xs + k * 8, x[v]);       // shared memory: no read-only load
            for (int j = 0; j < parts; ++j) {
                float t[8];
                Vec8<T>::load(ys + j * p.stride + k * 8, t);
#pragma unroll
                for (int e = 0; e < 8; ++e) y[v][e] += t[e];
            }
        }
        if (!sums) __syncthreads();
        finish_row<T, NV, TOKENS>(p, r, x, y, nvec, part);
        if (++s == stages) { s = 0; parity ^= 1u; }
    }
    if (abort_flag && threadIdx.x == 0) {                    // gave up: the copies in flight still write shared memory
        report(p.status, KTK_STATUS_TIMEOUT);
        volatile int never = 0;
        for (int i = issued > stages ? issued - stages : 0; i < issued; ++i) mbar_wait(&full[i % stages], (i / stages) & 1, &never);
    }
}

template <typename T, bool TOKENS>
static int residual_norm_launch(const ResidualNormParams& p, cudaStream_t st) {
    const char* who = "ktk_residual_norm";
    const int nvec = p.stride / 8;
    const int threads = nvec >= kRnThreads ? kRnThreads : (nvec + 31) / 32 * 32;
    const int nv = (nvec + threads - 1) / threads;
    // Walkers: rows of up to 4096 columns by three CTAs of 256 threads per SM; bf16 rows of 1793 to 2048 columns by six of 128, or by four of 256
    // (from 1921 columns on, whose threads are all busy) where only the part is normalised.  us, a CTA per row / walkers, next rows not in L2, part and next sublayer normed: 8192 x 4096 bf16
    // 111 / 94, 1776 x 4096 33 / 30.5, 8192 x 2048 bf16 58 / 54, 2400 x 2048 24 / 23, 8192 x 4096 fp32 129 / 112; the part alone 8192 x 4096
    // 96 / 79, 4100 x 2048 29.9 / 29.4 (six of 128: 30.4); embedding rows 8192 x 2048 48 / 41 and x 4096 90 / 68.  Not fp32 of 2048 columns
    // (68 / 70), sums of neither (2048 columns 24.4 / 25.4, fp32 4096 102 / 105), 1024 columns (25 / 28), several parts (8 of 2048 80 / 82, 4 of
    // 4096 110 / 110).
    const bool narrow = nvec <= kRnThreads, pre = p.h != nullptr && p.pre_w != nullptr, post = p.y != nullptr && p.post_w != nullptr;
    const bool fits = nvec > kRnThreads - 32 && nvec <= 2 * kRnThreads && (p.y == nullptr || p.parts == 1);
    if (fits && (pre || post || TOKENS || (!narrow && sizeof(T) == 2)) && (sizeof(T) == 2 || !narrow) &&
        p.rows >= (narrow ? 16 : 12) * (int64_t)sm_count()) {
        const size_t stage = (size_t)p.stride * (TOKENS ? sizeof(T) : 4) + (p.y ? (size_t)p.stride * sizeof(T) : 0);
        const auto walk = [&](auto kernel, int threads_of, int resident) {
            KTK_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(kRnStages * stage)), who);
            kernel<<<(unsigned)(sm_count() * resident), threads_of, kRnStages * stage, st>>>(p);
            KTK_CUDA_TRY(cudaGetLastError(), who);
            return (int)KTK_OK;
        };
        if (!narrow) return walk(residual_norm_walk_kernel<T, TOKENS, 2>, kRnThreads, 3);
        if constexpr (sizeof(T) == 2) {
            if constexpr (!TOKENS)
                if (!pre && nvec > kRnThreads - 16) return walk(residual_norm_walk_kernel<T, false, 1>, kRnThreads, 4);
            return walk(residual_norm_walk_kernel<T, TOKENS, 2>, kRnThreads / 2, 6);
        }
    }
    auto kernel = nv <= 1 ? residual_norm_kernel<T, 1, TOKENS>
                : nv <= 2 ? residual_norm_kernel<T, 2, TOKENS>
                : nv <= 4 ? residual_norm_kernel<T, 4, TOKENS>
                          : residual_norm_kernel<T, kRnMaxVec, TOKENS>;
    kernel<<<(unsigned)p.rows, threads, 0, st>>>(p);
    KTK_CUDA_TRY(cudaGetLastError(), who);
    return KTK_OK;
}

}  // namespace ktk

using namespace ktk;

extern "C" int ktk_residual_norm(const int64_t* tokens, const void* embed, int64_t vocab, float embed_scale, float* x,
                                 const void* y, int32_t parts, const float* post_w, const float* post_b, float mult,
                                 const float* pre_w, const float* pre_b, void* h, float eps, int32_t center,
                                 int64_t rows, int32_t cols, int32_t stride, int32_t* zero, int32_t zero_n,
                                 int32_t dtype, int32_t* status, void* stream) {
    const char* who = "ktk_residual_norm";
    if (rows < 0 || rows > 2147483647LL || cols <= 0 || stride < cols || stride % 8 != 0 || parts < 1 || zero_n < 0 ||
        (dtype != KTK_F32 && dtype != KTK_BF16)) {
        set_error("%s: rows=%lld cols=%d stride=%d parts=%d zero_n=%d dtype=%d", who, (long long)rows, cols, stride,
                  parts, zero_n, dtype);
        return KTK_ERR_ARG;
    }
    if (stride > 8 * kRnThreads * kRnMaxVec) {
        set_error("%s: rows of at most %d columns are built (got %d)", who, 8 * kRnThreads * kRnMaxVec, stride);
        return KTK_ERR_UNSUPPORTED;
    }
    if (rows == 0) return KTK_OK;
    if (!x || (tokens && (!embed || vocab <= 0)) || (!h && !y && !tokens)) {
        set_error("%s: null pointer argument", who);
        return KTK_ERR_ARG;
    }
    const uintptr_t al = (uintptr_t)embed | (uintptr_t)x | (uintptr_t)y | (uintptr_t)post_w | (uintptr_t)post_b |
                         (uintptr_t)pre_w | (uintptr_t)pre_b | (uintptr_t)h;
    if ((al & 15u) != 0) { set_error("%s: pointers must be 16-byte aligned", who); return KTK_ERR_ARG; }
    const ResidualNormParams p{tokens, embed, vocab, embed_scale, x, y, parts, post_w, post_b, mult, pre_w, pre_b, h, eps,
                               center, cols, stride, rows, zero, zero ? zero_n : 0, status};
    cudaStream_t st = (cudaStream_t)stream;
    if (dtype == KTK_F32) return tokens ? residual_norm_launch<float, true>(p, st) : residual_norm_launch<float, false>(p, st);
    return tokens ? residual_norm_launch<__nv_bfloat16, true>(p, st) : residual_norm_launch<__nv_bfloat16, false>(p, st);
}
