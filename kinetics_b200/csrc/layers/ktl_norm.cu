// The residual stream between two sublayers in one pass over each row: the previous sublayer's output (summed over
// its parts) is normalised and added, the new stream normalised for the next sublayer.  The stream and everything
// computed here is fp32; a CTA has one row at a time in registers, 8 elements per access.
//
// Bound by DRAM for prompts, by its chain of reductions for few rows: one barrier per sum.  8192 rows of 2048 columns in bf16, 201 MB:
// 60 us with two barriers per sum, 54 with one, 51 where CTAs walk rows with the next one in flight; eight parts 94, 88.  What keeps
// rows in flight otherwise is the number of CTAs that the registers allow (rn_resident): half as many, for the registers of a row
// ahead, made eight parts of 4096 columns 211 us instead of 167, of 5120 columns 178 for 112 (3000 rows).
#include <type_traits>

#include "../ktk_vec.cuh"
#include "ktk_layers.h"

namespace ktk {

constexpr int kRnThreads = 256;
constexpr int kRnMaxVec = 8;      // 8 x 8 elements per thread: rows of up to 16384 columns
// CTAs of full width that an SM's registers have to hold: where each takes a row, and of those that walk rows
__host__ __device__ constexpr int rn_resident(int nv) { return nv <= 1 ? 4 : nv <= 2 ? 3 : nv <= 4 ? 2 : 1; }
constexpr int kRnWalkers = 3;
// CTAs walk from this many rows each: 3000 rows of 2048 bf16 columns 19.7 us with a CTA per row and 20.0 with walkers, 8192 rows 54.3
// and 50.9.  Not rows of fewer warps (1024 columns: 23.4 and 24.3), of fp32 (61.3 and 62.4) or of several parts.
constexpr int kRnWalkRows = 8;

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

// 8 elements as they lie in memory
template <typename T> struct Raw8;
template <> struct Raw8<float> {
    float4 a, b;
    __device__ __forceinline__ void load(const float* p) { a = *reinterpret_cast<const float4*>(p); b = *(reinterpret_cast<const float4*>(p) + 1); }
    __device__ __forceinline__ void get(float (&f)[8]) const {
        f[0] = a.x; f[1] = a.y; f[2] = a.z; f[3] = a.w; f[4] = b.x; f[5] = b.y; f[6] = b.z; f[7] = b.w;
    }
};
template <> struct Raw8<__nv_bfloat16> {
    uint4 a;
    __device__ __forceinline__ void load(const __nv_bfloat16* p) { a = *reinterpret_cast<const uint4*>(p); }
    __device__ __forceinline__ void get(float (&f)[8]) const { unpack8(a, f); }
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

// TOKENS: the stream starts as embedding rows.  WALK: the CTA walks rows, the next one in flight
template <typename T, int NV, bool TOKENS, bool WALK>
__global__ void __launch_bounds__(kRnThreads, WALK ? kRnWalkers : rn_resident(NV)) residual_norm_kernel(const ResidualNormParams p) {
    using Stream = typename std::conditional<TOKENS, T, float>::type;
    __shared__ __align__(16) float part_s[2 * (kRnThreads / 32)];
    RowParts part{part_s};
    part.clear();
    const int nvec = p.stride / 8;
    if (p.zero != nullptr && blockIdx.x == 0)
        for (int i = threadIdx.x; i < p.zero_n; i += blockDim.x) p.zero[i] = 0;
    auto token = [&](int64_t r) -> int64_t {
        if (!TOKENS || r >= p.rows) return 0;
        const int64_t t = p.tokens[r];
        if (t >= 0 && t < p.vocab) return t;
        if (threadIdx.x == 0) report(p.status, KTK_STATUS_BAD_TABLE);
        return 0;
    };
    auto stream_row = [&](int64_t r, int64_t tok) {
        return TOKENS ? (const Stream*)p.embed + tok * p.stride : (const Stream*)p.x + r * p.stride;
    };
    Raw8<Stream> xr[WALK ? NV : 1];
    Raw8<T> yr[WALK ? NV : 1];
    auto fetch = [&](int64_t r, int64_t tok) {             // WALK
        if (r >= p.rows) return;
        const Stream* from = stream_row(r, tok);
#pragma unroll
        for (int i = 0; i < NV; ++i) {
            const int k = threadIdx.x + i * blockDim.x;
            if (k >= nvec) continue;
            xr[WALK ? i : 0].load(from + k * 8);
            if (p.y != nullptr) yr[WALK ? i : 0].load((const T*)p.y + r * p.stride + k * 8);
        }
    };
    int64_t r = blockIdx.x, ahead = token(r);
    if (WALK) {
        fetch(r, ahead);
        ahead = token(r + gridDim.x);
    }
    for (; r < p.rows; r += gridDim.x) {
        float x[NV][8], y[NV][8];
        float* xrow = p.x + r * p.stride;
#pragma unroll
        for (int i = 0; i < NV; ++i) {
            const int k = threadIdx.x + i * blockDim.x;
#pragma unroll
            for (int e = 0; e < 8; ++e) x[i][e] = 0.0f;
            if (k >= nvec) continue;
            if (!WALK) xr[0].load(stream_row(r, ahead) + k * 8);
            xr[WALK ? i : 0].get(x[i]);
            if (TOKENS) {
#pragma unroll
                for (int e = 0; e < 8; ++e) x[i][e] *= p.embed_scale;
            }
        }
        if (p.y != nullptr) {
#pragma unroll
            for (int i = 0; i < NV; ++i) {
                const int k = threadIdx.x + i * blockDim.x;
#pragma unroll
                for (int e = 0; e < 8; ++e) y[i][e] = 0.0f;
                if (k >= nvec) continue;
                if (WALK) {
                    yr[i].get(y[i]);
                } else {
                    for (int j = 0; j < p.parts; ++j) {
                        float t[8];
                        Vec8<T>::load((const T*)p.y + (r * p.parts + j) * p.stride + k * 8, t);
#pragma unroll
                        for (int e = 0; e < 8; ++e) y[i][e] += t[e];
                    }
                }
            }
        }
        if (WALK) {
            fetch(r + gridDim.x, ahead);
            ahead = token(r + 2 * (int64_t)gridDim.x);
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
                if (k < nvec) Vec8<float>::store(xrow + k * 8, x[i]);
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
        if (!WALK) break;
    }
}

template <typename T, bool TOKENS>
static int residual_norm_launch(const ResidualNormParams& p, cudaStream_t st) {
    const int nvec = p.stride / 8;
    const int threads = nvec >= kRnThreads ? kRnThreads : (nvec + 31) / 32 * 32;
    const int nv = (nvec + threads - 1) / threads;
    const int64_t walkers = (int64_t)sm_count() * kRnWalkers;
    if constexpr (sizeof(T) == 2) {
        if (threads == kRnThreads && nv == 1 && p.parts == 1 && p.rows >= kRnWalkRows * walkers) {
            residual_norm_kernel<T, 1, TOKENS, true><<<(unsigned)walkers, threads, 0, st>>>(p);
            KTK_CUDA_TRY(cudaGetLastError(), "ktk_residual_norm");
            return KTK_OK;
        }
    }
    auto kernel = nv <= 1 ? residual_norm_kernel<T, 1, TOKENS, false>
                : nv <= 2 ? residual_norm_kernel<T, 2, TOKENS, false>
                : nv <= 4 ? residual_norm_kernel<T, 4, TOKENS, false>
                          : residual_norm_kernel<T, kRnMaxVec, TOKENS, false>;
    kernel<<<(unsigned)p.rows, threads, 0, st>>>(p);
    KTK_CUDA_TRY(cudaGetLastError(), "ktk_residual_norm");
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
