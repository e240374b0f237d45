// Products of a few rows with a weight matrix, y = x W^T (+ bias) (+ residual), or silu(x W^T) * (x W2^T), in one launch.
//
// A decode step of up to 16 sequences reads every weight once and does next to nothing with it: bound by DRAM for large matrices,
// by launches and latency for small ones.  A CTA takes a few weight rows and all rows of x; its warps share the columns out, a lane
// has 16 bytes of every weight row and of every row of x on their way at a time; products in fp32 by FMA, partial sums
// folded over the lanes (each lane ends with one of them) and over the warps in shared memory.
// us, cuBLAS / this, weights not in L2: fp32, 4 rows, 512 x 512 4.5 / 2.2, 512 x 1024 7.4 / 2.3, gated 1024 x 512 15.9 / 2.9, 4096 x 4096
// 58 / 14; bf16, 4 rows, 768 x 4096 9.1 / 5.7, gated 1536 x 4096 21.7 / 10.6 (3.9 by the bytes).  Which shapes gain: linear_rows_wins in
// ops.py.
#include "ktk_common.cuh"
#include "ktk_vec.cuh"

namespace ktk {

constexpr int kLrThreads = 256, kLrWarps = kLrThreads / 32, kLrMaxRows = 16;

struct LinearParams {
    const void *x, *w, *w2, *bias, *residual;
    void* out;
    int rows, n, k;
};

template <typename T> struct LrVec;                              // 16 bytes as fp32
template <> struct LrVec<float> {
    static constexpr int kN = 4;
    static __device__ __forceinline__ void load(const float* p, float (&f)[4]) {
        const float4 a = __ldg(reinterpret_cast<const float4*>(p));
        f[0] = a.x; f[1] = a.y; f[2] = a.z; f[3] = a.w;
    }
};
template <> struct LrVec<__nv_bfloat16> {
    static constexpr int kN = 8;
    static __device__ __forceinline__ void load(const __nv_bfloat16* p, float (&f)[8]) { load8(p, f); }
};

// N sums over the warp's 32 lanes at once, N a power of two.  Afterwards lane l holds, for N >= 32, sum l * (N / 32) + j in v[j], for
// fewer sum l / (32 / N) in v[0]
template <int N> __device__ __forceinline__ void fold_lanes(float (&v)[N]) {
    const int lane = threadIdx.x & 31;
    int have = N;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        if (have > (N > 32 ? N / 32 : 1)) {                      // halve what a lane keeps
            const bool upper = lane & o;
#pragma unroll
            for (int i = 0; i < N / 2; ++i)
                if (i < have / 2) {
                    const float give = upper ? v[i] : v[i + have / 2], keep = upper ? v[i + have / 2] : v[i];
                    v[i] = keep + __shfl_xor_sync(0xffffffffu, give, o);
                }
            have /= 2;
        } else {
#pragma unroll
            for (int i = 0; i < N; ++i)
                if (i < have) v[i] += __shfl_xor_sync(0xffffffffu, v[i], o);
        }
    }
}
// the sum that v[j] of this lane is, after fold_lanes<N>
template <int N> __device__ __forceinline__ int folded(int j) {
    const int lane = threadIdx.x & 31;
    int at = 0, have = N;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
        if (have > (N > 32 ? N / 32 : 1)) {
            have /= 2;
            if (lane & o) at += have;
        }
    return at + j;
}

// COLS weight rows per CTA (GATED: half of them of W, half of W2), ROWS rows of x
template <typename T, int ROWS, int COLS, bool GATED>
__global__ void __launch_bounds__(kLrThreads) linear_rows_kernel(const LinearParams p) {
    constexpr int kVec = LrVec<T>::kN, kSums = ROWS * COLS, kOwn = GATED ? COLS / 2 : COLS, kLeft = kSums > 32 ? kSums / 32 : 1;
    __shared__ float part[kLrWarps][kSums];
    wait_for_front();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int n0 = blockIdx.x * kOwn;
    const T* wrow[COLS];
#pragma unroll
    for (int c = 0; c < COLS; ++c) {
        const int n = n0 + c % kOwn < p.n ? n0 + c % kOwn : p.n - 1;     // rows behind the last are computed and dropped
        wrow[c] = (const T*)(GATED && c >= kOwn ? p.w2 : p.w) + (int64_t)n * p.k;
    }
    const T* x = (const T*)p.x;
    float acc[kSums];                                            // [row][column]
#pragma unroll
    for (int i = 0; i < kSums; ++i) acc[i] = 0.0f;
#pragma unroll(ROWS <= 2 ? 2 : 1)
    for (int k = (warp * 32 + lane) * kVec; k < p.k; k += kLrThreads * kVec) {
        float w[COLS][kVec];
#pragma unroll
        for (int c = 0; c < COLS; ++c) LrVec<T>::load(wrow[c] + k, w[c]);
#pragma unroll
        for (int r = 0; r < ROWS; ++r) {
            float v[kVec];
            LrVec<T>::load(x + (int64_t)(r < p.rows ? r : 0) * p.k + k, v);
#pragma unroll
            for (int c = 0; c < COLS; ++c)
#pragma unroll
                for (int e = 0; e < kVec; ++e) acc[r * COLS + c] = fmaf(v[e], w[c][e], acc[r * COLS + c]);
        }
    }
    fold_lanes(acc);
#pragma unroll
    for (int j = 0; j < kLeft; ++j) part[warp][folded<kSums>(j)] = acc[j];       // fewer than 32 sums: several lanes, one value
    __syncthreads();
    for (int i = threadIdx.x; i < ROWS * kOwn; i += kLrThreads) {
        const int r = i / kOwn, c = i - r * kOwn, n = n0 + c;
        if (r >= p.rows || n >= p.n) continue;
        float v = 0.0f, u = 0.0f;
#pragma unroll
        for (int w = 0; w < kLrWarps; ++w) {
            v += part[w][r * COLS + c];
            if (GATED) u += part[w][r * COLS + kOwn + c];
        }
        if (GATED) v = v / (1.0f + __expf(-v)) * u;
        if (p.bias) v += to_f32(((const T*)p.bias)[n]);
        const int64_t at = (int64_t)r * p.n + n;
        if (p.residual) v += to_f32(((const T*)p.residual)[at]);
        ((T*)p.out)[at] = from_f32<T>(v);
    }
}

template <typename T, bool GATED> static int linear_rows_launch(const LinearParams& p, cudaStream_t st) {
    auto go = [&](auto kernel, int own) {
        return launch_behind(true, kernel, (unsigned)((p.n + own - 1) / own), kLrThreads, 0, st, p);
    };
    constexpr int kHalf = GATED ? 2 : 1;
    KTK_CUDA_TRY(p.rows <= 1   ? go(linear_rows_kernel<T, 1, 8, GATED>, 8 / kHalf)
                 : p.rows <= 2 ? go(linear_rows_kernel<T, 2, 8, GATED>, 8 / kHalf)
                 : p.rows <= 4 ? go(linear_rows_kernel<T, 4, 8, GATED>, 8 / kHalf)
                 : p.rows <= 8 ? go(linear_rows_kernel<T, 8, 8, GATED>, 8 / kHalf)
                               : go(linear_rows_kernel<T, 16, 4, GATED>, 4 / kHalf),
                 "ktk_linear_rows");
    return KTK_OK;
}

}  // namespace ktk

using namespace ktk;

extern "C" int ktk_linear_rows(const void* x, const void* w, const void* w2, const void* bias, const void* residual, void* out,
                               int64_t rows, int64_t n, int64_t k, int32_t dtype, void* stream) {
    const char* who = "ktk_linear_rows";
    if (rows < 0 || rows > kLrMaxRows || n < 0 || n > 2147483647LL || k <= 0 || k > 2147483647LL || k % 8 != 0 ||
        (dtype != KTK_F32 && dtype != KTK_BF16)) {
        set_error("%s: rows=%lld (at most %d) n=%lld k=%lld dtype=%d", who, (long long)rows, kLrMaxRows, (long long)n, (long long)k, dtype);
        return KTK_ERR_ARG;
    }
    if (rows == 0 || n == 0) return KTK_OK;
    if (!x || !w || !out || (((uintptr_t)x | (uintptr_t)w | (uintptr_t)w2) & 15u) != 0) {
        set_error("%s: null or misaligned pointer", who);
        return KTK_ERR_ARG;
    }
    const LinearParams p{x, w, w2, bias, residual, out, (int)rows, (int)n, (int)k};
    cudaStream_t st = (cudaStream_t)stream;
    if (dtype == KTK_F32) return w2 ? linear_rows_launch<float, true>(p, st) : linear_rows_launch<float, false>(p, st);
    return w2 ? linear_rows_launch<__nv_bfloat16, true>(p, st) : linear_rows_launch<__nv_bfloat16, false>(p, st);
}
