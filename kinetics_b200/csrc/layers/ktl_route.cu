// Router of a mixture of experts: fp32 logits of every row against every expert, the best `top` of them, the softmax
// over those, and each row's place in its experts' buckets -- one launch.
//
// Many rows of bf16: tiles on the tensor cores; few rows, and fp32: a CTA per row with FMA.  Then a warp per row picks the
// experts.
#include "../ktk_pipeline.cuh"
#include "ktl_common.cuh"

namespace ktk {

constexpr int kRtThreads = 256;
constexpr int kRtWarps = kRtThreads / 32;
constexpr int kRtRows = 32;          // rows of a CTA, tensor-core variant
constexpr int kRtCols = 64;          // experts per pass
constexpr int kRtByRow = 256;        // up to this many rows: a CTA per row
constexpr int kRtRowThreads = 512;

struct RouteParams {
    ktk_moe m;
    const void *h, *w;
    const float* b;
    int32_t* ids;
    float* weights;
    int32_t* counts;
    int32_t* bucket;
    int64_t rows;
};

// One warp: the `top` largest of z[0 .. experts) (ties to the lower index), weighted by the softmax over them or over all.
// z is overwritten.
// ids_s [top], shared memory of the warp: the choice, for the caller.
__device__ __forceinline__ void pick_experts(const RouteParams& p, float* z, int64_t row, int32_t* ids_s) {
    const int lane = threadIdx.x & 31;
    const int E = p.m.experts, top = p.m.top;
    float best0 = 0.0f, denom = 0.0f, denom_all = 0.0f;
    if (p.m.scoring == 1) {
        float mx = -INFINITY;
        for (int i = lane; i < E; i += 32) mx = fmaxf(mx, z[i]);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        for (int i = lane; i < E; i += 32) denom_all += expf(z[i] - mx);
        denom_all = warp_sum_f(denom_all);
    }
    for (int j = 0; j < top; ++j) {
        uint32_t key = 0;
        int e = E - 1;
        for (int i = lane; i < E; i += 32) {
            const uint32_t k = score_to_key(z[i]);
            if (k > key) { key = k; e = i; }
        }
        const uint32_t best = __reduce_max_sync(0xffffffffu, key);
        e = (int)__reduce_min_sync(0xffffffffu, key == best ? (uint32_t)e : 0x7fffffffu);
        const float v = z[e];
        if (j == 0) best0 = v;
        const float ex = expf(v - best0);
        denom += ex;
        __syncwarp();
        if (lane == 0) {
            z[e] = -INFINITY;
            ids_s[j] = e;
            p.ids[row * top + j] = e;
            p.weights[row * top + j] = ex;
        }
        __syncwarp();
    }
    if (p.m.scoring == 1) denom = denom_all;
    for (int j = lane; j < top; j += 32) p.weights[row * top + j] /= denom;
}

// One CTA per row: warp w takes experts w, w + 16, ..., two at a time; lanes share the width, 8 elements per load and up
// to 16 loads in flight.  For fp32 and for the few rows of a decode step (the weights stay in L2).
template <typename T>
__global__ void __launch_bounds__(kRtRowThreads) route_row_kernel(const RouteParams p) {
    extern __shared__ float rt_z[];                       // [experts] | the row [width_stride] | ids [top]
    constexpr int kWarps = kRtRowThreads / 32, kUnroll = 8;
    const int64_t row = blockIdx.x;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int K = p.m.width_stride, E = p.m.experts, top = p.m.top;
    float* hs = rt_z + (E + 3) / 4 * 4;
    int32_t* ids_s = reinterpret_cast<int32_t*>(hs + K);
    for (int i = threadIdx.x * 8; i < K; i += kRtRowThreads * 8) {
        float v[8];
        load8((const T*)p.h + row * K + i, v);
#pragma unroll
        for (int e = 0; e < 8; ++e) hs[i + e] = v[e];
    }
    __syncthreads();
    for (int e0 = warp; e0 < E; e0 += 2 * kWarps) {
        const int e1 = e0 + kWarps < E ? e0 + kWarps : e0;
        const T* w0 = (const T*)p.w + (int64_t)e0 * K;
        const T* w1 = (const T*)p.w + (int64_t)e1 * K;
        float s0 = 0.0f, s1 = 0.0f;
        for (int i0 = lane * 8; i0 < K; i0 += 256 * kUnroll) {
#pragma unroll
            for (int u = 0; u < kUnroll; ++u) {
                const int i = i0 + u * 256;
                if (i < K) {
                    float hv[8], a[8], b[8];
                    load8(w0 + i, a);
                    load8(w1 + i, b);
                    Vec8<float>::load(hs + i, hv);
#pragma unroll
                    for (int x = 0; x < 8; ++x) { s0 = fmaf(hv[x], a[x], s0); s1 = fmaf(hv[x], b[x], s1); }
                }
            }
        }
        s0 = warp_sum_f(s0);
        s1 = warp_sum_f(s1);
        if (lane == 0) {
            rt_z[e0] = p.b ? s0 + p.b[e0] : s0;
            if (e1 != e0) rt_z[e1] = p.b ? s1 + p.b[e1] : s1;
        }
    }
    __syncthreads();
    if (warp == 0) {
        pick_experts(p, rt_z, row, ids_s);
        for (int j = lane; j < top; j += 32) {
            const int e = ids_s[j], at = atomicAdd(p.counts + e, 1);
            if (at < p.rows) p.bucket[(int64_t)e * p.rows + at] = (int32_t)(row * top + j);
        }
    }
}

// The same for the four rows z, z + ld, ... of a warp side by side, whose lookups then share their latency: up to 256 experts, top up
// to 32, the scores in registers.  The same choice and the same sums in the same order.
constexpr int kRtPick = 4, kRtPickExperts = 256, kRtPickTop = 32;
template <int kPer> __device__ __forceinline__ void pick_experts4(const RouteParams& p, float* z, int ld, int64_t row, int32_t* ids_s) {
    const int lane = threadIdx.x & 31;
    const int E = p.m.experts, top = p.m.top;
    uint32_t key[kRtPick][kPer];
    float denom[kRtPick], val[kRtPick];
    int id[kRtPick];
#pragma unroll
    for (int r = 0; r < kRtPick; ++r) {
        val[r] = 0.0f;
        id[r] = 0;
#pragma unroll
        for (int i = 0; i < kPer; ++i) key[r][i] = lane + 32 * i < E ? score_to_key(z[r * ld + lane + 32 * i]) : 0u;
        if (p.m.scoring == 1) {
            float mx = -INFINITY, sum = 0.0f;
            for (int i = lane; i < E; i += 32) mx = fmaxf(mx, z[r * ld + i]);
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
            for (int i = lane; i < E; i += 32) sum += expf(z[r * ld + i] - mx);
            denom[r] = warp_sum_f(sum);
        } else denom[r] = 0.0f;
    }
    const uint32_t gone = score_to_key(-INFINITY);
    for (int j = 0; j < top; ++j) {
        uint32_t best[kRtPick];
        int e[kRtPick];
#pragma unroll
        for (int r = 0; r < kRtPick; ++r) {
            best[r] = 0u;
            e[r] = E - 1;
#pragma unroll
            for (int i = 0; i < kPer; ++i)
                if (key[r][i] > best[r]) { best[r] = key[r][i]; e[r] = lane + 32 * i; }
        }
#pragma unroll
        for (int r = 0; r < kRtPick; ++r) {
            const uint32_t most = __reduce_max_sync(0xffffffffu, best[r]);
            e[r] = (int)__reduce_min_sync(0xffffffffu, best[r] == most ? (uint32_t)e[r] : 0x7fffffffu);
        }
#pragma unroll
        for (int r = 0; r < kRtPick; ++r) {
            const float v = z[r * ld + e[r]];
            if (lane == j) { val[r] = v; id[r] = e[r]; }
#pragma unroll
            for (int i = 0; i < kPer; ++i)
                if (e[r] == lane + 32 * i) key[r][i] = gone;
        }
        __syncwarp();
        if (lane < kRtPick) z[lane * ld + (lane == 0 ? e[0] : lane == 1 ? e[1] : lane == 2 ? e[2] : e[3])] = -INFINITY;
        __syncwarp();
    }
#pragma unroll
    for (int r = 0; r < kRtPick; ++r) {
        const float ex = expf(val[r] - __shfl_sync(0xffffffffu, val[r], 0));
        if (p.m.scoring != 1)
            for (int j = 0; j < top; ++j) denom[r] += __shfl_sync(0xffffffffu, ex, j);
        const int64_t at = row + r;
        if (lane < top && at < p.rows) {
            ids_s[r * top + lane] = id[r];
            p.ids[at * top + lane] = id[r];
            p.weights[at * top + lane] = ex / denom[r];
        }
    }
}

// A CTA takes 32 rows.  Columns 128 at a time: h [32 x 128] and W [64 experts x 128] through a ring of cp.async stages; warp
// w accumulates 16 rows and 16 experts of the pass with mma.m16n8k16 (exact products, fp32 sums).  Bound by latency: 8192 rows of 2048
// columns, 64 experts, 41 us with stages of 64 columns, a fragment per load and each row's choices one behind the other, 25 us this way;
// 13 of 64 warps resident, an SM reads 26 bytes a clock from L2, tensor pipe 18 %.
constexpr int kRtK = 128, kRtLd = kRtK + 8;                      // padded rows: no bank conflicts
constexpr int kRtStageElems = (kRtRows + kRtCols) * kRtLd;
constexpr int kRtPieces = (kRtRows + kRtCols) * (kRtK / 8) / kRtThreads, kRtPieceRows = kRtThreads / (kRtK / 8);
static_assert(kMaxExperts * 2 * 4 <= 2 * kRtStageElems * 2, "the expert counters fit the ring");
constexpr size_t kRtMostRest = 227 * 1024 - 54 * 1024;           // logits and choices; two stages fit beside them
static_assert(2 * kRtStageElems * 2 <= 54 * 1024, "two stages fit");
static_assert(kRtRows % kRtPieceRows == 0, "a thread's piece is one of h or one of W");

template <int STAGES> __global__ void __launch_bounds__(kRtThreads) route_mma_kernel(const RouteParams p) {
    extern __shared__ __align__(16) uint8_t rt_raw[];     // ring | logits [32][experts padded to 64] | ids, places [32][top]
    __nv_bfloat16* ring = reinterpret_cast<__nv_bfloat16*>(rt_raw);
    float* rt_z = reinterpret_cast<float*>(rt_raw + STAGES * kRtStageElems * 2);
    int32_t* ids_s = reinterpret_cast<int32_t*>(rt_z + kRtRows * ((p.m.experts + kRtCols - 1) / kRtCols * kRtCols));
    int32_t* place_s = ids_s + kRtRows * p.m.top;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int gid = lane >> 2, tig = lane & 3;
    const int E = p.m.experts, ld = (E + kRtCols - 1) / kRtCols * kRtCols;
    const int64_t row0 = (int64_t)blockIdx.x * kRtRows;
    const int K = p.m.width_stride, steps = (K + kRtK - 1) / kRtK;
    // a thread copies columns `col` .. of every kRtPieceRows-th row, of h first, then of W
    const int first = tid / (kRtK / 8), col = tid % (kRtK / 8) * 8;
    const int m0 = (warp & 1) * 16, n0 = (warp >> 1) * 16;
    for (int c0 = 0; c0 < E; c0 += kRtCols) {
        const __nv_bfloat16* src[kRtPieces];
        bool on[kRtPieces];
#pragma unroll
        for (int i = 0; i < kRtPieces; ++i) {
            const int r = first + i * kRtPieceRows;
            const bool is_h = i * kRtPieceRows < kRtRows;
            const int64_t at = is_h ? row0 + r : c0 + r - kRtRows;
            on[i] = at < (is_h ? p.rows : (int64_t)E);
            src[i] = (const __nv_bfloat16*)(is_h ? p.h : p.w) + (on[i] ? at * K + col : 0);
        }
        auto load = [&](int s) {
            const uint32_t dst = smem_u32(ring + (s % STAGES) * kRtStageElems + first * kRtLd + col);
            const bool in = s * kRtK + col < K;
#pragma unroll
            for (int i = 0; i < kRtPieces; ++i)
                cp_async16(dst + i * kRtPieceRows * kRtLd * 2, in ? src[i] + s * kRtK : (const __nv_bfloat16*)p.h, in && on[i] ? 16u : 0u);
        };
        float acc[2][4];
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[i][e] = 0.0f;
        for (int s = 0; s < STAGES - 1; ++s) {
            if (s < steps) load(s);
            cp_async_commit();
        }
        for (int s = 0; s < steps; ++s) {
            asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
            __syncthreads();                              // stage s is in place; everyone is done with stage s - 1
            if (s + STAGES - 1 < steps) load(s + STAGES - 1);
            cp_async_commit();
            const __nv_bfloat16* st = ring + (s % STAGES) * kRtStageElems;
            const uint32_t ha = smem_u32(st + (m0 + (lane & 15)) * kRtLd + (lane >> 4) * 8);
            const uint32_t wa = smem_u32(st + (kRtRows + n0 + (lane & 7) + (lane >> 4) * 8) * kRtLd + ((lane >> 3) & 1) * 8);
#pragma unroll
            for (int k = 0; k < kRtK; k += 16) {
                uint32_t a[4], b[4];
                ldmatrix_x4(a, ha + k * 2);
                ldmatrix_x4(b, wa + k * 2);
                mma_bf16(acc[0], a, b[0], b[1]);
                mma_bf16(acc[1], a, b[2], b[3]);
            }
        }
        asm volatile("cp.async.wait_group 0;" ::: "memory");
#pragma unroll
        for (int t = 0; t < 2; ++t)
#pragma unroll
            for (int x = 0; x < 4; ++x) {
                const int e = c0 + n0 + 8 * t + 2 * tig + (x & 1);
                rt_z[(m0 + gid + (x >= 2 ? 8 : 0)) * ld + e] = acc[t][x] + (p.b && e < E ? p.b[e] : 0.0f);
            }
        __syncthreads();
    }
    static_assert(kRtRows == kRtPick * kRtWarps, "a warp's rows at once");
    if (E <= kRtPickExperts && p.m.top <= kRtPickTop) {
        float* z = rt_z + warp * kRtPick * ld;
        int32_t* ids = ids_s + warp * kRtPick * p.m.top;
        const int64_t row = row0 + warp * kRtPick;
        if (E <= 64) pick_experts4<2>(p, z, ld, row, ids);
        else if (E <= 128) pick_experts4<4>(p, z, ld, row, ids);
        else pick_experts4<8>(p, z, ld, row, ids);
    } else
        for (int r = warp; r < kRtRows; r += kRtWarps)
            if (row0 + r < p.rows) pick_experts(p, rt_z + r * ld, row0 + r, ids_s + r * p.m.top);
    // places in the buckets: counted in shared memory, one global addition per expert and CTA
    int32_t* count = reinterpret_cast<int32_t*>(ring);    // [experts] | [experts] first place
    for (int e = tid; e < E; e += kRtThreads) count[e] = 0;
    __syncthreads();
    const int left = p.rows - row0 < kRtRows ? (int)(p.rows - row0) : kRtRows;
    for (int i = tid; i < left * p.m.top; i += kRtThreads) place_s[i] = atomicAdd(count + ids_s[i], 1);
    __syncthreads();
    for (int e = tid; e < E; e += kRtThreads)
        if (count[e] > 0) count[E + e] = atomicAdd(p.counts + e, count[e]);
    __syncthreads();
    for (int i = tid; i < left * p.m.top; i += kRtThreads) {
        const int e = ids_s[i], at = count[E + e] + place_s[i];
        if (at < p.rows) p.bucket[(int64_t)e * p.rows + at] = (int32_t)(row0 * p.m.top + i);
    }
}

}  // namespace ktk

using namespace ktk;

static int check_moe(const ktk_moe* m, int64_t rows, const char* who) {
    if (m == nullptr || rows < 0 || m->experts <= 0 || m->top <= 0 || m->top > m->experts || m->width <= 0 ||
        m->ff <= 0 || m->width_stride < m->width || m->ff_stride < m->ff || m->width_stride % 8 != 0 ||
        m->ff_stride % 8 != 0 || (m->dtype != KTK_F32 && m->dtype != KTK_BF16) ||
        m->scoring < 0 || m->scoring > 1 || !(m->limit > 0.0f)) {
        set_error("%s: bad sizes", who);
        return KTK_ERR_ARG;
    }
    if (m->experts > kMaxExperts || rows > 2147483647LL / m->top || rows > 65535LL * 1024) {
        set_error("%s: at most %d experts; %lld rows", who, kMaxExperts, (long long)rows);
        return KTK_ERR_TOO_LARGE;
    }
    return KTK_OK;
}

extern "C" int ktk_moe_route(const void* h, const void* w, const float* b, int32_t* ids, float* weights,
                             int32_t* counts, int32_t* bucket, int64_t rows, const ktk_moe* shape, int32_t variant,
                             void* stream) {
    const char* who = "ktk_moe_route";
    const int rc = check_moe(shape, rows, who);
    if (rc != KTK_OK) return rc;
    if (rows == 0) return KTK_OK;
    if (!h || !w || !ids || !weights || !counts || !bucket || (((uintptr_t)h | (uintptr_t)w) & 15u) != 0) {
        set_error("%s: null or misaligned pointer", who);
        return KTK_ERR_ARG;
    }
    const RouteParams p{*shape, h, w, b, ids, weights, counts, bucket, rows};
    cudaStream_t st = (cudaStream_t)stream;
    const bool by_row = shape->dtype == KTK_F32 || variant == KTK_VARIANT_SIMT ||
                        (variant == KTK_VARIANT_AUTO && (rows <= kRtByRow || shape->top > 64));
    if (by_row) {
        const size_t smem = ((shape->experts + 3) / 4 * 4 + shape->width_stride + shape->top) * sizeof(float);
        if (smem > 200 * 1024) { set_error("%s: rows of %d columns", who, shape->width); return KTK_ERR_UNSUPPORTED; }
        auto kernel = shape->dtype == KTK_F32 ? route_row_kernel<float> : route_row_kernel<__nv_bfloat16>;
        KTK_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem), who);
        kernel<<<(unsigned)rows, kRtRowThreads, smem, st>>>(p);
    } else {
        const size_t ring = (size_t)kRtStageElems * 2;    // of a stage
        const size_t rest = (size_t)kRtRows * ((shape->experts + kRtCols - 1) / kRtCols * kRtCols) * sizeof(float) +
                            (size_t)2 * kRtRows * shape->top * sizeof(int32_t);
        const int stages = rest + 3 * ring <= 227 * 1024 ? 3 : 2;
        const size_t smem = rest + stages * ring;
        if (rest > kRtMostRest) {
            set_error("%s: top %d of %d experts", who, shape->top, shape->experts);
            return KTK_ERR_UNSUPPORTED;
        }
        auto kernel = stages == 3 ? route_mma_kernel<3> : route_mma_kernel<2>;
        KTK_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem), who);
        kernel<<<(unsigned)((rows + kRtRows - 1) / kRtRows), kRtThreads, smem, st>>>(p);
    }
    KTK_CUDA_TRY(cudaGetLastError(), who);
    return KTK_OK;
}

extern "C" int ktk_moe_gemm(int32_t stage, const void* in, const void* w, void* out, const float* weights,
                            const int32_t* counts, const int32_t* bucket, int64_t rows, const ktk_moe* shape,
                            int32_t variant, int32_t* status, void* stream) {
    const char* who = "ktk_moe_gemm";
    const int rc = check_moe(shape, rows, who);
    if (rc != KTK_OK) return rc;
    if (stage != 0 && stage != 1) { set_error("%s: stage %d", who, stage); return KTK_ERR_ARG; }
    if (rows == 0) return KTK_OK;
    if (!in || !w || !out || !counts || !bucket || (stage == 1 && !weights) ||
        (((uintptr_t)in | (uintptr_t)w | (uintptr_t)out) & 15u) != 0) {
        set_error("%s: null or misaligned pointer", who);
        return KTK_ERR_ARG;
    }
    if (variant == KTK_VARIANT_UMMA && !moe_umma_supported(*shape)) {
        set_error("%s: variant %d is not built for this case", who, variant);
        return KTK_ERR_UNSUPPORTED;
    }
    const MoeParams p{*shape, in, w, out, weights, counts, bucket, rows, status};
    return variant != KTK_VARIANT_SIMT && moe_umma_supported(*shape) ? launch_moe_umma(stage, p, (cudaStream_t)stream)
                                                                     : launch_moe_simt(stage, p, (cudaStream_t)stream);
}
