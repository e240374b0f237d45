// Causal attention of a prompt's tokens over keys and values expanded from latents: per head an unrotated key and a value
// of its own, one rotated key part for all heads; a sink in the denominator, a gate on the output.  bf16 on the
// fifth-generation tensor cores, fp32 scores and sums.
//
// One CTA per (head, two tiles of 128 tokens): both tiles share every block of 128 keys that comes in by TMA: the unrotated columns
// of the head, then the shared rotated ones.  The softmax and the order of the matrix instructions: ktk_flash.cuh.
// 8192 tokens, 32 heads of 128 + 64 and 128 columns in a model: 694 us (990 TFLOP/s), 899 us with blocks of 64 keys.  Heads are walked
// in groups whose keys and values fit L2, so that the CTAs left for the end are short ones.
#include "../ktk_flash.cuh"
#include "ktl_score.cuh"

namespace ktk {

constexpr int kAeKeys = 128;
constexpr int kAeMaxChunks = 4;               // of the key: 64 columns each
constexpr int64_t kAeGroupBytes = 48 << 20;   // keys and values that the CTAs of a wave share through L2 (126 MB)

struct ExpandedParams {
    ktk_latent a;
    const __nv_bfloat16* q;
    int64_t q_stride;
    int n, total;
    const float* sink;
    const __nv_bfloat16* gate;
    int64_t gate_stride;
    __nv_bfloat16* o;
    int32_t* status;
};

// heads_per: heads whose tiles are walked together, those with the longest history first
template <int VC, int NK>
__global__ void __launch_bounds__(kFlThreads, 1)
attn_expanded_kernel(const ExpandedParams p, const int heads_per, const __grid_constant__ CUtensorMap k_map,
                     const __grid_constant__ CUtensorMap r_map, const __grid_constant__ CUtensorMap v_map) {
    extern __shared__ uint8_t ae_raw[];
    __shared__ __align__(8) FlashShared sh;
    using F = Flash<kAeKeys, VC, NK>;
    const ktk_latent& a = p.a;
    const int nc = (a.dim_stride + 63) / 64, dc = nc + (a.rot_stride + 63) / 64;     // chunks of a key
    uint8_t* sm = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(ae_raw) + 1023) & ~uintptr_t(1023));

    const int tid = threadIdx.x, warp = tid >> 5;
    // CTA -> (group of heads, tile pair from the last, head of the group)
    const int pairs = (p.n + 2 * kUmRows - 1) / (2 * kUmRows);
    const int group = (int)(blockIdx.x / ((unsigned)heads_per * pairs)), head0 = group * heads_per;
    const int here = a.heads - head0 < heads_per ? a.heads - head0 : heads_per;
    const int at = (int)(blockIdx.x - (unsigned)head0 * pairs);
    const int head = head0 + at % here;
    const int tok0 = (pairs - 1 - at / here) * 2 * kUmRows;
    const int base = p.total - p.n;
    int keys[2];                                        // keys of each tile
#pragma unroll
    for (int m = 0; m < 2; ++m) {
        const int t0 = tok0 + m * kUmRows, t1 = t0 + kUmRows < p.n ? t0 + kUmRows : p.n;
        keys[m] = t0 < p.n ? base + t1 : 0;
    }
    const int tile = warp >> 2, row = tid & (kUmRows - 1);
    const int tok = tok0 + tile * kUmRows + row;
    const bool row_on = warp < 8 && tok < p.n;
    const int vis = row_on ? base + tok + 1 : 0;        // keys at positions < vis are seen

    F fl(sh, sm, dc, dc, keys[0], keys[1]);
    // warp 9; columns and tokens outside come as zeros
    auto load_k = [&](int blk, uint8_t* dst, uint64_t* bar) {
        if (elect_one()) {
            mbar_arrive_expect_tx(bar, (uint32_t)(dc * F::kTile));
            for (int c = 0; c < dc; ++c) {
                if (c < nc) tma_load_3d(dst + c * F::kTile, &k_map, bar, c * 64, head, blk * kAeKeys);
                else tma_load_3d(dst + c * F::kTile, &r_map, bar, (c - nc) * 64, 0, blk * kAeKeys);
            }
        }
        __syncwarp();
    };
    auto load_v = [&](int blk, uint8_t* dst, uint64_t* bar) {
        if (elect_one()) {
            mbar_arrive_expect_tx(bar, (uint32_t)F::kVBuf);
#pragma unroll
            for (int c = 0; c < VC; ++c) tma_load_3d(dst + c * F::kTile, &v_map, bar, c * 64, head, blk * kAeKeys);
        }
        __syncwarp();
    };
    if (warp < 8) {
        fl.queries(tile, [&](int r, int chunk, int i) -> const uint4* {
            const int t = tok0 + tile * kUmRows + r;
            const bool rot = chunk >= nc;
            const int col = (rot ? chunk - nc : chunk) * 64 + i * 8;
            if (t >= p.n || col >= (rot ? a.rot_stride : a.dim_stride)) return nullptr;
            return reinterpret_cast<const uint4*>(p.q + t * p.q_stride + (int64_t)head * (a.dim_stride + a.rot_stride) +
                                                  (rot ? a.dim_stride : 0) + col);
        });
    } else if (warp == 8) {
        tmem_alloc(&sh.tmem, kFlTmemCols);
    } else if (warp == 9) {
        if (elect_one()) {
            prefetch_tensormap(&k_map);
            prefetch_tensormap(&r_map);
            prefetch_tensormap(&v_map);
            sh.init();
        }
        __syncwarp();
        fl.first_copies(load_k, load_v);
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();

    if (warp >= kFlSoftmaxWarps) {
        fewer_registers();
        if (warp == 8) {
            const int ksteps = (a.dim_stride + 15) / 16, rsteps = (a.rot_stride + 15) / 16;
            fl.issue([&](int c) { return c < nc ? (ksteps - 4 * c < 4 ? ksteps - 4 * c : 4)
                                                : (rsteps - 4 * (c - nc) < 4 ? rsteps - 4 * (c - nc) : 4); },
                     0, (a.vdim_stride + 15) / 16 * 16);
        } else if (warp == 9) {
            fl.copy(load_k, load_v);
        }
    } else {
        more_registers();
        const int tile_min_vis = base + tok0 + tile * kUmRows + 1;
        float m_ref = p.sink ? p.sink[head] * kLog2eF : -INFINITY, l_run = p.sink ? 1.0f : 0.0f;
        const bool done = fl.template softmax<false>(tile, a.scale * kLog2eF, m_ref, l_run, [&](float (&s)[kAeKeys], int j) {
            if ((j + 1) * kAeKeys > tile_min_vis) {                       // some row of the tile does not see the whole block
                const int lim = vis - j * kAeKeys;
#pragma unroll
                for (int c = 0; c < kAeKeys; ++c) s[c] = c < lim ? s[c] : -INFINITY;
            }
            return false;
        }, [](float&, float&) {}, [](int) {});
        if (done && fl.blocks_of(tile) > 0) {
            float g = l_run > 0.0f ? 1.0f / l_run : 0.0f;
            if (row_on && p.gate) g *= sigmoid_f(__bfloat162float(p.gate[(int64_t)tok * p.gate_stride + head]));
            const uint32_t o_at = sh.tmem + ((uint32_t)((warp & 3) * 32) << 16) + kFlColO + tile * 128;
            __nv_bfloat16* dst = p.o + ((int64_t)tok * a.heads + head) * a.vdim_stride;
#pragma unroll
            for (int c = 0; c < VC * 64; c += 32) {
                float o[32];
                tmem_ld32(o_at + c, o);
#pragma unroll
                for (int i = 0; i < 32; i += 8)
                    if (row_on && c + i < a.vdim_stride) {
                        float e[8];
#pragma unroll
                        for (int x = 0; x < 8; ++x) e[x] = o[i + x] * g;
                        Vec8<__nv_bfloat16>::store(dst + c + i, e);
                    }
                __syncwarp();
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (sh.abort && tid == 0) report(p.status, KTK_STATUS_TIMEOUT);
    if (warp == 8) {
        __syncwarp();
        tmem_free(sh.tmem, kFlTmemCols);
    }
}

// The rows of one sequence out of their pages, in order: 16 bytes per thread.
__global__ void __launch_bounds__(256)
gather_rows_kernel(const uint4* __restrict__ pages, uint4* __restrict__ out, const ktk_paged t, int pieces, int total, int32_t* status) {
    const Span s = span_of(t, 0);
    if (s.bad || s.total < total) {
        if (threadIdx.x == 0) report(status, KTK_STATUS_BAD_TABLE);
        return;
    }
    const int64_t n = (int64_t)total * pieces;
    for (int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x; i < n; i += (int64_t)gridDim.x * 256) {
        const int tok = (int)(i / pieces), c = (int)(i - (int64_t)tok * pieces);
        const int64_t page = t.kv_indices[s.start + tok / t.page_size];
        if (page < 0 || page >= t.num_pages) { report(status, KTK_STATUS_BAD_PAGE); continue; }
        out[i] = pages[(page * t.page_size + tok % t.page_size) * pieces + c];
    }
}

static int chunks_of(const ktk_latent& a) { return (a.dim_stride + 63) / 64 + (a.rot_stride + 63) / 64; }

template <int VC, int NK>
static int expanded_launch(const ExpandedParams& p, const __nv_bfloat16* kv, const __nv_bfloat16* rows, cudaStream_t st) {
    const char* who = "ktk_expanded_attention";
    const ktk_latent& a = p.a;
    const uint64_t H = a.heads, line = H * (a.dim_stride + a.vdim_stride) * 2, row = (uint64_t)(a.rank_stride + a.rot_stride) * 2;
    CUtensorMap km, rm, vm;
    const uint32_t box[3] = {64, 1, kAeKeys};
    // innermost first: columns of a head, heads, tokens
    const uint64_t kd[3] = {(uint64_t)a.dim_stride, H, (uint64_t)p.total}, ks[2] = {(uint64_t)a.dim_stride * 2, line};
    const uint64_t vd[3] = {(uint64_t)a.vdim_stride, H, (uint64_t)p.total}, vs[2] = {(uint64_t)a.vdim_stride * 2, line};
    const uint64_t rd[3] = {(uint64_t)a.rot_stride, 1, (uint64_t)p.total}, rs[2] = {row, row};
    int rc = make_tensor_map_3d(&km, kv, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, kd, ks, box, CU_TENSOR_MAP_SWIZZLE_128B, who);
    if (rc == KTK_OK)
        rc = make_tensor_map_3d(&vm, kv + H * a.dim_stride, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, vd, vs, box,
                                CU_TENSOR_MAP_SWIZZLE_128B, who);
    if (rc == KTK_OK)
        rc = make_tensor_map_3d(&rm, rows + a.rank_stride, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, rd, rs, box,
                                CU_TENSOR_MAP_SWIZZLE_128B, who);
    if (rc != KTK_OK) return rc;
    const int dc = chunks_of(a), smem = Flash<kAeKeys, VC, NK>::bytes(dc, dc);
    const int64_t pairs = ((int64_t)p.n + 2 * kUmRows - 1) / (2 * kUmRows), per_head = (int64_t)p.total * (a.dim_stride + a.vdim_stride) * 2;
    int64_t heads_per = kAeGroupBytes / per_head;
    heads_per = heads_per < 1 ? 1 : (heads_per > a.heads ? a.heads : heads_per);
    auto kernel = attn_expanded_kernel<VC, NK>;
    KTK_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem), who);
    kernel<<<(unsigned)(pairs * a.heads), kFlThreads, smem, st>>>(p, (int)heads_per, km, rm, vm);
    KTK_CUDA_TRY(cudaGetLastError(), who);
    return KTK_OK;
}

static bool expanded_supported(const ktk_latent& a) {
    return a.dtype == KTK_BF16 && a.rot_stride > 0 && a.scale > 0.0f && chunks_of(a) <= kAeMaxChunks && a.vdim_stride <= 128 && a.heads <= 65535;
}

}  // namespace ktk

using namespace ktk;

extern "C" int ktk_expanded_attention_supported(const ktk_latent* shape) {
    return check_latent(shape, "ktk_expanded_attention_supported") == KTK_OK && expanded_supported(*shape) ? 1 : 0;
}

extern "C" int ktk_gather_rows(const void* pages, void* out, int64_t total, int32_t row_bytes, const ktk_paged* table,
                               int32_t* status, void* stream) {
    const char* who = "ktk_gather_rows";
    if (total < 0 || total > 2147483647LL || row_bytes <= 0 || row_bytes % 16 != 0 || table == nullptr || table->batch != 1 ||
        table->page_size <= 0 || (total > 0 && (!pages || !out || (((uintptr_t)pages | (uintptr_t)out) & 15u) != 0))) {
        set_error("%s: total=%lld row_bytes=%d", who, (long long)total, row_bytes);
        return KTK_ERR_ARG;
    }
    if (total == 0) return KTK_OK;
    const int pieces = row_bytes / 16;
    const int64_t blocks = (total * pieces + 255) / 256, cap = (int64_t)sm_count() * 16;
    gather_rows_kernel<<<(unsigned)(blocks < cap ? blocks : cap), 256, 0, (cudaStream_t)stream>>>(
        (const uint4*)pages, (uint4*)out, *table, pieces, (int)total, status);
    KTK_CUDA_TRY(cudaGetLastError(), who);
    return KTK_OK;
}

extern "C" int ktk_expanded_attention(const void* q, int64_t q_stride, int64_t rows, int64_t total, const void* kv,
                                      const void* latents, const float* sink, const void* gate, int64_t gate_stride, void* o,
                                      const ktk_latent* shape, int32_t* status, void* stream) {
    const char* who = "ktk_expanded_attention";
    const int rc = check_latent(shape, who);
    if (rc != KTK_OK) return rc;
    if (!expanded_supported(*shape)) { set_error("%s: not built for these sizes", who); return KTK_ERR_UNSUPPORTED; }
    if (rows < 0 || total < rows || total > (1 << 30) || q_stride % 8 != 0 ||
        q_stride < (int64_t)shape->heads * (shape->dim_stride + shape->rot_stride) || (gate && gate_stride < shape->heads)) {
        set_error("%s: %lld rows of %lld, stride %lld", who, (long long)rows, (long long)total, (long long)q_stride);
        return KTK_ERR_ARG;
    }
    if (rows == 0) return KTK_OK;
    if (!q || !kv || !latents || !o || (((uintptr_t)q | (uintptr_t)kv | (uintptr_t)latents | (uintptr_t)o) & 15u) != 0) {
        set_error("%s: null or misaligned pointer", who);
        return KTK_ERR_ARG;
    }
    const ExpandedParams p{*shape, (const __nv_bfloat16*)q, q_stride, (int)rows, (int)total, sink, (const __nv_bfloat16*)gate,
                           gate_stride, (__nv_bfloat16*)o, status};
    // Queries of four chunks leave room for one buffer of K: the next block comes in during the softmax of this one.  4000 keys, 32
    // CTAs: 121 us with blocks of 64 keys and two buffers.
    const bool wide = chunks_of(*shape) > 3;
    auto launch = shape->vdim_stride <= 64 ? (wide ? expanded_launch<1, 1> : expanded_launch<1, 2>)
                                           : (wide ? expanded_launch<2, 1> : expanded_launch<2, 2>);
    return launch(p, (const __nv_bfloat16*)kv, (const __nv_bfloat16*)latents, (cudaStream_t)stream);
}
