// Causal attention of a prompt's tokens on the fifth-generation tensor cores: two softmax maps per head over shared
// values, head sizes up to 128, softcap, query temperature; the difference of the maps and its unit norm in the
// epilogue.  bf16 operands, fp32 scores and sums.
//
// One CTA per (sequence, kv head, tile of 128 (token, head of the group) rows).  A row exists once per map: the two tiles of
// ktk_flash.cuh are the two maps, each with keys of its own; a block is 128 keys of both maps and their values.
// With a softcap the exponentials have a fixed reference (ktl_score.cuh): nothing is ever rescaled.  Without one (or
// with a large one) the reference is the first block's maximum until half a block's sum passes 2^8 (ktk_flash.cuh).
// Bound by what the softmax issues: 8192 tokens, 16 heads of 2 x 64 and 128 columns, softcap: 523 us, 792 us with blocks of
// 64 keys.
#include "../ktk_flash.cuh"
#include "ktl_score.cuh"

namespace ktk {

constexpr int kAuKeys = 128;

__device__ __forceinline__ void st_row16(__nv_bfloat16* d, const float* o, float f) {
    uint4 v;
    v.x = pack_bf16(o[0] * f, o[1] * f);
    v.y = pack_bf16(o[2] * f, o[3] * f);
    v.z = pack_bf16(o[4] * f, o[5] * f);
    v.w = pack_bf16(o[6] * f, o[7] * f);
    *reinterpret_cast<uint4*>(d) = v;
}

// TILE_MAJOR: the grid is (kv heads, sequences, tiles), so that the last tiles of all heads and sequences, which see most of their own
// sequence, come first; otherwise (tiles, kv heads, sequences), for more than 65535 tiles
template <int DC, int VC, bool FIXED, bool TILE_MAJOR>
__global__ void __launch_bounds__(kFlThreads, 1)
attn_umma_kernel(const AttnParams p, const __grid_constant__ CUtensorMap k_map, const __grid_constant__ CUtensorMap v_map) {
    extern __shared__ uint8_t au_raw[];
    __shared__ __align__(8) FlashShared sh;
    using F = Flash<kAuKeys, VC>;
    uint8_t* sm = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(au_raw) + 1023) & ~uintptr_t(1023));

    const ktk_attn& a = p.a;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int b = TILE_MAJOR ? blockIdx.y : blockIdx.z, kvh = TILE_MAJOR ? blockIdx.x : blockIdx.y;
    const int group = a.heads / a.kv_heads, tpc = kUmRows / group;
    const int q0 = p.new_indptr[b], n_new = p.new_indptr[b + 1] - q0;
    const int tok0 = (TILE_MAJOR ? (int)(gridDim.z - 1 - blockIdx.z) : (int)(gridDim.x - 1 - blockIdx.x)) * tpc;
    if (tok0 >= n_new) return;                          // uniform for the CTA: nothing allocated yet
    const Span s = span_of(p.t, b);
    const int base_pos = s.total - n_new;
    if (s.bad || base_pos < 0) {
        if (tid == 0) report(p.status, KTK_STATUS_BAD_TABLE);
        return;
    }
    const int tok_hi = (tok0 + tpc < n_new ? tok0 + tpc : n_new) - 1;
    const int seen = base_pos + tok_hi + 1;             // keys the tile's last row sees
    const int ps = p.t.page_size;

    const int map = warp >> 2, row = tid & (kUmRows - 1);
    const int my_tok = tok0 + row / group, my_head = kvh * group + row % group;
    const bool row_on = warp < 8 && row / group < tpc && my_tok < n_new;
    const int vis = row_on ? base_pos + my_tok + 1 : 0; // keys at positions < vis are seen

    F fl(sh, sm, DC, 2 * DC, seen, seen);
    // warp 9.  A box is a page of one head (of one map); lane i: page i of a block
    const int pages = kAuKeys / ps, box = ps * 128;
    auto load = [&](int blk, int which, uint8_t* dst, uint64_t* bar) {
        const int tok = blk * kAuKeys + lane * ps;
        const int64_t pg = lane < pages && tok < seen ? p.t.kv_indices[s.start + tok / ps] : -1;
        const bool on = pg >= 0 && pg < p.t.num_pages;
        if (lane < pages && tok < seen && !on) report(p.status, KTK_STATUS_BAD_PAGE);
        const uint32_t n = __popc(__ballot_sync(0xffffffffu, on));
        if (lane == 0) {
            if (n) mbar_arrive_expect_tx(bar, n * (uint32_t)((which ? VC : 2 * DC) * box));
            else mbar_arrive(bar);
        }
        __syncwarp();
        if (on && which) {
    #pragma unroll
            for (int c = 0; c < VC; ++c)
                tma_load_3d(dst + c * F::kTile + lane * box, &v_map, bar, c * 64, 0, (int)(pg * a.kv_heads) + kvh);
        } else if (on) {
    #pragma unroll
            for (int mc = 0; mc < 2 * DC; ++mc)
                tma_load_3d(dst + mc * F::kTile + lane * box, &k_map, bar, (mc % DC) * 64, 0,
                            (int)(pg * (2 * a.kv_heads)) + kvh * 2 + mc / DC);
        }
        __syncwarp();
    };
    auto load_k = [&](int blk, uint8_t* dst, uint64_t* bar) { load(blk, 0, dst, bar); };
    auto load_v = [&](int blk, uint8_t* dst, uint64_t* bar) { load(blk, 1, dst, bar); };
    if (warp < 8) {
        const int per = (65536 + group - 1) / group;            // r / group = r per / 65536 for r (group - 1) < 65536
        fl.queries(map, [&](int r, int chunk, int i) -> const uint4* {
            const int at = r * per >> 16, t = tok0 + at, col = chunk * 64 + i * 8;
            if (at >= tpc || t >= n_new || col >= a.dim_stride) return nullptr;
            return reinterpret_cast<const uint4*>((const __nv_bfloat16*)p.q + (int64_t)(q0 + t) * p.q_stride +
                                                  ((int64_t)(kvh * group + r - at * group) * 2 + map) * a.dim_stride + col);
        });
    } else if (warp == 8) {
        tmem_alloc(&sh.tmem, kFlTmemCols);
    } else if (warp == 9) {
        if (lane == 0) {
            prefetch_tensormap(&k_map);
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
            const int ksteps = (a.dim_stride + 15) / 16;
            fl.template issue<true>([&](int c) { return ksteps - 4 * c < 4 ? ksteps - 4 * c : 4; }, DC * F::kTile, (a.vdim_stride + 15) / 16 * 16);
        } else if (warp == 9) {
            fl.copy(load_k, load_v);
        }
    } else {
        more_registers();
        const float factor = a.scale * query_temperature(a.temp_coef, a.temp_every, vis > 0 ? vis - 1 : 0);
        const bool capped = FIXED || a.softcap > 0.0f;
        const float plain = factor * kLog2eF;
        CapPoly poly;
        CapCoef exact;
        poly.set(factor, capped ? a.softcap : 1.0f);
        exact.set(factor, capped ? a.softcap : 1.0f);
        const int tile_min_vis = base_pos + tok0 + 1;
        auto prepare = [&](float (&v)[kAuKeys], int j) {
            const bool masked = (j + 1) * kAuKeys > tile_min_vis;      // some row of the tile does not see the whole block
            if (capped) {
                float mx[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
                for (int c = 0; c < kAuKeys; c += 8)
#pragma unroll
                    for (int i = 0; i < 4; ++i) mx[i] = max3(mx[i], fabsf(v[c + i]), fabsf(v[c + 4 + i]));
                // rows without a token and keys behind a row's own hold stale numbers: they decide the branch at most
                if (__any_sync(0xffffffffu, !(max3(fmaxf(mx[0], mx[1]), mx[2], mx[3]) <= poly.limit))) {
#pragma unroll
                    for (int c = 0; c < kAuKeys; ++c) v[c] = exact(v[c]);
                } else if (FIXED && !masked) {
                    return true;                                       // beside the exponentials
                } else {
#pragma unroll
                    for (int c = 0; c < kAuKeys; c += 2) poly.two(v[c], v[c + 1]);
                }
            } else {
#pragma unroll
                for (int c = 0; c < kAuKeys; ++c) v[c] *= plain;
            }
            if (masked) {
                const int lim = vis - j * kAuKeys;
#pragma unroll
                for (int c = 0; c < kAuKeys; ++c) v[c] = c < lim ? v[c] : -INFINITY;
            }
            return false;
        };
        auto clear = [&](int j) {                                      // the last block: rows of V without a key
            if ((j + 1) * kAuKeys > seen) fl.clear_rows(map, j, [&](int r) { return j * kAuKeys + r < seen; });
        };
        float m_ref = -INFINITY, l_run = 0.0f;
        fl.template softmax<FIXED>(map, 1.0f, m_ref, l_run, prepare, [&](float& x, float& y) { poly.two(x, y); }, clear);
        // ---- o = O_1 / l_1 - lambda O_2 / l_2, unit norm: warps 0..3 the first half of the columns, 4..7 the second.
        // Row sums go over the queries, which each map's last block has read.
        float* row_l = reinterpret_cast<float*>(fl.q + map * DC * kFlQTile);
        const float* other = reinterpret_cast<const float*>(fl.q + (map ^ 1) * DC * kFlQTile);
        row_l[row] = l_run;
        asm volatile("bar.sync 1, 256;" ::: "memory");
        constexpr int kHalf = VC * 32;
        const float l1 = map ? other[row] : l_run, l2 = map ? l_run : other[row];
        const float i1 = l1 > 0.0f ? 1.0f / l1 : 0.0f, i2 = l2 > 0.0f ? a.lambda / l2 : 0.0f;
        const uint32_t o_at = sh.tmem + ((uint32_t)((warp & 3) * 32) << 16) + kFlColO + map * kHalf;
        float o[kHalf], ss = 0.0f;
        const bool ok = sh.abort == 0;                  // tensor memory holds both maps' results
        if (__all_sync(0xffffffffu, ok)) {
            tc_fence_after();
#pragma unroll
            for (int c = 0; c < kHalf; c += 32) {
                float t1[32], t2[32];
                tmem_ld32(o_at + c, t1);
                tmem_ld32(o_at + 128 + c, t2);
#pragma unroll
                for (int i = 0; i < 32; ++i) {
                    o[c + i] = map * kHalf + c + i < a.vdim ? t1[i] * i1 - t2[i] * i2 : 0.0f;
                    ss += o[c + i] * o[c + i];
                }
            }
        }
        row_l[kUmRows + row] = ss;
        asm volatile("bar.sync 1, 256;" ::: "memory");
        if (row_on && ok) {
            const float f = a.out_scale / sqrtf((map ? other[kUmRows + row] + ss : ss + other[kUmRows + row]) / (float)a.vdim + a.eps);
            __nv_bfloat16* dst = (__nv_bfloat16*)p.o + ((int64_t)(q0 + my_tok) * a.heads + my_head) * a.vdim_stride;
#pragma unroll
            for (int c = 0; c < kHalf; c += 8)
                if (map * kHalf + c < a.vdim_stride) st_row16(dst + map * kHalf + c, o + c, f);
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

bool attn_umma_supported(const ktk_attn& a) {
    return a.dtype == KTK_BF16 && a.maps == 2 && a.dim_stride <= 128 && a.vdim_stride <= 128 &&
           a.heads / a.kv_heads <= kUmRows;
}

template <int DC, int VC, bool FIXED> static int umma_launch(const AttnParams& p, cudaStream_t st) {
    const char* who = "ktk_paged_attention";
    CUtensorMap km, vm;
    const int rc = make_cache_maps(p, &km, &vm, (uint32_t)p.t.page_size, who);
    if (rc != KTK_OK) return rc;
    using F = Flash<kAuKeys, VC>;
    constexpr int smem = F::bytes(DC, 2 * DC);
    const int tpc = kUmRows / (p.a.heads / p.a.kv_heads);
    const unsigned tiles = (unsigned)(((int64_t)p.max_new + tpc - 1) / tpc), heads = (unsigned)p.a.kv_heads, batch = (unsigned)p.t.batch;
    const bool tile_major = tiles <= 65535;
    auto kernel = tile_major ? attn_umma_kernel<DC, VC, FIXED, true> : attn_umma_kernel<DC, VC, FIXED, false>;
    KTK_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem), who);
    kernel<<<tile_major ? dim3(heads, batch, tiles) : dim3(tiles, heads, batch), kFlThreads, smem, st>>>(p, km, vm);
    KTK_CUDA_TRY(cudaGetLastError(), who);
    return KTK_OK;
}

int launch_attn_umma(const AttnParams& p, cudaStream_t st) {
    if (p.max_new <= 0) return KTK_OK;
    if (p.t.batch > 65535 || p.a.kv_heads > 65535) {
        set_error("ktk_paged_attention: more than 65535 sequences or kv heads in one launch");
        return KTK_ERR_TOO_LARGE;
    }
    const bool d1 = p.a.dim_stride <= 64, v1 = p.a.vdim_stride <= 64, fx = fixed_reference(p.a);
    if (d1 && v1) return fx ? umma_launch<1, 1, true>(p, st) : umma_launch<1, 1, false>(p, st);
    if (d1) return fx ? umma_launch<1, 2, true>(p, st) : umma_launch<1, 2, false>(p, st);
    return fx ? umma_launch<2, 2, true>(p, st) : umma_launch<2, 2, false>(p, st);
}

}  // namespace ktk
