// Causal prefill attention over the paged KV cache on the fifth-generation tensor cores (tcgen05, accumulators
// in tensor memory).  Same contract as prefill_mma_kernel (ktk_prefill.cu); replaces
// flashinfer.single_prefill_with_kv_cache of LiteSys/litesys/attention/batch_cache.py:129-145.
//
// One CTA per (sequence, kv head, two tiles of 128 / G new tokens); the 128 rows of a tile are the (token, head of the query
// group) pairs.  Both tiles share every block of 128 keys (eight pages, 16-row x 128-byte boxes under the 128-byte swizzle, which
// is the operand layout tcgen05.mma reads).  The softmax and the order of the matrix instructions: ktk_flash.cuh.
// Bound by the chain of a tile's block: matrix instructions, softmax, matrix instructions.  8192 tokens, 32 heads over 8 kv
// heads: 489 us (1124 TFLOP/s), 855 us with one tile per CTA, blocks of 64 keys and two CTAs per SM.
#include "ktk_decode_mma.cuh"
#include "ktk_flash.cuh"
#include "ktk_prefill_umma.cuh"

namespace ktk {

constexpr int kPuKeys = 128;
constexpr int kPuPages = kPuKeys / kPageSize;             // of a block
using PrefillFlash = Flash<kPuKeys, kHeadDim / 64>;
constexpr int kPuSmem = PrefillFlash::bytes(2, 2);

// Which tiles a CTA takes.  A later tile sees more keys, and the work of a launch that leaves SMs idle at its end should end with
// short ones.
//   kByTile       grid (kv heads, sequences, tile pairs): the last pairs of all heads and sequences first
//   kByEither     the same grid; where histories differ, the items of all sequences from the most keys to the fewest
//   kBySequence   grid (tile pairs, kv heads, sequences), for more than 65535 pairs
enum Order { kBySequence, kByTile, kByEither };
constexpr int kPuOrdered = 32;                            // sequences that an ordered launch may have: one per lane

// Item `rank` of the launch: a sequence and which `step` of its new tokens.  Its length counts in steps, those of the history rounded
// up: item p of a sequence with h of history has length p + h.  Lane s brings sequence s: its new tokens (0 behind the last) and its history.
// A warp finds the length at `rank`, 32 probes at a time.  The sequence * 65536 + the step, or -1 behind the last item.  A call, so that
// launches without it do not fetch it (one to two us a CTA: 32 portions of 40 tokens 23.2 us, 27 with it).
__device__ __noinline__ int item_by_length(int rank, int step, int batch, int n, int history) {
    const int lane = threadIdx.x & 31, count = (n + step - 1) / step, first = n > 0 ? (history + step - 1) / step : 0;
    // items of length L or more, every lane for its own L; all lanes take part
    auto at_least = [&](int L) {
        int have = 0;
        for (int s = 0; s < batch; ++s) {
            const int f = __shfl_sync(0xffffffffu, first, s), c = __shfl_sync(0xffffffffu, count, s);
            have += min(max(f + c - L, 0), c);
        }
        return have;
    };
    int lo = 0, hi = (int)__reduce_max_sync(0xffffffffu, (unsigned)(first + count)), behind = 0;
    // more than `rank` items have length lo or more, `behind` <= rank of them hi or more
    for (bool begun = false; hi - lo > 1 || !begun; begun = true) {
        const int each = (hi - lo + 31) / 32, L = lo + lane * each, seen = at_least(L), have = L < hi ? seen : behind;
        const unsigned more = __ballot_sync(0xffffffffu, L < hi && have > rank);       // a prefix of the lanes
        if (more == 0) return -1;                          // only of the first probes, which start at 0
        const int at = 31 - __clz((int)more);
        const int next = __shfl_sync(0xffffffffu, have, at < 31 ? at + 1 : 31);
        if (at < 31 && lo + (at + 1) * each < hi) { hi = lo + (at + 1) * each; behind = next; }
        lo += at * each;
    }
    // among the sequences with an item of length lo
    const unsigned has = __ballot_sync(0xffffffffu, lo >= first && lo < first + count);
    const bool mine = (has >> lane & 1u) && __popc(has & ((1u << lane) - 1u)) == rank - behind;
    const int b = __ffs((int)__ballot_sync(0xffffffffu, mine)) - 1;
    return b * 65536 + lo - __shfl_sync(0xffffffffu, first, b);
}

// Whether a launch in either order goes by length, and the CTA's item if so.  Histories, counted in whole pages, that lie within a
// quarter of the longest sequence are left in the order of the tiles, which is that of the lengths or close to it.
__device__ __forceinline__ bool item_of_either(const PrefillUmmaParams& p, int& item) {
    const int lane = threadIdx.x & 31, seq = lane < p.batch ? lane : p.batch - 1;
    const int n = p.q_indptr[seq + 1] - p.q_indptr[seq];
    const int tokens = (p.page_count ? p.page_count[seq] : p.kv_indptr[seq + 1] - p.kv_indptr[seq]) * kPageSize;
    const int history = tokens > n ? tokens - n : 0;
    const int longest = (int)__reduce_max_sync(0xffffffffu, (unsigned)(n > 0 ? history + n : 0));
    const int spread = (int)(__reduce_max_sync(0xffffffffu, n > 0 ? (unsigned)history : 0u) -
                             __reduce_min_sync(0xffffffffu, n > 0 ? (unsigned)history : 0x7fffffffu));
    if (spread <= longest / 4) return false;               // the same for all CTAs
    item = item_by_length(blockIdx.z * gridDim.y + blockIdx.y, p.tiles * (kUmRows / p.G), p.batch, lane < p.batch && n > 0 ? n : 0, history);
    return true;
}

template <Order ORDER>
__global__ void __launch_bounds__(kFlThreads, 1)
prefill_umma_kernel(const PrefillUmmaParams p, const __grid_constant__ CUtensorMap kv_map) {
    extern __shared__ uint8_t um_raw[];
    __shared__ __align__(8) FlashShared sh;
    uint8_t* sm = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(um_raw) + 1023) & ~uintptr_t(1023));

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int h = ORDER == kBySequence ? blockIdx.y : blockIdx.x;
    int b = ORDER == kBySequence ? blockIdx.z : blockIdx.y;
    int pair = ORDER == kBySequence ? (int)(gridDim.x - 1 - blockIdx.x) : (int)(gridDim.z - 1 - blockIdx.z);
    int item;
    if (ORDER == kByEither && item_of_either(p, item)) {
        if (item < 0) return;
        b = item >> 16;
        pair = item & 65535;
    }
    const int q0 = p.q_indptr[b], n_new = p.q_indptr[b + 1] - q0;
    const SeqPages sp = seq_pages(p.kv_indptr, p.page_count, p.kv_last_page_len, p.sink_tokens, b);
    const int G = p.G, Hq = p.Hkv * G;
    const int tpc = kUmRows / G;                    // new tokens per tile
    const int tok0 = pair * p.tiles * tpc;
    if (tok0 >= n_new) return;                      // uniform for the CTA: nothing allocated yet

    const int base_pos = sp.total - n_new;          // position of the sequence's first new token
    if (sp.bad || base_pos < 0) {
        if (tid == 0) report(p.status, KTK_STATUS_BAD_TABLE);
        return;
    }
    const int shift = kPageSize - sp.first_fill;    // slots of the first page that never hold a token
    int keys[2], n_need = 0;                        // key columns of each tile; pages that the last row sees
#pragma unroll
    for (int m = 0; m < 2; ++m) {
        const int t0 = tok0 + m * tpc, t1 = t0 + tpc < n_new ? t0 + tpc : n_new;
        keys[m] = 0;
        if (m < p.tiles && t0 < n_new) {
            int unused;
            pages_for(base_pos + t1, sp.first_fill, n_need, unused);
            if (n_need > sp.n_pages) n_need = sp.n_pages;
            keys[m] = n_need * kPageSize;
        }
    }

    // a softmax thread's row
    const int tile = warp >> 2, row = tid & (kUmRows - 1);
    const int my_tok = tok0 + tile * tpc + row / G, my_head = h * G + row % G;
    const bool row_on = warp < 8 && tile < p.tiles && my_tok < n_new;
    const int vis = row_on ? base_pos + my_tok + 1 : 0;     // keys at positions < vis are seen

    PrefillFlash fl(sh, sm, 2, 2, keys[0], keys[1]);
    // warp 9.  Lane i < 8: page i of a block; entries are read one block ahead of their first use
    auto entry = [&](int blk) {
        const int e = blk * kPuPages + lane;
        return lane < kPuPages && e < n_need ? p.kv_indices[sp.start + e] : -1;
    };
    int at[3], first = 0;                           // of blocks first, first + 1, first + 2
    auto load = [&](int blk, int which, uint8_t* dst, uint64_t* bar) {
        while (first + 2 < blk || (which && first < blk)) {
            at[0] = at[1];
            at[1] = at[2];
            ++first;
            at[2] = entry(first + 2);
        }
        const int pg = blk == first ? at[0] : (blk == first + 1 ? at[1] : at[2]);
        const bool on = pg >= 0 && pg < p.num_pages;
        if (which == 0 && !on && lane < kPuPages && blk * kPuPages + lane < n_need) report(p.status, KTK_STATUS_BAD_PAGE);
        const uint32_t pages = __popc(__ballot_sync(0xffffffffu, on));
        if (lane == 0) {
            if (pages) mbar_arrive_expect_tx(bar, pages * (2u * kPageSize * 128u));
            else mbar_arrive(bar);
        }
        __syncwarp();
        if (on) {
            const int z = pg * (2 * kPageSize) + which * kPageSize;      // token row of slot 0
            tma_load_3d(dst + lane * (kPageSize * 128), &kv_map, bar, 0, h, z);
            tma_load_3d(dst + PrefillFlash::kTile + lane * (kPageSize * 128), &kv_map, bar, 64, h, z);
        }
        __syncwarp();
    };
    auto load_k = [&](int blk, uint8_t* dst, uint64_t* bar) { load(blk, 0, dst, bar); };
    auto load_v = [&](int blk, uint8_t* dst, uint64_t* bar) { load(blk, 1, dst, bar); };
    if (warp < 8) {
        const int shift_g = 31 - __clz(G);              // 1, 2, 4 or 8
        if (fl.blocks_of(tile) > 0) fl.queries(tile, [&](int r, int chunk, int i) -> const uint4* {
            const int t = tok0 + tile * tpc + (r >> shift_g);
            if (t >= n_new) return nullptr;
            const int64_t q_row = (int64_t)(q0 + t) * Hq + h * G + (r & (G - 1));
            return reinterpret_cast<const uint4*>((const __nv_bfloat16*)p.q + q_row * kHeadDim) + chunk * 8 + i;
        });
    } else if (warp == 8) {
        tmem_alloc(&sh.tmem, kFlTmemCols);
    } else if (warp == 9) {
        if (lane == 0) {
            prefetch_tensormap(&kv_map);
            sh.init();
        }
#pragma unroll
        for (int i = 0; i < 3; ++i) at[i] = entry(i);
        __syncwarp();
        fl.first_copies(load_k, load_v);
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();

    if (warp >= kFlSoftmaxWarps) {
        fewer_registers();
        if (warp == 8) {
            fl.issue([](int) { return 4; }, 0, kHeadDim);
        } else if (warp == 9) {
            fl.copy(load_k, load_v);
        }
    } else {
        more_registers();
        const int tile_min_vis = base_pos + tok0 + tile * tpc + 1;
        auto prepare = [&](float (&s)[kPuKeys], int j) {
            // column c of block j: position j * 128 + c - shift, but for the first page's own
            if ((j + 1) * kPuKeys - shift > tile_min_vis || (j == 0 && shift > 0)) {       // uniform for the tile
                const int lim = (j == 0 && vis <= sp.first_fill) ? vis : vis + shift - j * kPuKeys;
#pragma unroll
                for (int c = 0; c < kPuKeys; ++c) s[c] = c < lim ? s[c] : -INFINITY;
                if (j == 0 && shift > 0) {
#pragma unroll
                    for (int c = 0; c < kPageSize; ++c) s[c] = c < sp.first_fill ? s[c] : -INFINITY;
                }
            }
            return false;
        };
        // the rows of V that hold no key: pages that are not read, the places of a page that is not full
        auto clear = [&](int j) {
            const int e0 = j * kPuPages, e1 = e0 + kPuPages;
            if (e1 <= n_need && !(e0 == 0 && shift > 0) && !(e1 == sp.n_pages && sp.last_fill != kPageSize)) return;
            fl.clear_rows(tile, j, [&](int r) {
                const int e = e0 + r / kPageSize, slot = r % kPageSize;
                return e < n_need && slot < (e == sp.n_pages - 1 ? sp.last_fill : (e == 0 ? sp.first_fill : kPageSize));
            });
        };
        float m_ref = -INFINITY, l_run = 0.0f;
        const bool done = fl.softmax<false>(tile, p.scale_log2, m_ref, l_run, prepare, [](float&, float&) {}, clear);
        if (done && fl.blocks_of(tile) > 0) {
            const float inv = l_run > 0.0f ? 1.0f / l_run : 0.0f;
            const uint32_t o_at = sh.tmem + ((uint32_t)((warp & 3) * 32) << 16) + kFlColO + tile * 128;
            __nv_bfloat16* dst = (__nv_bfloat16*)p.o + ((int64_t)(q0 + (row_on ? my_tok : 0)) * Hq + my_head) * kHeadDim;
#pragma unroll
            for (int c = 0; c < kHeadDim; c += 32) {
                float o[32];
                tmem_ld32(o_at + c, o);
                if (row_on) {
#pragma unroll
                    for (int i = 0; i < 32; i += 8) {
                        uint4 v;
                        v.x = pack_bf16(o[i] * inv, o[i + 1] * inv);
                        v.y = pack_bf16(o[i + 2] * inv, o[i + 3] * inv);
                        v.z = pack_bf16(o[i + 4] * inv, o[i + 5] * inv);
                        v.w = pack_bf16(o[i + 6] * inv, o[i + 7] * inv);
                        *reinterpret_cast<uint4*>(dst + c + i) = v;
                    }
                }
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

int launch_prefill_umma(PrefillUmmaParams p, int max_new_tokens, cudaStream_t st) {
    const char* who = "ktk_prefill_attention";
    // Two tiles to a CTA share its copies and hide one another's latencies; where all tiles find an SM each, one is faster:
    // 64 tokens of 32 heads over 8 9.7 us, 11.7 with two; 2300 tokens of 8 heads over one 41.6 and 46.3 (144 tiles).
    const int tpc = kUmRows / p.G;
    const int64_t per_seq = ((int64_t)max_new_tokens + tpc - 1) / tpc, most = p.total_new / tpc + p.batch;
    const int64_t tiles = (p.batch * per_seq < most ? p.batch * per_seq : most) * p.Hkv;
    p.tiles = tiles <= sm_count() ? 1 : 2;
    const unsigned pairs = (unsigned)((per_seq + p.tiles - 1) / p.tiles);
    // By length, if histories differ, where several sequences take between one round of CTAs and two and a half: the more rounds, the less
    // the last one leaves idle.  Six portions of 350 to 1050 tokens behind 2500 to 7500, 16 heads over 8: 255 us by tile, 229 by length
    // (280 CTAs); eight of 150 to 450 behind 450 to 1350 59 and 56; the first with 32 heads (544 CTAs) 446 either way.  Where histories do
    // not differ the look costs a CTA half a microsecond: 16 portions of 300 behind 300 60 us, 62 with it.
    const int64_t about = p.total_new / (tpc * p.tiles) + p.batch / 2;
    const bool by_tile = pairs <= 65535;
    const bool either = by_tile && p.batch > 1 && p.batch <= kPuOrdered && about * p.Hkv > sm_count() && 2 * about * p.Hkv <= 5 * (int64_t)sm_count();
    auto kernel = either ? prefill_umma_kernel<kByEither> : by_tile ? prefill_umma_kernel<kByTile> : prefill_umma_kernel<kBySequence>;
    KTK_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kPuSmem), who);
    const dim3 grid = by_tile ? dim3((unsigned)p.Hkv, (unsigned)p.batch, pairs) : dim3(pairs, (unsigned)p.Hkv, (unsigned)p.batch);
    DecodeParams d{};                               // only what the tensor map needs
    d.cache = p.cache; d.Hkv = p.Hkv; d.num_pages = p.num_pages;
    CUtensorMap map;
    const int rc = make_kv_tensor_map(&map, d);
    if (rc != KTK_OK) return rc;
    kernel<<<grid, kFlThreads, kPuSmem, st>>>(p, map);
    KTK_CUDA_TRY(cudaGetLastError(), who);
    return KTK_OK;
}

}  // namespace ktk
