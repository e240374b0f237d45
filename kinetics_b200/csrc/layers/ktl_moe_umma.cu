// The experts' matrix products on the fifth-generation tensor cores, for prompts and for decode steps alike.
//
// The weights are the M operand and the routed rows the N operand: D[128 weight rows x N rows] += A[128 x 64] . B^T[64
// x N].  A work item is one tile of up to 256 rows of an expert and a block of 128 weight rows (stage 0: the gate and
// the up rows of 64 inner columns, which the copy brings as eight gates, eight ups, and so on).  N
// follows the tile's row count, and the ring's stages shrink with the rows a tile can have: a decode step with a few
// rows per expert keeps many weight tiles in flight and moves little else.  Persistent CTAs; the item list follows
// from the experts' row counts, which each CTA reads and scans itself.  Roles:
//     loading warp      weight tiles by TMA; stage 1 also the rows, which lie in place
//     gathering warps   stage 0: the bucket's rows of h, 16 bytes per cp.async, into the layout of the operand
//     issuing warp      4 x tcgen05.mma per ring stage, accumulators double-buffered in tensor memory (2 x 256 columns)
//     warps 0..3        epilogue of the previous item: activation or routing weight, bf16 rows to their places.  The
//                       accumulators hold the output transposed: 16x256b loads give them as 8 x 8 fragments, gate and up
//                       of a column in one thread, which stmatrix.trans lays down as rows that leave in 16-byte pieces.
//                       Lanes that swapped neighbours and stored 2 or 4 bytes each held the tensor cores up: 8192 rows,
//                       8 of 64 experts, 2048 -> 768 columns 415 + 247 us (stages 0 and 1), 381 + 195 this way.
// Now 354 + 166 us, 1.16 and 1.24 PFLOP/s.  By the counters no unit is full: the tensor pipe is busy 62 and 69 % of the cycles, an SM
// reads 42 and 51 bytes a clock from L2 (of 64; 32 KiB per 64 columns, in stage 0 half of it by cp.async), L2 as a whole runs at 40
// and 45 %.
// Full tiles (prompts) run on pairs of CTAs (cta_group::2): 256 weight rows x 256 routed rows per item, each CTA with its
// half of both in shared memory, which takes a third off the traffic from L2.  The second CTA's issuing warp tells the
// first one's when its part of a stage has landed.
// Every wait is bounded; a wait that runs out ends the CTA's roles, drains the copies in flight and frees tensor
// memory.
#include "../ktk_umma.cuh"
#include "ktl_common.cuh"

namespace ktk {

constexpr int kMuRows = 256;                       // most routed rows of a tile; of a CTA: half of that in a pair
constexpr int kMuK = 64;                           // columns per ring stage
constexpr int kMuMaxStages = 12;
constexpr int kMuABytes = kUmRows * kMuK * 2;      // 16 KiB
constexpr int kMuRing = 200 * 1024;                // bytes for the ring
constexpr int kMuTmemCols = 512;
constexpr int kMuGatherers = 128;                  // threads
constexpr int kMuBox = 32;                         // rows per TMA box of the rows in place

// 64-column chunks of a ring stage.  Waits, votes and copies of a stage take the loading warp 600 clocks, the products of one chunk
// 512: two where it loads both operands (8192 rows, 8 of 64 experts, 768 -> 2048 columns 174 -> 166 us), one where it loads only the
// weights (354 us, with two 359).
__host__ __device__ constexpr int mu_chunks(bool pair, int stage) { return pair && stage == 1 ? 2 : 1; }
// rows of a copy of the rows in place: those of a CTA in a pair, whose tiles are full or nearly so
__host__ __device__ constexpr int mu_box(bool pair) { return pair ? kMuRows / 2 : kMuBox; }

// Position in a ring of `stages` stages: advanced by one, without a division.
struct RingPos {
    int stage = 0;
    uint32_t round = 0;                                      // parity of a full barrier's next phase = round & 1
    __device__ __forceinline__ void next(int stages) {
        if (++stage == stages) { stage = 0; ++round; }
    }
};

// tile_rows: most rows of a tile; cta_rows: of them in a CTA's ring stage (half in a pair)
template <int STAGE, bool PAIR>
__global__ void __launch_bounds__(STAGE == 0 ? 320 : 192, 1)
moe_umma_kernel(const MoeParams p, const int tile_rows, const int cta_rows, const int stages,
                const __grid_constant__ CUtensorMap w_map, const __grid_constant__ CUtensorMap in_map) {
    extern __shared__ uint8_t mu_raw[];
    __shared__ ExpertPlan plan;
    __shared__ __align__(8) uint64_t full[kMuMaxStages], empty[kMuMaxStages], peer_full[kMuMaxStages],
        acc_full[2], acc_free[2];
    __shared__ uint32_t tmem_base_s;
    __shared__ int abort_flag;
    __shared__ __align__(16) uint8_t staged[4][2048];        // a warp's 32 routed rows on their way out
    uint8_t* ring = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(mu_raw) + 1023) & ~uintptr_t(1023));
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int N = STAGE == 0 ? 2 * p.m.ff_stride : p.m.width_stride;       // weight rows
    const int K = STAGE == 0 ? p.m.width_stride : p.m.ff_stride;
    constexpr int kCtas = PAIR ? 2 : 1, kChunks = mu_chunks(PAIR, STAGE);
    const int steps = (K + kChunks * kMuK - 1) / (kChunks * kMuK);
    auto chunks_of = [&](int k) { return kChunks == 2 && (2 * k + 1) * kMuK >= K ? 1 : kChunks; };      // of step k
    constexpr int kPer = kMuRows / kCtas / 16;               // gathered rows per thread
    const int rank = PAIR ? (int)cluster_rank() : 0;
    const int unit = blockIdx.x / kCtas, num_units = gridDim.x / kCtas;
    const int blocks = (N + kCtas * kUmRows - 1) / (kCtas * kUmRows);
    const int chunk_bytes = kMuABytes + cta_rows * 128, stage_bytes = kChunks * chunk_bytes;

    if (tid == 0) {
        for (int s = 0; s < stages; ++s) {
            mbar_init(&full[s], STAGE == 0 ? 1 + kMuGatherers : 1);
            mbar_init(&empty[s], 1);
            mbar_init(&peer_full[s], 1);
        }
        for (int i = 0; i < 2; ++i) { mbar_init(&acc_full[i], 1); mbar_init(&acc_free[i], 4 * kCtas); }
        abort_flag = 0;
        mbar_init_fence();
    }
    if (warp == 0) plan_experts(plan, p.counts, p.m.experts, p.rows, tile_rows);
    if (warp == 4) {
        if (PAIR) tmem_alloc_pair(&tmem_base_s, kMuTmemCols);
        else tmem_alloc(&tmem_base_s, kMuTmemCols);
    }
    tc_fence_before();
    __syncthreads();
    if (PAIR) cluster_sync();                                // both CTAs' barriers are initialised
    tc_fence_after();
    const uint32_t tmem = tmem_base_s;
    const int work = plan.first_tile[p.m.experts] * blocks;

    // item w: expert, first row of the tile within the expert, rows; this CTA's part of the rows (m0, m); its first weight
    // row.  An expert's rows are shared out evenly over its tiles, in multiples of what a matrix instruction takes.
    constexpr int kStep = 16 * kCtas;
    struct Item { int e, r0, n, m0, m, wrow; };
    auto item = [&](int w) {
        Item it;
        const int t = w / blocks;
        it.wrow = ((w - t * blocks) * kCtas + rank) * kUmRows;
        it.e = expert_of_tile(plan, p.m.experts, t);
        const int rows = plan.first_row[it.e + 1] - plan.first_row[it.e];
        const int tiles = plan.first_tile[it.e + 1] - plan.first_tile[it.e];
        const int each = ((rows + tiles - 1) / tiles + kStep - 1) / kStep * kStep;
        it.r0 = (t - plan.first_tile[it.e]) * each;
        it.n = rows - it.r0 < each ? rows - it.r0 : each;
        const int half = (it.n + kStep - 1) / kStep * 16;    // a CTA's share
        it.m0 = rank * half;
        it.m = it.n - it.m0 < half ? (it.n > it.m0 ? it.n - it.m0 : 0) : half;
        return it;                                           // n <= 0 for a tile that the rounding left empty
    };

    if (warp == 5) {
        // ---------------- loads ----------------
        if (lane == 0) { prefetch_tensormap(&w_map); prefetch_tensormap(&in_map); }
        RingPos pos;
        int issued = 0;
        bool alive = true;
        for (int w = unit; w < work && alive; w += num_units) {
            const Item it = item(w);
            if (it.n <= 0) continue;
            const int box = mu_box(PAIR), boxes = STAGE == 0 ? 0 : (it.m + box - 1) / box;
            const uint32_t bytes = (uint32_t)(kMuABytes + boxes * box * 128);
            const int row = plan.first_row[it.e] + it.r0 + it.m0;
            for (int k = 0; k < steps; ++k, ++issued, pos.next(stages)) {
                const int s = pos.stage;
                bool ok = true;
                if (pos.round > 0) ok = mbar_wait_fast(&empty[s], (pos.round - 1) & 1, &abort_flag);
                if (!__all_sync(0xffffffffu, ok)) { alive = false; break; }
                uint8_t* st = ring + s * stage_bytes;
                const int chunks = chunks_of(k);
                if (elect_one()) {
                    mbar_arrive_expect_tx(&full[s], bytes * chunks);
#pragma unroll
                    for (int c = 0; c < kChunks; ++c) {
                        if (c >= chunks) break;
                        uint8_t* at = st + c * chunk_bytes;
                        const int col = (k * kChunks + c) * kMuK;
                        if (STAGE == 0) tma_load_5d(at, &w_map, &full[s], col, 0, 0, it.wrow / 16, it.e);
                        else tma_load_3d(at, &w_map, &full[s], col, it.wrow, it.e);
                        if (STAGE == 1)                      // written out: a copy takes 13 clocks to issue, in a loop 170
#pragma unroll
                            for (int i = 0; i < (PAIR ? 1 : kMuRows / kMuBox); ++i)
                                if (i < boxes) tma_load_3d(at + kMuABytes + i * box * 128, &in_map, &full[s], col, row + i * box, 0);
                    }
                }
                __syncwarp();
            }
        }
        if (!alive && lane == 0) {                           // gave up: the copies in flight still write shared memory
            volatile int never = 0;
            for (int i = issued > stages ? issued - stages : 0; i < issued; ++i)
                mbar_wait(&full[i % stages], (i / stages) & 1, &never);
        }
    } else if (STAGE == 0 && warp >= 6) {
        // ---------------- gathered rows: thread t copies chunk t % 8 of rows t / 8, + 16, ... ----------------
        const int t = tid - 192, chunk = t & 7, row0 = t >> 3;
        const char* base = (const char*)p.in + chunk * 16;
        const uint32_t dst0 = smem_u32(ring) + kMuABytes + swz(row0, chunk);     // + i * 2048: row0 + 16 i
        RingPos pos;
        bool alive = true;
        int next[kPer];                                      // bucket entries of the next item, fetched one item ahead
        auto fetch = [&](int w) {
            Item it;
            it.n = it.m = 0;
            while (w < work && (it = item(w)).n <= 0) w += num_units;
#pragma unroll
            for (int i = 0; i < kPer; ++i) {
                const int r = row0 + 16 * i;
                next[i] = r < it.m ? p.bucket[(int64_t)it.e * p.rows + it.r0 + it.m0 + r] : -1;
            }
        };
        fetch(unit);
        for (int w = unit; w < work && alive; w += num_units) {
            const Item it = item(w);
            if (it.n <= 0) continue;
            uint32_t off[kPer];                              // 16-byte pieces from `base`; rows outside: zeros
            uint32_t bytes[kPer];
#pragma unroll
            for (int i = 0; i < kPer; ++i) {
                off[i] = 0u;
                bytes[i] = 0u;
                if (16 * i < it.m && next[i] >= 0) {
                    off[i] = (uint32_t)(next[i] / p.m.top) * (uint32_t)(K / 8);
                    bytes[i] = 16u;
                }
            }
            fetch(w + num_units);
            for (int k = 0; k < steps; ++k, pos.next(stages)) {
                const int s = pos.stage;
                bool ok = true;
                if (pos.round > 0) ok = mbar_wait_fast(&empty[s], (pos.round - 1) & 1, &abort_flag);
                if (!__all_sync(0xffffffffu, ok)) { alive = false; break; }
                static_assert(STAGE == 1 || kChunks == 1, "a stage of gathered rows is one chunk");
                const uint32_t dst = dst0 + s * stage_bytes;
                const bool in_row = k * kMuK + chunk * 8 < K;
                const char* from = in_row ? base + (int64_t)k * (kMuK * 2) : base;
                const uint32_t on = in_row ? 16u : 0u;
#pragma unroll
                for (int i = 0; i < kPer; ++i)
                    if (16 * i < it.m)                       // uniform
                        cp_async16(dst + i * 2048, from + (uint64_t)off[i] * 16, bytes[i] & on);
                cp_async_arrive(&full[s]);
            }
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
    } else if (warp == 4) {
        // ---------------- tensor cores ----------------
        RingPos pos;
        bool alive = true;
        auto landed = [&](uint64_t* bar) {
            return __all_sync(0xffffffffu, mbar_wait_fast(bar, pos.round & 1, &abort_flag)) != 0;
        };
        // One look for both, a lane each: two waits one behind the other take longer than the matrix instructions in the queue.  What a lane
        // saw land is ordered before the other lanes' instructions by the __syncwarp; the ballot orders no memory.
        auto both_landed = [&](uint64_t* a, uint64_t* b) {
            for (uint32_t i = 0; i < (1u << 24); ++i) {
                if ((__ballot_sync(0xffffffffu, mbar_test(lane == 0 ? a : b, pos.round & 1)) & 3u) == 3u) {
                    __syncwarp();
                    return true;
                }
                if ((i & 63u) == 63u && __any_sync(0xffffffffu, *(volatile int*)&abort_flag)) return false;
            }
            abort_flag = 1;
            return false;
        };
        if (PAIR && rank == 1) {
            // the second CTA of a pair only reports what has landed
            for (int w = unit; w < work && alive; w += num_units) {
                if (item(w).n <= 0) continue;
                for (int k = 0; k < steps; ++k, pos.next(stages)) {
                    if (!landed(&full[pos.stage])) { alive = false; break; }
                    if (STAGE == 0) fence_proxy_async();
                    if (elect_one()) mbar_arrive_at(&peer_full[pos.stage], 0);
                    __syncwarp();
                }
            }
        } else {
            int j = 0;
            const uint64_t a0 = umma_desc(smem_u32(ring), 0, 1024), b0 = umma_desc(smem_u32(ring) + kMuABytes, 0, 1024);
            for (int w = unit; w < work && alive; w += num_units) {
                const Item it = item(w);
                if (it.n <= 0) continue;
                const int cols = (it.n + kStep - 1) / kStep * kStep;
                const uint32_t idesc = PAIR ? umma_idesc_pair(cols) : umma_idesc(cols, false);
                const int buf = j & 1;
                const uint32_t d = tmem + buf * 256;
                if (j >= 2 && !__all_sync(0xffffffffu, mbar_wait_fast(&acc_free[buf], ((j >> 1) - 1) & 1, &abort_flag)))
                    break;
                tc_fence_after();
                for (int k = 0; k < steps; ++k, pos.next(stages)) {
                    const int s = pos.stage;
                    if (PAIR ? !both_landed(&full[s], &peer_full[s]) : !landed(&full[s])) { alive = false; break; }
                    if (STAGE == 0) fence_proxy_async();     // the gathered rows came through the generic proxy
                    tc_fence_after();
                    const uint64_t a = umma_desc_at(a0, s * stage_bytes), b = umma_desc_at(b0, s * stage_bytes);
                    const int chunks = chunks_of(k);
                    if (elect_one()) {
#pragma unroll
                        for (int c = 0; c < kChunks; ++c) {
                            if (c >= chunks) break;
#pragma unroll
                            for (int q = 0; q < kMuK / 16; ++q) {
                                const uint32_t more = (k > 0 || c > 0 || q > 0) ? 1u : 0u, at = c * chunk_bytes + q * 32;
                                if (PAIR) umma_f16_pair(d, umma_desc_at(a, at), umma_desc_at(b, at), idesc, more);
                                else umma_f16(d, umma_desc_at(a, at), umma_desc_at(b, at), idesc, more);
                            }
                        }
                        if (PAIR) umma_commit_pair(&empty[s]);
                        else umma_commit(&empty[s]);
                        if (k + 1 == steps) {
                            if (PAIR) umma_commit_pair(&acc_full[buf]);
                            else umma_commit(&acc_full[buf]);
                        }
                    }
                    __syncwarp();
                }
                ++j;
            }
        }
    } else if (warp < 4) {
        // ---------------- epilogue ----------------
        const uint32_t lanes = tmem + ((uint32_t)(warp * 32) << 16);
        __nv_bfloat16* out = (__nv_bfloat16*)p.out;
        const int out_cols = STAGE == 0 ? p.m.ff_stride : p.m.width_stride;
        const uint32_t st = smem_u32(staged[warp]);
        int j = 0;
        for (int w = unit; w < work; w += num_units) {
            const Item it = item(w);
            if (it.n <= 0) continue;
            const int buf = j & 1;
            int entry[kMuRows / 32];
            float weight[kMuRows / 32];
            if (STAGE == 1) {                                // in flight while the tensor cores work on the item
#pragma unroll
                for (int c = 0; c < kMuRows / 32; ++c) {
                    const int r = c * 32 + lane;
                    entry[c] = r < it.n ? p.bucket[(int64_t)it.e * p.rows + it.r0 + r] : 0;
                }
#pragma unroll
                for (int c = 0; c < kMuRows / 32; ++c) weight[c] = c * 32 < it.n ? p.weights[entry[c]] : 0.0f;
            }
            const bool ok = mbar_wait_fast(&acc_full[buf], (j >> 1) & 1, &abort_flag);
            if (!__all_sync(0xffffffffu, ok)) break;
            tc_fence_after();
            // first column of the output that this warp's 32 weight rows give
            const int col0 = STAGE == 0 ? (it.wrow >> 1) + warp * 16 : it.wrow + warp * 32;
#pragma unroll
            for (int ch = 0; ch < kMuRows / 32; ++ch) {
                const int c0 = ch * 32;
                if (c0 >= it.n) break;                       // uniform for the CTA
                uint32_t v[32];                              // [16 weight rows][8 routed rows]: an 8 x 8 matrix per two registers
                tmem_ld_rows32(lanes + buf * 256 + c0, v);
                if (STAGE == 0) {
#pragma unroll
                    for (int k = 0; k < 4; k += 2) {
                        uint32_t m[4];                       // (routed rows 8 (k + i / 2) .., inner columns 8 (i % 2) ..)
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            const uint32_t* x = v + 16 * (i & 1) + 4 * (k + (i >> 1));      // gate, gate, up, up
                            m[i] = pack_bf16(
                                gated<true>(__uint_as_float(x[0]), __uint_as_float(x[2]), p.m.limit, p.m.slope, p.m.shift),
                                gated<true>(__uint_as_float(x[1]), __uint_as_float(x[3]), p.m.limit, p.m.slope, p.m.shift));
                        }
                        const int row = 8 * (k + (lane >> 4)) + (lane & 7), chunk = (lane >> 3) & 1;
                        stmatrix_x4_trans(st + row * 32 + ((chunk ^ ((row >> 2) & 1)) << 4), m);
                    }
                } else {
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        const float w0 = __shfl_sync(0xffffffffu, weight[ch], 8 * k + 2 * (lane & 3));
                        const float w1 = __shfl_sync(0xffffffffu, weight[ch], 8 * k + 2 * (lane & 3) + 1);
                        uint32_t m[4];                       // (routed rows 8 k .., weight rows 8 i ..)
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            const uint32_t* x = v + 16 * (i >> 1) + 4 * k + 2 * (i & 1);
                            m[i] = pack_bf16(__uint_as_float(x[0]) * w0, __uint_as_float(x[1]) * w1);
                        }
                        const int row = 8 * k + (lane & 7), chunk = lane >> 3;
                        stmatrix_x4_trans(st + row * 64 + ((chunk ^ ((row >> 1) & 3)) << 4), m);
                    }
                }
                __syncwarp();
                constexpr int kPieces = STAGE == 0 ? 2 : 4;  // 16-byte pieces of a row
#pragma unroll
                for (int i = 0; i < kPieces; ++i) {
                    const int row = lane / kPieces + i * (32 / kPieces), chunk = lane % kPieces;
                    const int place = STAGE == 0 ? chunk ^ ((row >> 2) & 1) : chunk ^ ((row >> 1) & 3);
                    const uint4 x = *reinterpret_cast<const uint4*>(staged[warp] + row * (kPieces * 16) + place * 16);
                    const int64_t dst = STAGE == 0 ? plan.first_row[it.e] + it.r0 + c0 + row
                                                   : __shfl_sync(0xffffffffu, entry[ch], row);
                    const int col = col0 + chunk * 8;
                    if (c0 + row < it.n && col < out_cols) *reinterpret_cast<uint4*>(out + dst * out_cols + col) = x;
                }
                __syncwarp();
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) {
                if (PAIR) mbar_arrive_at(&acc_free[buf], 0);
                else mbar_arrive(&acc_free[buf]);
            }
            ++j;
        }
    }
    tc_fence_before();
    __syncthreads();
    if (PAIR) cluster_sync();                                // neither CTA leaves while the other may use its memory
    if (abort_flag && tid == 0) report(p.status, KTK_STATUS_TIMEOUT);
    if (warp == 4) {
        __syncwarp();
        if (PAIR) tmem_free_pair(tmem, kMuTmemCols);
        else tmem_free(tmem, kMuTmemCols);
    }
}

bool moe_umma_supported(const ktk_moe& m) { return m.dtype == KTK_BF16; }

template <int STAGE> static int moe_umma(const MoeParams& p, cudaStream_t st) {
    const char* who = "ktk_moe_gemm";
    const uint64_t N = STAGE == 0 ? 2 * p.m.ff_stride : p.m.width_stride;
    const uint64_t K = STAGE == 0 ? p.m.width_stride : p.m.ff_stride;
    const int64_t routed = p.rows * p.m.top;
    CUtensorMap w_map, in_map;
    int rc;
    if (STAGE == 0) {
        // Rows 16 b + 2 j + i of the matrix (i: gate, up) come as rows 16 b + 8 i + j of the operand: of every 16 lanes of
        // the accumulators the first eight then hold the gates, the others the ups, as the epilogue's registers want them.
        const uint64_t wd[5] = {K, 8, 2, N / 16, (uint64_t)p.m.experts}, ws[4] = {K * 4, K * 2, K * 32, K * N * 2};
        const uint32_t wb[5] = {kMuK, 8, 2, kUmRows / 16, 1};
        rc = make_tensor_map(&w_map, p.w, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 5, wd, ws, wb, CU_TENSOR_MAP_SWIZZLE_128B, who);
    } else {
        const uint64_t wd[3] = {K, N, (uint64_t)p.m.experts}, ws[2] = {K * 2, K * N * 2};
        const uint32_t wb[3] = {kMuK, kUmRows, 1};
        rc = make_tensor_map_3d(&w_map, p.w, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, wd, ws, wb, CU_TENSOR_MAP_SWIZZLE_128B, who);
    }
    if (rc != KTK_OK) return rc;
    // tiles for twice the rows that an expert has on average (and never more than all of them): the ring's stages are
    // no larger than they have to be
    int64_t most = 2 * ((routed + p.m.experts - 1) / p.m.experts);
    if (most > p.rows) most = p.rows;
    const int tile_rows = (int)(most >= kMuRows ? kMuRows : (most + kMuBox - 1) / kMuBox * kMuBox);
    const bool pair = tile_rows == kMuRows;
    const int cta_rows = pair ? tile_rows / 2 : tile_rows;
    const uint64_t id[3] = {K, (uint64_t)(STAGE == 0 ? p.rows : routed), 1}, is[2] = {K * 2, K * id[1] * 2};
    const uint32_t ib[3] = {kMuK, (uint32_t)mu_box(pair), 1};
    rc = make_tensor_map_3d(&in_map, p.in, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, id, is, ib, CU_TENSOR_MAP_SWIZZLE_128B, who);
    if (rc != KTK_OK) return rc;
    const int stage_bytes = mu_chunks(pair, STAGE) * (kMuABytes + cta_rows * 128);
    const int stages = kMuRing / stage_bytes < kMuMaxStages ? kMuRing / stage_bytes : kMuMaxStages;
    const int ctas = pair ? 2 : 1;
    const int64_t per = (N + ctas * kUmRows - 1) / (ctas * kUmRows);
    const int64_t tiles = routed / tile_rows + (routed < p.m.experts ? routed : p.m.experts);
    if (tiles * per > 2147483647LL || p.rows * (int64_t)(K / 8) > 4294967295LL) {
        set_error("%s: too many rows", who);
        return KTK_ERR_TOO_LARGE;
    }
    const int64_t units = tiles * per < sm_count() / ctas ? tiles * per : sm_count() / ctas;
    auto kernel = pair ? moe_umma_kernel<STAGE, true> : moe_umma_kernel<STAGE, false>;
    KTK_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kMuRing + 1024), who);
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)(units * ctas));
    cfg.blockDim = dim3(STAGE == 0 ? 320 : 192);
    cfg.dynamicSmemBytes = (size_t)stages * stage_bytes + 1024;
    cfg.stream = st;
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = ctas;
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = pair ? 1 : 0;
    KTK_CUDA_TRY(cudaLaunchKernelEx(&cfg, kernel, p, tile_rows, cta_rows, stages, w_map, in_map), who);
    return KTK_OK;
}

int launch_moe_umma(int stage, const MoeParams& p, cudaStream_t st) {
    return stage == 0 ? moe_umma<0>(p, st) : moe_umma<1>(p, st);
}

}  // namespace ktk
