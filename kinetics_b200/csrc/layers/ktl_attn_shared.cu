// Attention of many heads over one cached row per token whose first columns are also the value (attention over
// latents): bf16 on the fifth-generation tensor cores, for decode steps and for short portions of a prompt.
//
// A row is wide (up to 576 columns) and serves every head, so the tokens are the M operand and up to 64 (row, head)
// pairs the N operand; each tile of 64 tokens comes into shared memory once and is used twice:
//     S^T[64 tokens x N]  = K[64 x dim] . Q^T                  A read K-major
//     O^T[vdim x N]      += V^T[vdim x 64] . P                 A = the same tile read MN-major, 128 columns at a time
// Decode steps, balanced: a CTA per SM and chunk of heads; the page lists of all sequences, one behind the other, are cut into
// equal parts, and a CTA walks the pieces of sequences that fall into its part with its ring running on from one to the next.
// Else, and for portions: one CTA per (split of a sequence's tokens, chunk of heads, group of rows).  Roles:
//     loading warp     TMA: tiles of 64 tokens into a ring
//     issuing warps    one for each product
//     softmax warps    warp w holds tokens 16 w .., two per thread; exponentials against a reference per column, at first
//                      the largest of its sink and the first tile's scores, that moves only when a score exceeds it by 2^8
// The sum of a column's weights stays spread over the threads until the end.  Tensor memory: S of two tiles, then
// O^T in blocks of 128 columns of V.  Every wait is bounded.
#include "ktl_score.cuh"

namespace ktk {

constexpr int kAsTok = 64;
constexpr int kAsThreads = 224;               // 4 softmax warps, the loading warp, one that issues each product
constexpr int kAsChunk = kAsTok * 128;        // [64 tokens][64 columns]
constexpr int kAsMaxStages = 8;
constexpr int kAsSmem = 232448 - 2048;        // for Q, the ring and P; static arrays and alignment aside
constexpr int kAsMinTiles = 4;                // a split is not worth less
constexpr int kAsMaxSplits = 256, kAsStartTiles = 5;
constexpr int kAsMaxDim = 576, kAsMaxVdim = 512;
constexpr float kAsSlack = 8.0f;
constexpr float kAsNone = -1e30f;             // reference of a column without a sink

// (row, head) pairs of a CTA: `heads` heads of `rows` rows, N columns
struct Packing { int n, heads, rows, chunks; };
__host__ __device__ inline Packing packing_of(int heads, bool one_row) {
    Packing k;
    k.heads = heads < 64 ? heads : 64;
    k.chunks = (heads + k.heads - 1) / k.heads;
    k.heads = (heads + k.chunks - 1) / k.chunks;
    k.rows = one_row ? 1 : 64 / k.heads;
    const int cols = k.heads * k.rows;
    k.n = cols <= 16 ? 16 : cols <= 32 ? 32 : 64;
    return k;
}

// partial of one (row, head, split): reference, sum, O [vdim_stride]
__host__ __device__ inline int64_t as_partial_floats(int vdim_stride) { return 4 + (int64_t)vdim_stride; }

template <int N> __device__ __forceinline__ void tmem_ld_cols(uint32_t addr, float (&v)[N]) {
    if constexpr (N == 16) tmem_ld16(addr, v);
    else if constexpr (N == 32) tmem_ld32(addr, v);
    else tmem_ld64(addr, *reinterpret_cast<float (*)[32]>(&v[0]), *reinterpret_cast<float (*)[32]>(&v[32]));
}
template <int N> __device__ __forceinline__ void tmem_st_cols(uint32_t addr, const float (&v)[N]) {
    if constexpr (N == 16) tmem_st16(addr, v);
    else {
        tmem_st32(addr, *reinterpret_cast<const float (*)[32]>(&v[0]));
        if constexpr (N == 64) tmem_st32(addr + 32, *reinterpret_cast<const float (*)[32]>(&v[32]));
    }
}
__device__ __forceinline__ bool any_of_softmax_warps(bool x) {
    uint32_t r;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\tbar.red.or.pred q, 1, 128, p;\n\tselp.u32 %0, 1, 0, q;\n\t}"
        : "=r"(r) : "r"((uint32_t)x) : "memory");
    return r != 0;
}
__device__ __forceinline__ void softmax_warps_sync() { asm volatile("bar.sync 1, 128;" ::: "memory"); }

// Balanced: CTA c of `ctas` takes positions [c * chunk, (c + 1) * chunk), a position being an entry of the page lists counted
// from the first one on; chunk is a whole number of tiles.
struct AsCut { int64_t total, chunk; };
__device__ __forceinline__ AsCut as_cut(const ktk_paged& t, int ctas) {
    const int per = kAsTok / t.page_size;
    AsCut c;
    c.total = (int64_t)t.kv_indptr[t.batch] - t.kv_indptr[0];
    c.chunk = ((c.total + ctas - 1) / ctas + per - 1) / per * per;
    if (c.chunk < kAsMinTiles * per) c.chunk = kAsMinTiles * per;
    return c;
}

// Tokens that a CTA runs of one sequence: n tiles from tok0 on; rows from `end` on are not its own (or lie behind the sequence).
struct AsPiece {
    int b, start, tok0, n, end;                          // start: the sequence's first entry
    bool first, whole;                                  // holds the sequence's first token; all of them
};
// The pieces of a CTA in order; the roles walk them each by itself.
struct AsPieces {
    AsPiece one;
    int64_t p0, p1;                                      // balanced: this CTA's positions
    int b;                                               // the next sequence
    bool balanced, left;
    __device__ __forceinline__ bool next(const AttnParams& p, AsPiece& pc) {
        if (!balanced) {
            const bool on = left;
            left = false;
            pc = one;
            return on;
        }
        const int ps = p.t.page_size;
        for (; b < p.t.batch; ++b) {
            const Span s = span_of(p.t, b);
            const int64_t start = (int64_t)s.start - p.t.kv_indptr[0];
            if (start >= p1) break;
            const int64_t lo = p0 > start ? p0 : start, hi = p1 < start + s.pages ? p1 : start + s.pages;
            if (hi <= lo || s.bad || s.total <= 0) continue;             // the combine kernel reports malformed ones
            pc.b = b++;
            pc.start = s.start;
            pc.tok0 = (int)(lo - start) * ps;
            const int64_t end = (hi - start) * ps;
            pc.end = end < s.total ? (int)end : s.total;
            pc.n = (pc.end - pc.tok0 + kAsTok - 1) / kAsTok;
            pc.first = lo == start;
            pc.whole = pc.first && hi == start + s.pages;
            return true;
        }
        return false;
    }
};

// the sequence whose entries contain position q; all lanes of the warp take part, 32 probes per round
__device__ __forceinline__ int as_sequence_at(const ktk_paged& t, int64_t q) {
    const int lane = threadIdx.x & 31;
    const int64_t base = t.kv_indptr[0];
    int lo = 0, hi = t.batch;
    while (hi - lo > 1) {
        const int step = (hi - lo + 31) / 32, at = lo + lane * step;
        const unsigned m = __ballot_sync(0xffffffffu, at < hi && (lane == 0 || (int64_t)t.kv_indptr[at] - base <= q));
        const int k = 31 - __clz((int)m);
        lo += k * step;
        hi = lo + step < hi ? lo + step : hi;
    }
    return lo;
}

template <int N>
__global__ void __launch_bounds__(kAsThreads, 1)
attn_shared_kernel(const AttnParams p, const __grid_constant__ CUtensorMap k_map,
                   const __grid_constant__ CUtensorMap four_map, const int kc, const int stages,
                   const uint32_t tmem_cols) {
    extern __shared__ uint8_t as_raw[];
    // a stage has landed; its first four chunks, and the others, have been read out
    __shared__ __align__(8) uint64_t full[kAsMaxStages], free_[2 * kAsMaxStages], bar_s[2], bar_p[2], bar_o, bar_q;
    __shared__ __align__(16) float ref_s[N], alpha_s[N];
    __shared__ __align__(16) int vis_s[N], off_s[N];
    __shared__ uint32_t tmem_base_s;
    __shared__ int abort_flag;
    uint8_t* sQ = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(as_raw) + 1023) & ~uintptr_t(1023));
    uint8_t* sK = sQ + kc * (N * 128);                  // [stage][chunk]
    const int stage_bytes = kc * kAsChunk;
    uint8_t* sP = sK + stages * stage_bytes;            // [64 tokens][N], rows of 128 bytes
    float* scratch = reinterpret_cast<float*>(sP);

    const ktk_attn& a = p.a;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const bool issuer = warp == 4, loader = warp == 5, scores = warp == 6;
    const Packing pk = packing_of(a.heads, p.new_indptr == nullptr);
    const bool one = pk.rows == 1, balanced = p.splits < 0;
    const int head0 = blockIdx.y * pk.heads, heads = a.heads - head0 < pk.heads ? a.heads - head0 : pk.heads;
    const int ps = p.t.page_size;
    AsPieces pieces;
    pieces.balanced = balanced;
    int first = 0, rows = 1, r0 = 0, base = 0;          // the CTA's first row within the sequence, rows; first row, tokens in front
    if (balanced) {
        const AsCut cut = as_cut(p.t, gridDim.x);
        pieces.p0 = blockIdx.x * cut.chunk;
        pieces.p1 = pieces.p0 + cut.chunk < cut.total ? pieces.p0 + cut.chunk : cut.total;
        if (pieces.p1 <= pieces.p0) return;             // uniform for the CTA: nothing allocated yet
        pieces.b = as_sequence_at(p.t, pieces.p0);
    } else {
        const int groups = p.new_indptr ? (p.max_new + pk.rows - 1) / pk.rows : 1;
        const int b = blockIdx.z / groups;
        r0 = p.new_indptr ? p.new_indptr[b] : b;
        const int n_new = p.new_indptr ? p.new_indptr[b + 1] - r0 : 1;
        first = (int)(blockIdx.z % groups) * pk.rows;
        if (first >= n_new) return;
        rows = n_new - first < pk.rows ? n_new - first : pk.rows;
        const Span s = span_of(p.t, b);
        base = s.total - n_new;
        if (s.bad || base < 0 || s.total <= 0) {
            if (tid == 0) report(p.status, KTK_STATUS_BAD_TABLE);
            return;
        }
        const int seen = base + first + rows;           // tokens the CTA's last row sees
        const int tiles = (seen + kAsTok - 1) / kAsTok, per = (tiles + p.splits - 1) / p.splits, j0 = blockIdx.x * per;
        const int n = (j0 + per < tiles ? j0 + per : tiles) - j0;        // this split's tiles
        pieces.one = AsPiece{b, s.start, j0 * kAsTok, n > 0 ? n : 0, s.total, j0 == 0, p.splits == 1};
        pieces.left = true;
    }

    if (tid == 0) {
        for (int i = 0; i < stages; ++i) mbar_init(&full[i], 1);
        for (int i = 0; i < 2 * stages; ++i) mbar_init(&free_[i], 1);
        mbar_init(&bar_s[0], 1); mbar_init(&bar_s[1], 1);
        mbar_init(&bar_p[0], 128); mbar_init(&bar_p[1], 128);
        mbar_init(&bar_q, 128);
        mbar_init(&bar_o, 1);
        abort_flag = 0;
        mbar_init_fence();
    }
    if (issuer) tmem_alloc(&tmem_base_s, tmem_cols);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_base_s, tmem_o = tmem + 2 * N;
    const int vblocks = (a.vdim_stride + kUmRows - 1) / kUmRows;

    if (scores) {
        // S of every tile as soon as its rows are there and its place in tensor memory has been read.  Its own warp: a look at a
        // barrier waits behind the products that the warp has queued, and one warp for both left the tensor cores idle for
        // 600 clocks between two products.
        const uint32_t idesc = umma_idesc_of(kAsTok, N, false, false);
        const uint64_t q_desc = umma_desc(smem_u32(sQ), 0, 1024), k_desc = umma_desc(smem_u32(sK), 0, 1024);
        int t = 0, st = 0;
        uint32_t par = 0, q_par = 0;
        bool alive = true;
        AsPiece pc;
        while (alive && pieces.next(p, pc)) {
            if (pc.n == 0) continue;
            alive = mbar_wait_all(&bar_q, q_par, &abort_flag);
            q_par ^= 1u;
            fence_proxy_async();                         // Q came through the generic proxy
            for (int i = 0; i < pc.n && alive; ++i, ++t) {
                alive = mbar_wait_all(&full[st], par, &abort_flag);
                if (alive && t >= 2) alive = mbar_wait_all(&bar_p[t & 1], ((t >> 1) - 1) & 1, &abort_flag);
                if (!alive) break;
                tc_fence_after();
                if (elect_one()) {
                    uint64_t ka = umma_desc_at(k_desc, st * stage_bytes), qa = q_desc;
                    const uint32_t d = tmem + (t & 1) * N;
                    for (int c = 0; c < kc; ++c) {       // columns past `dim` are zero in Q and in K
#pragma unroll
                        for (int k = 0; k < 4; ++k)
                            umma_f16(d, umma_desc_at(ka, k * 32), umma_desc_at(qa, k * 32), idesc, (c > 0 || k > 0) ? 1u : 0u);
                        ka = umma_desc_at(ka, kAsChunk);
                        qa = umma_desc_at(qa, N * 128);
                    }
                    umma_commit(&bar_s[t & 1]);
                    if (vblocks <= 2) umma_commit(&free_[2 * st + 1]);                 // no values in these
                }
                __syncwarp();
                if (++st == stages) { st = 0; par ^= 1u; }
            }
        }
    } else if (issuer) {
        const uint32_t idesc = umma_idesc_of(kUmRows, N, true, true);
        const uint64_t v_desc = umma_desc(smem_u32(sK), kAsChunk, 1024), p_desc = umma_desc(smem_u32(sP), 0, 1024);
        const int first_free = vblocks > 1 ? 1 : 0;      // the last block of values in a tile's first four chunks
        int t = 0, st = 0;
        bool alive = true;
        AsPiece pc;
        while (alive && pieces.next(p, pc)) {
            for (int i = 0; i < pc.n; ++i, ++t) {
                alive = mbar_wait_all(&bar_p[t & 1], (t >> 1) & 1, &abort_flag);
                if (!alive) break;
                tc_fence_after();
                if (elect_one()) {
                    uint64_t va = umma_desc_at(v_desc, st * stage_bytes);
                    uint32_t d = tmem_o;
                    for (int v = 0; v < vblocks; ++v, d += N, va = umma_desc_at(va, 2 * kAsChunk)) {
#pragma unroll
                        for (int k = 0; k < kAsTok / 16; ++k)
                            umma_f16(d, umma_desc_at(va, k * (16 * 128)), umma_desc_at(p_desc, k * (16 * 128)), idesc,
                                     (i > 0 || k > 0) ? 1u : 0u);
                        if (v == first_free) umma_commit(&free_[2 * st]);
                    }
                    if (vblocks > 2) umma_commit(&free_[2 * st + 1]);
                    umma_commit(&bar_o);
                }
                __syncwarp();
                if (++st == stages) st = 0;
            }
        }
    } else if (loader) {
        const int per = kAsTok / ps;                     // pages of a tile: one box of rows each
        int st = 0, issued = 0;
        uint32_t par = 1;
        bool alive = true;
        if (lane == 0) { prefetch_tensormap(&k_map); prefetch_tensormap(&four_map); }
        const int whole = per == 1 ? a.dim_stride / 64 : 0;      // whole chunks of a page that is a tile: four per copy
        auto load_chunks = [&](int c0, int c1, uint8_t* dst, uint64_t* bar, const int (&z)[kAsTok / 16]) {
#pragma unroll
            for (int c = c0; c < c1; ++c)
#pragma unroll
                for (int k = 0; k < kAsTok / 16; ++k)
                    if (c < kc && z[k] >= 0) tma_load_3d(dst + c * kAsChunk + k * ps * 128, &k_map, bar, c * 64, 0, z[k]);
        };
        AsPiece pc;
        while (alive && pieces.next(p, pc)) {
            // page numbers: a lane keeps one of 32, the next 32 on their way
            const int32_t* list = p.t.kv_indices + pc.start + pc.tok0 / ps;
            const int last = pc.tok0 + pc.n * kAsTok < pc.end ? pc.tok0 + pc.n * kAsTok : pc.end;
            const int pages = (last - pc.tok0 + ps - 1) / ps;
            int ids = lane < pages ? list[lane] : -1, next_ids = 32 + lane < pages ? list[32 + lane] : -1;
            for (int i = 0; i < pc.n && alive; ++i) {
                const int e0 = i * per;
                if (i > 0 && (e0 & 31) == 0) {
                    ids = next_ids;
                    next_ids = e0 + 32 + lane < pages ? list[e0 + 32 + lane] : -1;
                }
                int z[kAsTok / 16], have = 0;
#pragma unroll
                for (int k = 0; k < kAsTok / 16; ++k) {
                    const int pg = __shfl_sync(0xffffffffu, ids, (e0 + k) & 31);
                    z[k] = -1;
                    if (k < per && e0 + k < pages) {
                        if (pg < 0 || pg >= p.t.num_pages) { if (lane == 0) report(p.status, KTK_STATUS_BAD_PAGE); }
                        else { z[k] = pg; ++have; }
                    }
                }
                const uint32_t bytes = (uint32_t)(have * ps * 128 * kc);
                uint64_t* bar = &full[st];
                // Two waits a tile and straight code with one lane elected around it: a loop over the chunks behind a branch on the
                // lane number took 470 clocks per 8 KiB (17 bytes a clock and SM), one with a wait per pair of chunks 590 per 16.
                uint8_t* dst = sK + st * stage_bytes;
                if (issued >= stages) alive = mbar_wait_all(&free_[2 * st], par, &abort_flag);
                if (!alive) break;
                if (elect_one()) {
                    if (bytes) mbar_arrive_expect_tx(bar, bytes);
                    else mbar_arrive(bar);
                    if (whole >= 4) {
                        if (z[0] >= 0) tma_load_4d(dst, &four_map, bar, 0, 0, 0, z[0]);
                    } else load_chunks(0, 4, dst, bar, z);
                }
                __syncwarp();
                if (kc > 4) {
                    if (issued >= stages) alive = mbar_wait_all(&free_[2 * st + 1], par, &abort_flag);
                    if (elect_one() && alive) {
                        if (whole >= 8) {
                            if (z[0] >= 0) tma_load_4d(dst + 4 * kAsChunk, &four_map, bar, 0, 0, 4, z[0]);
                            if (kc > 8 && z[0] >= 0) tma_load_3d(dst + 8 * kAsChunk, &k_map, bar, 512, 0, z[0]);
                        } else load_chunks(4, kAsMaxDim / 64, dst, bar, z);
                    }
                    __syncwarp();
                }
                if (!alive) {
                    ++issued;                            // its first half is on its way
                    break;
                }
                ++issued;
                if (++st == stages) { st = 0; par ^= 1u; }
            }
        }
        if (lane == 0 && (abort_flag || !alive)) {           // the copies in flight still write shared memory
            volatile int never = 0;
            for (int i = issued > stages ? issued - stages : 0; i < issued; ++i)
                mbar_wait(&full[i % stages], (i / stages) & 1, &never);
        }
        __syncwarp();
    } else {
        const uint32_t my = tmem + ((uint32_t)(warp * 32) << 16);
        // column c: row first + c / heads of the sequence, head head0 + c % heads.  Q comes while the first tiles are on their
        // way: 8 threads take a column, 16 bytes of every chunk each.  A further piece's Q takes the place of the one before
        // when the last scores are there, under the last values' products.
        auto load_q = [&](const AsPiece& pc) {
            const int64_t row0 = balanced ? pc.b : r0 + first;
            for (int c = tid >> 3; c < N; c += 16) {
                const int lr = one ? 0 : c / pk.heads, h = c - lr * pk.heads;
                const bool on = lr < rows && h < heads;
                const __nv_bfloat16* src = (const __nv_bfloat16*)p.q + (row0 + (on ? lr : 0)) * p.q_stride +
                                           (int64_t)(head0 + (on ? h : 0)) * a.dim_stride + (tid & 7) * 8;
                const uint32_t dst = smem_u32(sQ) + swz(c, tid & 7);
#pragma unroll
                for (int k = 0; k < kAsMaxDim / 64; ++k) {
                    const bool in = on && k * 64 + (tid & 7) * 8 < a.dim_stride;
                    if (k < kc) cp_async16(dst + k * (N * 128), in ? src + k * 64 : (const __nv_bfloat16*)p.q, in ? 16u : 0u);
                }
            }
            cp_async_arrive(&bar_q);
        };
        AsPiece pc, pc_next;
        bool more = pieces.next(p, pc);
        if (more) load_q(pc);
        // a thread holds two tokens of the tile and, of every 8 columns, the two from 2 (lane % 4) on
        const int tok = warp * 16 + (lane >> 2), col = 2 * (lane & 3);
        const float f = a.scale * kLog2eF;
        for (int t0 = 0; more; t0 += pc.n, pc = pc_next) {       // t0: tiles of the pieces before
        const int n = pc.n;
        more = pieces.next(p, pc_next);
        const int clean_end = balanced ? pc.end : base + first + 1;      // tokens before this are seen by every row of the CTA
        for (int c = tid; c < N; c += 128) {
            const int lr = one ? 0 : c / pk.heads, h = c - lr * pk.heads;
            const bool on = lr < rows && h < heads;
            ref_s[c] = on && p.sink ? p.sink[head0 + h] * kLog2eF : kAsNone;
            vis_s[c] = on ? clean_end + lr : 0;
        }
        softmax_warps_sync();
        float l[N / 4];
#pragma unroll
        for (int c = 0; c < N / 4; ++c) l[c] = 0.0f;
        // waits that ran out raise abort_flag; the loop still runs to its end, so that no warp misses a barrier
        for (int j = 0; j < n; ++j) {
            const int nth = t0 + j, tile0 = pc.tok0 + j * kAsTok, at = tile0 + tok;
            mbar_wait_all(&bar_s[nth & 1], (nth >> 1) & 1, &abort_flag);
            tc_fence_after();
            uint32_t raw[N / 2];
            RowPairs<N / 8>::load(my + (nth & 1) * N, raw);
            float t[N / 2];
            bool over = false;
            const bool clean = tile0 + kAsTok <= clean_end;
#pragma unroll
            for (int k = 0; k < N / 8; ++k) {
                const float2 r = *reinterpret_cast<const float2*>(ref_s + 8 * k + col);
                const int2 v = clean ? make_int2(0x7fffffff, 0x7fffffff) : *reinterpret_cast<const int2*>(vis_s + 8 * k + col);
                t[4 * k] = at < v.x ? __uint_as_float(raw[4 * k]) * f : -INFINITY;
                t[4 * k + 1] = at < v.y ? __uint_as_float(raw[4 * k + 1]) * f : -INFINITY;
                t[4 * k + 2] = at + 8 < v.x ? __uint_as_float(raw[4 * k + 2]) * f : -INFINITY;
                t[4 * k + 3] = at + 8 < v.y ? __uint_as_float(raw[4 * k + 3]) * f : -INFINITY;
                over |= fmaxf(t[4 * k], t[4 * k + 2]) > r.x + kAsSlack || fmaxf(t[4 * k + 1], t[4 * k + 3]) > r.y + kAsSlack;
            }
            const bool move = any_of_softmax_warps(over || j == 0);
            if (j > 0) mbar_wait_all(&bar_o, (nth - 1) & 1, &abort_flag);     // P and O of the previous tile are settled
            if (move) {
                // some reference moves: every column's largest score of the tile, then O and the sums are rescaled
#pragma unroll
                for (int k = 0; k < N / 8; ++k)
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        float mx = fmaxf(t[4 * k + e], t[4 * k + 2 + e]);
#pragma unroll
                        for (int o = 4; o <= 16; o <<= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
                        if (lane < 4) scratch[warp * N + 8 * k + col + e] = mx;
                    }
                softmax_warps_sync();
                for (int c = tid; c < N; c += 128) {
                    const float old = ref_s[c];
                    const float mx = fmaxf(fmaxf(scratch[c], scratch[N + c]), fmaxf(scratch[2 * N + c], scratch[3 * N + c]));
                    const float now = fmaxf(mx, old);
                    ref_s[c] = now;
                    alpha_s[c] = ex2(old - now);
                }
                softmax_warps_sync();
                tc_fence_after();
#pragma unroll
                for (int k = 0; k < N / 8; ++k) {
                    const float2 al = *reinterpret_cast<const float2*>(alpha_s + 8 * k + col);
                    l[2 * k] *= al.x;
                    l[2 * k + 1] *= al.y;
                }
                if (j > 0)
                    for (int v = 0; v < vblocks; ++v) {
                        float o[N];
                        tmem_ld_cols<N>(my + 2 * N + v * N, o);
#pragma unroll
                        for (int c = 0; c < N; ++c) o[c] *= alpha_s[c];
                        tmem_st_cols<N>(my + 2 * N + v * N, o);
                    }
                tmem_st_wait();
            }
#pragma unroll
            for (int k = 0; k < N / 8; ++k) {
                const float2 r = *reinterpret_cast<const float2*>(ref_s + 8 * k + col);
                const float p0 = ex2(t[4 * k] - r.x), p1 = ex2(t[4 * k + 1] - r.y);
                const float p2 = ex2(t[4 * k + 2] - r.x), p3 = ex2(t[4 * k + 3] - r.y);
                l[2 * k] += p0 + p2;
                l[2 * k + 1] += p1 + p3;
                *reinterpret_cast<uint32_t*>(sP + swz(tok, k) + 2 * col) = pack_bf16(p0, p1);
                *reinterpret_cast<uint32_t*>(sP + swz(tok + 8, k) + 2 * col) = pack_bf16(p2, p3);
            }
            const int left = pc.end - tile0;
            if (left < kAsTok && lane < 16 && warp * 16 + lane >= left) {
                // rows that no copy has written may hold anything: 0 * x has to stay 0
                uint8_t* st = sK + (nth % stages) * stage_bytes;
                for (int c = 0; c < kc * 8; ++c)
                    *reinterpret_cast<uint4*>(st + (c >> 3) * kAsChunk + swz(warp * 16 + lane, c & 7)) = make_uint4(0u, 0u, 0u, 0u);
            }
            fence_proxy_async();
            tc_fence_before();
            mbar_arrive(&bar_p[nth & 1]);
        }
        if (more) load_q(pc_next);
        if (n > 0) mbar_wait_all(&bar_o, (t0 + n - 1) & 1, &abort_flag);
        tc_fence_after();
        // ---- sums over the tokens, then O^T: lane = column of V, register = (row, head)
#pragma unroll
        for (int k = 0; k < N / 8; ++k)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                float v = l[2 * k + e];
#pragma unroll
                for (int o = 4; o <= 16; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
                if (lane < 4) scratch[warp * N + 8 * k + col + e] = v;
            }
        // partial of head h, row r: (slot0 + r * heads * splits + h * step), in floats of a partial; balanced: two slots per CTA, for
        // a sequence that began before it and for one that goes on behind it
        const int64_t row0 = balanced ? pc.b : r0 + first;
        const int64_t slot0 = balanced ? ((int64_t)blockIdx.x * 2 + (pc.first ? 1 : 0)) * a.heads : row0 * a.heads * p.splits + blockIdx.x;
        const int64_t row_step = balanced ? 0 : (int64_t)a.heads * p.splits, head_step = balanced ? 1 : p.splits;
        for (int c = tid; c < N; c += 128) {              // where the columns go: nowhere, or offsets from the CTA's first
            const int lr = one ? 0 : c / pk.heads, h = c - lr * pk.heads;
            const int64_t to = pc.whole ? (int64_t)(lr * a.heads + h) * a.vdim_stride
                                        : (lr * row_step + h * head_step) * as_partial_floats(a.vdim_stride);
            off_s[c] = h < heads && lr < rows ? (int)to : -1;
        }
        softmax_warps_sync();
        for (int c = tid; c < N; c += 128) {
            float L = scratch[c] + scratch[N + c] + scratch[2 * N + c] + scratch[3 * N + c];
            const int lr = one ? 0 : c / pk.heads, h = head0 + c - lr * pk.heads;
            if (c - lr * pk.heads < heads && lr < rows) {
                const int64_t row = row0 + lr;
                if (!pc.whole) {
                    float* w = p.ws + (slot0 + lr * row_step + h * head_step) * as_partial_floats(a.vdim_stride);
                    w[0] = ref_s[c];
                    w[1] = L;
                } else {
                    if (p.sink) L += ex2(p.sink[h] * kLog2eF - ref_s[c]);
                    float g = L > 0.0f ? 1.0f / L : 0.0f;
                    if (p.gate) g *= sigmoid_f(to_f32(((const __nv_bfloat16*)p.gate)[row * p.gate_stride + h]));
                    alpha_s[c] = g;
                }
            }
        }
        softmax_warps_sync();
        if (n > 0 && !abort_flag) {
            // Predicated stores at tabled offsets: with a row and a head counted along and branched on per column this was 10
            // to 15 us of a call, at 95 to 145 clocks a column.
            float* w = p.ws + (slot0 + head0 * head_step) * as_partial_floats(a.vdim_stride) + 4;
            __nv_bfloat16* out = (__nv_bfloat16*)p.o + (row0 * a.heads + head0) * a.vdim_stride;
#pragma unroll 1
            for (int v = 0; v < vblocks; ++v) {
                const int col = v * kUmRows + tid;
                const bool on = col < a.vdim_stride, zero = col >= a.vdim;
#pragma unroll 1
                for (int c0 = 0; c0 < N; c0 += 16) {
                    float o[16], al[16];
                    int off[16];
#pragma unroll
                    for (int i = 0; i < 16; i += 4) {    // all before the first store, which might alias them
                        *reinterpret_cast<int4*>(off + i) = *reinterpret_cast<const int4*>(off_s + c0 + i);
                        *reinterpret_cast<float4*>(al + i) = *reinterpret_cast<const float4*>(alpha_s + c0 + i);
                    }
                    tmem_ld16(my + 2 * N + v * N + c0, o);
                    if (pc.whole) {
#pragma unroll
                        for (int i = 0; i < 16; ++i)
                            if (on && off[i] >= 0) out[off[i] + col] = __float2bfloat16_rn(zero ? 0.0f : o[i] * al[i]);
                    } else {
#pragma unroll
                        for (int i = 0; i < 16; ++i)
                            if (on && off[i] >= 0) w[off[i] + col] = o[i];
                    }
                    __syncwarp();
                }
            }
        }
        tc_fence_before();                               // the next piece's values overwrite O
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    if (abort_flag && tid == 0) report(p.status, KTK_STATUS_TIMEOUT);
    if (issuer) {
        __syncwarp();
        tmem_free(tmem, tmem_cols);
    }
}

// One CTA per (head, row): merges the splits, adds the sink, applies the gate.
__global__ void __launch_bounds__(128) attn_shared_combine_kernel(const AttnParams p) {
    __shared__ float weight[kAsMaxSplits];
    const ktk_attn& a = p.a;
    const int64_t row = blockIdx.y;
    const int head = blockIdx.x;
    const int64_t stride = as_partial_floats(a.vdim_stride);
    const float* w = p.ws + (row * a.heads + head) * p.splits * stride;
    const float sk = p.sink ? p.sink[head] * kLog2eF : kAsNone;
    // every warp reads all the splits' references and sums, a lane some of them
    const int lane = threadIdx.x & 31;
    float M = sk, L = 0.0f;
    for (int s = lane; s < p.splits; s += 32) {
        const float2 ml = *reinterpret_cast<const float2*>(w + s * stride);
        if (ml.y > 0.0f) M = fmaxf(M, ml.x);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, o));
    for (int s = lane; s < p.splits; s += 32) {
        const float2 ml = *reinterpret_cast<const float2*>(w + s * stride);
        const float f = ml.y > 0.0f ? ex2(ml.x - M) : 0.0f;
        L += f * ml.y;
        if (threadIdx.x < 32) weight[s] = f;
    }
    L = warp_sum_f(L);
    __syncthreads();
    if (p.sink) L += ex2(sk - M);
    float g = L > 0.0f ? 1.0f / L : 0.0f;
    if (p.gate) g *= sigmoid_f(to_f32(((const __nv_bfloat16*)p.gate)[row * p.gate_stride + head]));
    __nv_bfloat16* o = (__nv_bfloat16*)p.o + (row * a.heads + head) * a.vdim_stride;
    for (int c = threadIdx.x * 4; c < a.vdim_stride; c += 512) {
        float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll 4
        for (int s = 0; s < p.splits; ++s) {
            const float f = weight[s];
            if (f == 0.0f) continue;                     // an empty split has written no columns
            const float4 x = *reinterpret_cast<const float4*>(w + s * stride + 4 + c);
            v.x += f * x.x; v.y += f * x.y; v.z += f * x.z; v.w += f * x.w;
        }
        uint2 r;
        r.x = pack_bf16(c < a.vdim ? v.x * g : 0.0f, c + 1 < a.vdim ? v.y * g : 0.0f);
        r.y = pack_bf16(c + 2 < a.vdim ? v.z * g : 0.0f, c + 3 < a.vdim ? v.w * g : 0.0f);
        *reinterpret_cast<uint2*>(o + c) = r;
    }
}

// The same for the pieces of a sequence that the balanced form has cut: a warp per (head, row), as most have two or three.  A
// CTA per (head, row) took 15 us for 128 rows of 32 heads, two pieces each: the latency of the table, of the pieces'
// sums and of their columns, over 1.7 rounds of CTAs.
constexpr int kAsHeads = 8;
__global__ void __launch_bounds__(kAsHeads * 32) attn_shared_join_kernel(const AttnParams p, const int ctas) {
    __shared__ float weight_s[kAsHeads][kAsMaxSplits];
    const ktk_attn& a = p.a;
    const int lane = threadIdx.x & 31, head = blockIdx.x * kAsHeads + (threadIdx.x >> 5);
    const int64_t row = blockIdx.y;
    float* weight = weight_s[threadIdx.x >> 5];
    if (head >= a.heads) return;
    const float sk = p.sink ? p.sink[head] * kLog2eF : kAsNone;
    const float gate = p.gate ? to_f32(((const __nv_bfloat16*)p.gate)[row * p.gate_stride + head]) : 0.0f;
    const Span sp = span_of(p.t, (int)row);
    if (sp.bad || sp.total <= 0) {
        if (head == 0 && lane == 0) report(p.status, KTK_STATUS_BAD_TABLE);
        return;
    }
    const AsCut cut = as_cut(p.t, ctas);
    const int64_t start = (int64_t)sp.start - p.t.kv_indptr[0], c0 = start / cut.chunk;
    const int splits = (int)((start + sp.pages - 1) / cut.chunk - c0) + 1;
    if (splits == 1 || start < 0 || start + sp.pages > cut.total) return;              // whole: written already
    // the first piece lies in the second slot of its CTA, the others in the first
    const int64_t first = a.heads * as_partial_floats(a.vdim_stride), stride = 2 * first;
    const float* w = p.ws + c0 * stride + head * as_partial_floats(a.vdim_stride);
    float M = sk, L = 0.0f;
    for (int s = lane; s < splits; s += 32) {
        const float2 ml = *reinterpret_cast<const float2*>(w + s * stride + (s == 0 ? first : 0));
        if (ml.y > 0.0f) M = fmaxf(M, ml.x);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, o));
    for (int s = lane; s < splits; s += 32) {
        const float2 ml = *reinterpret_cast<const float2*>(w + s * stride + (s == 0 ? first : 0));
        const float f = ml.y > 0.0f ? ex2(ml.x - M) : 0.0f;
        L += f * ml.y;
        weight[s] = f;
    }
    L = warp_sum_f(L);
    __syncwarp();
    if (p.sink) L += ex2(sk - M);
    float g = L > 0.0f ? 1.0f / L : 0.0f;
    if (p.gate) g *= sigmoid_f(gate);
    __nv_bfloat16* o = (__nv_bfloat16*)p.o + (row * a.heads + head) * a.vdim_stride;
    constexpr int kBlocks = kAsMaxVdim / 128;            // a lane holds 4 columns of every 128
    float4 v[kBlocks];
#pragma unroll
    for (int k = 0; k < kBlocks; ++k) v[k] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll 2
    for (int s = 0; s < splits; ++s) {
        const float f = weight[s];
        const float* src = w + s * stride + (s == 0 ? first : 0) + 4;
#pragma unroll
        for (int k = 0; k < kBlocks; ++k) {
            const int c = k * 128 + lane * 4;
            if (f == 0.0f || c >= a.vdim_stride) continue;               // an empty split has written no columns
            const float4 x = *reinterpret_cast<const float4*>(src + c);
            v[k].x += f * x.x; v[k].y += f * x.y; v[k].z += f * x.z; v[k].w += f * x.w;
        }
    }
#pragma unroll
    for (int k = 0; k < kBlocks; ++k) {
        const int c = k * 128 + lane * 4;
        if (c >= a.vdim_stride) continue;
        uint2 r;
        r.x = pack_bf16(c < a.vdim ? v[k].x * g : 0.0f, c + 1 < a.vdim ? v[k].y * g : 0.0f);
        r.y = pack_bf16(c + 2 < a.vdim ? v[k].z * g : 0.0f, c + 3 < a.vdim ? v[k].w * g : 0.0f);
        *reinterpret_cast<uint2*>(o + c) = r;
    }
}

static int shared_stages(const ktk_attn& a, int n) {
    const int kc = (a.dim_stride + 63) / 64, fixed = kc * n * 128 + kAsTok * 128;
    int fit = (kAsSmem - fixed) / (kc * kAsChunk);
    return fit < kAsMaxStages ? fit : kAsMaxStages;
}

bool attn_shared_supported(const ktk_attn& a) {
    return a.dtype == KTK_BF16 && a.maps == 1 && a.kv_heads == 1 && a.v_row_stride == a.dim_stride && a.softcap == 0.0f &&
           a.temp_coef == 0.0f && a.dim_stride <= kAsMaxDim && a.vdim_stride <= kAsMaxVdim && shared_stages(a, 64) >= 2;
}

// rounds of CTAs x (tiles of each + what starting and finishing one costs, in tiles of 1.75 us); *splits: the count of least cost
static int64_t splits_cost(int64_t units, int64_t tiles, int64_t* splits) {
    int64_t most = (tiles + kAsMinTiles - 1) / kAsMinTiles, best_cost = -1;
    if (most > kAsMaxSplits) most = kAsMaxSplits;
    *splits = 1;
    for (int64_t s = 1; s <= most && units > 0; ++s) {
        const int64_t rounds = (units * s + sm_count() - 1) / sm_count();
        const int64_t cost = rounds * ((tiles + s - 1) / s + kAsStartTiles) + (s > 1 ? kAsStartTiles : 0);
        if (best_cost < 0 || cost < best_cost) { best_cost = cost; *splits = s; }
        if (rounds > 8) break;
    }
    return best_cost;
}

// new_rows: 0 for one row of each of `batch` sequences, else the rows of one sequence
int32_t attn_shared_splits(const ktk_attn& a, int batch, int new_rows, int64_t max_keys) {
    const Packing k = packing_of(a.heads, new_rows == 0);
    const int64_t units = (int64_t)batch * k.chunks * (new_rows == 0 ? 1 : (new_rows + k.rows - 1) / k.rows);
    int64_t splits;
    splits_cost(units, (max_keys + kAsTok - 1) / kAsTok, &splits);
    return (int32_t)splits;
}

// CTAs of the balanced form per chunk of heads
static int balanced_ctas(const ktk_attn& a) {
    const int ctas = sm_count() / packing_of(a.heads, true).chunks;
    return ctas < 1 ? 1 : ctas < kAsMaxSplits ? ctas : kAsMaxSplits;
}

// Whether a decode step is cut over all sequences instead of sequence by sequence.  Its CTAs run the mean of the tiles, which for
// lengths that differ is well under that of the longest sequence's (counted here as four fifths of it; the host knows no more), but pay for each
// sequence (13 tiles' time) and for a second launch that joins the pieces of a sequence one behind the other.  So never below 25 tiles a CTA,
// where few sequences are cut into many pieces.  Fitted to 412 shapes of 8 to 128 heads, 576 columns; us by sequence / balanced, 32 heads:
// 128 x 4000 tokens 121 / 120, ragged (a sixteenth of it upwards) 116 / 92; 32 x 16384 122 / 119, ragged 117 / 89; 150 x 2000 139 / 103;
// 100 x 4000 116 / 102; but 1 x 16384 34 / 56, 4 x 4000 27 / 38, 16 x 4000 33 / 37, 48 x 2000 38 / 44, 128 x 600 31 / 39.
bool attn_shared_balanced(const ktk_attn& a, int batch, int64_t max_keys) {
    const int64_t tiles = (max_keys + kAsTok - 1) / kAsTok, ctas = balanced_ctas(a);
    int64_t splits;
    const int64_t cost = splits_cost((int64_t)batch * packing_of(a.heads, true).chunks, tiles, &splits);
    if (batch <= 0 || batch > 65535 || batch * tiles < 25 * ctas) return false;
    const double pieces = batch < ctas ? (double)ctas / batch : 1.0;             // of a sequence
    return (0.8 * (double)tiles + 13.0) * batch / (double)ctas + 10.0 + 2.0 * pieces < (double)cost;
}

size_t attn_shared_workspace(const ktk_attn& a, int64_t rows, int splits) {
    if (splits == KTK_SPLITS_BALANCED) return (size_t)balanced_ctas(a) * 2 * a.heads * as_partial_floats(a.vdim_stride) * sizeof(float);
    return splits <= 1 ? 0 : (size_t)rows * a.heads * splits * as_partial_floats(a.vdim_stride) * sizeof(float);
}

template <int N> static int shared_launch(const AttnParams& p, const Packing& k, cudaStream_t st) {
    const char* who = "ktk_paged_attention";
    const ktk_attn& a = p.a;
    const uint64_t ps = p.t.page_size;
    const uint64_t kd[3] = {(uint64_t)a.dim_stride, ps, (uint64_t)p.t.num_pages};
    const uint64_t ks[2] = {(uint64_t)a.dim_stride * 2, ps * a.dim_stride * 2};
    const uint32_t box[3] = {64, (uint32_t)(ps < kAsTok ? ps : kAsTok), 1};
    CUtensorMap km, pm;
    int rc = make_tensor_map_3d(&km, p.k, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, kd, ks, box, CU_TENSOR_MAP_SWIZZLE_128B, who);
    if (rc != KTK_OK) return rc;
    pm = km;
    if (ps == kAsTok && a.dim_stride >= 4 * 64) {
        // four chunks of 64 columns per copy: columns, tokens, chunks, pages
        const uint64_t pd[4] = {64, ps, (uint64_t)a.dim_stride / 64, (uint64_t)p.t.num_pages};
        const uint64_t pstr[3] = {(uint64_t)a.dim_stride * 2, 128, ps * a.dim_stride * 2};
        const uint32_t pbox[4] = {64, kAsTok, 4, 1};
        rc = make_tensor_map(&pm, p.k, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, pd, pstr, pbox, CU_TENSOR_MAP_SWIZZLE_128B, who);
        if (rc != KTK_OK) return rc;
    }
    const int kc = (a.dim_stride + 63) / 64, stages = shared_stages(a, N), vblocks = (a.vdim_stride + kUmRows - 1) / kUmRows;
    const int smem = kc * N * 128 + stages * kc * kAsChunk + kAsTok * 128 + 1024;
    uint32_t cols = 32;
    while (cols < (uint32_t)((2 + vblocks) * N)) cols *= 2;
    const int64_t groups = p.new_indptr ? (p.max_new + k.rows - 1) / k.rows : 1;
    if (groups * p.t.batch > 65535) {
        set_error("%s: more than 65535 groups of rows in one launch", who);
        return KTK_ERR_TOO_LARGE;
    }
    KTK_CUDA_TRY(cudaFuncSetAttribute(attn_shared_kernel<N>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem), who);
    const bool balanced = p.splits < 0;
    const int ctas = balanced_ctas(a);
    const dim3 grid((unsigned)(balanced ? ctas : p.splits), (unsigned)k.chunks, (unsigned)(balanced ? 1 : groups * p.t.batch));
    attn_shared_kernel<N><<<grid, kAsThreads, smem, st>>>(p, km, pm, kc, stages, cols);
    KTK_CUDA_TRY(cudaGetLastError(), who);
    if (balanced)
        attn_shared_join_kernel<<<dim3((unsigned)((a.heads + kAsHeads - 1) / kAsHeads), (unsigned)p.rows), kAsHeads * 32, 0, st>>>(p, ctas);
    else if (p.splits > 1)
        attn_shared_combine_kernel<<<dim3((unsigned)a.heads, (unsigned)p.rows), 128, 0, st>>>(p);
    KTK_CUDA_TRY(cudaGetLastError(), who);
    return KTK_OK;
}

int launch_attn_shared(const AttnParams& p, cudaStream_t st) {
    if (p.splits > kAsMaxSplits || (p.splits != 1 && p.rows > 65535)) {
        set_error("ktk_paged_attention: %d splits of %lld rows", p.splits, (long long)p.rows);
        return KTK_ERR_TOO_LARGE;
    }
    if (p.new_indptr && p.max_new <= 0) return KTK_OK;
    const Packing k = packing_of(p.a.heads, p.new_indptr == nullptr);
    return k.n == 16 ? shared_launch<16>(p, k, st) : k.n == 32 ? shared_launch<32>(p, k, st) : shared_launch<64>(p, k, st);
}

}  // namespace ktk
