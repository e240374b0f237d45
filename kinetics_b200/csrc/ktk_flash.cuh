// Softmax attention of two tiles of 128 rows per CTA on the fifth-generation tensor cores: what the prompt kernels share.
// A kernel brings the queries into shared memory and gives the copies of a block of keys and values, the scores' form and
// the mask; here are the order of the matrix instructions, the ring and the softmax.
//
// Roles of the 384 threads:
//     warps 0..3, 4..7   softmax of tile 0, of tile 1: thread r holds row r = lane r of tensor memory
//     warp 8             matrix instructions, per block j of KEYS keys and tile m
//                            O_m[128 x vdim] += P_m(j) . V(j)   P_m from tensor memory, V read MN-major as its rows lie
//                            S_m[128 x KEYS]  = Q_m . K(j + 1)^T
//                        While the tensor cores work on one tile, the other tile's threads do their softmax.
//     warp 9             TMA: NK blocks of K, `nv` of V in flight
// Tensor memory: S_m at column 128 m (P_m over its first KEYS / 2 columns), O_m at 256 + 128 m.  S_m(j + 1) is issued behind
// O_m += P_m(j) . V(j), whose operand it overwrites: matrix instructions of one thread execute in order.  The barrier of
// S_m(j) therefore also says that O_m is complete up to block j - 1, so a row may be rescaled without a wait of its own.
//
// Blocks of 128 keys: an instruction with N = 64 takes 32 cycles and its operands 48 cycles of shared memory (A 4 KiB, B 2 KiB
// at 128 B a cycle); with N = 128 both take 64.  Per tile and block of 128 keys, 128 columns: 1024 cycles of matrix instructions and
// 1024 of the special-function units (16 exponentials a cycle).
// The exponentials of one warp come at 12 cycles each instead of 8 (latencies), those of two at 10.  Two threads to a row (16 softmax
// warps) and a polynomial on the FMA pipes for a part of the exponentials were not faster; over seconds the power limit binds.
// Every wait is bounded; the caller reports `abort` and frees tensor memory.
#pragma once

#include <type_traits>

#include "ktk_umma.cuh"

namespace ktk {

constexpr int kFlThreads = 384;             // warps 10 and 11 only complete the warpgroup whose registers go to the softmax
constexpr int kFlTmemCols = 512;
constexpr int kFlColO = 256;
constexpr int kFlQTile = kUmRows * 128;      // [128 rows][64 columns]
constexpr float kFlMost = 256.0f;            // the exponentials' reference moves when half a block's sum is above it
constexpr int kFlMaxSmem = 225 * 1024;       // dynamic; the barriers are static

// Registers: 384 threads start with 168 each (64512 of the SM's); the softmax holds a row of scores, so its two warpgroups go
// to 200 and the third to 104: 256 * 200 + 128 * 104 = 64512.  All warps of a warpgroup have to execute the same instruction:
// each stands once in a kernel, on a branch that whole warpgroups take, and the third one's roles part behind it.
__device__ __forceinline__ void more_registers() { asm volatile("setmaxnreg.inc.sync.aligned.u32 200;"); }
__device__ __forceinline__ void fewer_registers() { asm volatile("setmaxnreg.dec.sync.aligned.u32 104;"); }
constexpr int kFlSoftmaxWarps = 8;

// -inf where no key has been seen: the exponentials then refer to 0
__device__ __forceinline__ float reference_or_zero(float m) { return m == -INFINITY ? 0.0f : m; }

__device__ __forceinline__ float max3(float a, float b, float c) {
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}

// S complete, the halves of P in place, O complete up to the first half of a block, O complete (tile) | K, V landed, K, V read out (buffer)
struct FlashShared {
    uint64_t s[2], p[2], p_rest[2], o_half[2], o[2], k[2], v[2], kfree[2], vfree[2];
    uint32_t tmem;
    int abort;
    __device__ __forceinline__ void init() {             // one thread
        for (int i = 0; i < 2; ++i) {
            mbar_init(&s[i], 1);
            mbar_init(&p[i], 4);
            mbar_init(&p_rest[i], 4);
            mbar_init(&o_half[i], 1);
            mbar_init(&o[i], 1);
            mbar_init(&k[i], 1);
            mbar_init(&v[i], 1);
            mbar_init(&kfree[i], 1);
            mbar_init(&vfree[i], 1);
        }
        abort = 0;
        mbar_init_fence();
    }
};

// NK: buffers of K, 1 or 2
template <int KEYS, int VC, int NK = 2> struct Flash {
    static constexpr int kTile = KEYS * 128;             // [KEYS keys][64 columns]
    static constexpr int kHalf = KEYS / 2;
    static constexpr int kVBuf = VC * kTile;
    FlashShared& sh;
    uint8_t *q, *k, *v;                                  // [tile][chunk] | [buffer][chunk] | [buffer][chunk]
    int q_chunks, k_chunks;                              // 64-column chunks of a tile's queries, of a block of K
    int nv;                                              // buffers of V: 1 or 2
    int keys0, keys1;                                    // key columns up to the last one that some row of each tile sees
    int blocks0, blocks1;                                // blocks that hold them

    __device__ __forceinline__ Flash(FlashShared& shared, uint8_t* smem, int qc, int kc, int n0, int n1)
        : sh(shared), q(smem), k(smem + 2 * qc * kFlQTile), v(k + NK * kc * kTile), q_chunks(qc), k_chunks(kc),
          nv(v_buffers(qc, kc)), keys0(n0), keys1(n1), blocks0((n0 + KEYS - 1) / KEYS), blocks1((n1 + KEYS - 1) / KEYS) {}
    // with 1 KiB to align it; the second buffer of V where shared memory holds it
    __host__ __device__ static constexpr int bytes_of(int qc, int kc, int v_bufs) {
        return 2 * qc * kFlQTile + NK * kc * kTile + v_bufs * kVBuf + 1024;
    }
    __host__ __device__ static constexpr int v_buffers(int qc, int kc) { return bytes_of(qc, kc, 2) <= kFlMaxSmem ? 2 : 1; }
    __host__ __device__ static constexpr int bytes(int qc, int kc) { return bytes_of(qc, kc, v_buffers(qc, kc)); }

    __device__ __forceinline__ int blocks() const { return blocks0 > blocks1 ? blocks0 : blocks1; }
    __device__ __forceinline__ int blocks_of(int m) const { return m ? blocks1 : blocks0; }
    __device__ __forceinline__ int k_buf(int blk) const { return blk & (NK - 1); }
    __device__ __forceinline__ uint32_t k_phase(int blk) const { return (uint32_t)(blk >> (NK - 1)) & 1u; }
    __device__ __forceinline__ int v_buf(int blk) const { return blk & (nv - 1); }
    __device__ __forceinline__ uint32_t v_phase(int blk) const { return (uint32_t)(blk >> (nv - 1)) & 1u; }

    // ---- queries of tile m, by its four warps.  piece(row, chunk, i): where 16 bytes of the row lie, the i-th of 64 columns, or
    // null for zeros.  Eight lanes to a row's 128 bytes: a lane for each row took 32
    // lines per access, 1 us per tile.
    template <class Piece> __device__ __forceinline__ void queries(int m, Piece piece) {
        const int warp = (threadIdx.x >> 5) & 3, lane = threadIdx.x & 31, at = lane & 7;
        uint8_t* dst = q + m * q_chunks * kFlQTile;
#pragma unroll 2
        for (int c = 0; c < q_chunks; ++c) {
            uint4 v[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const uint4* src = piece(warp * 32 + i * 4 + (lane >> 3), c, at);
                v[i] = src ? __ldg(src) : make_uint4(0u, 0u, 0u, 0u);
            }
#pragma unroll
            for (int i = 0; i < 8; ++i)
                *reinterpret_cast<uint4*>(dst + c * kFlQTile + swz(warp * 32 + i * 4 + (lane >> 3), at)) = v[i];
        }
        fence_proxy_async();
    }

    // ---- matrix instructions, by a converged warp.  steps(c): 16-column steps of chunk c; k_off: bytes between the keys of
    // the two tiles in a buffer of K (0: the same keys); vcols: columns of V, a multiple of 16; CLEARED: the rows of V
    // behind the last key that a tile sees are zeros
    template <bool CLEARED = false, class Steps> __device__ __forceinline__ void issue(Steps steps, int k_off, int vcols) {
        const uint32_t tmem = sh.tmem;
        const uint32_t idesc_s = umma_idesc(KEYS, false), idesc_o = umma_idesc(vcols, true);
        const uint64_t q_desc = umma_desc(smem_u32(q), 0, 1024), k_desc = umma_desc(smem_u32(k), 0, 1024);
        const uint64_t v_desc = umma_desc(smem_u32(v), kTile, 1024);
        const int n = blocks();
        auto scores = [&](int m, int blk) {
            const uint64_t qa = umma_desc_at(q_desc, m * q_chunks * kFlQTile);
            const uint64_t ka = umma_desc_at(k_desc, k_buf(blk) * k_chunks * kTile + m * k_off);
            if (elect_one()) {
                for (int c = 0; c < q_chunks; ++c) {
                    const int n_steps = steps(c);
#pragma unroll
                    for (int i = 0; i < 4; ++i)
                        if (i < n_steps)
                            umma_f16(tmem + m * 128, umma_desc_at(qa, c * kFlQTile + i * 32), umma_desc_at(ka, c * kTile + i * 32),
                                     idesc_s, (c > 0 || i > 0) ? 1u : 0u);
                }
                umma_commit(&sh.s[m]);
            }
            __syncwarp();
        };
        auto wait = [&](uint64_t* bar, uint32_t parity) {
            if (!mbar_wait_all(bar, parity, &sh.abort)) return false;
            tc_fence_after();
            return true;
        };
        // O_m += P_m(j) . V(j), the first half of the block's keys while the threads work on the second.  Not `whole`, a tile's last
        // block: values behind the last key that the tile sees are left out, for 0 times one that is not finite is not 0.
        auto products = [&](auto whole, int m, int j) {
            const int n_steps = whole ? KEYS / 16 : ((m ? keys1 : keys0) - j * KEYS + 15) / 16;
            const uint64_t va = umma_desc_at(v_desc, v_buf(j) * kVBuf);
#pragma unroll
            for (int part = 0; part < 2; ++part) {
                if (!wait(part ? &sh.p_rest[m] : &sh.p[m], j & 1)) return false;
                if (elect_one()) {
#pragma unroll
                    for (int i = part * (kHalf / 16); i < (part + 1) * (kHalf / 16); ++i)
                        if (whole || i < n_steps)
                            umma_f16_ts(tmem + kFlColO + m * 128, tmem + m * 128 + i * 8, umma_desc_at(va, i * (16 * 128)), idesc_o,
                                        (j > 0 || i > 0) ? 1u : 0u);
                    if (part == 0) umma_commit(&sh.o_half[m]);
                    else if (j + 1 == blocks_of(m)) umma_commit(&sh.o[m]);
                }
                __syncwarp();
            }
            return true;
        };
        if (n == 0 || !wait(&sh.k[0], 0)) return;
        if (blocks0 > 0) scores(0, 0);
        if (blocks1 > 0) scores(1, 0);
        if (elect_one()) umma_commit(&sh.kfree[0]);
        __syncwarp();
        for (int j = 0; j < n; ++j) {
            const bool more = j + 1 < n;
            // V, and K of the next block, before the probabilities, which are what the tensor cores are short of; an only buffer of
            // K is filled later
            if (!wait(&sh.v[v_buf(j)], v_phase(j)) || (more && NK > 1 && !wait(&sh.k[k_buf(j + 1)], k_phase(j + 1)))) return;
#pragma unroll
            for (int m = 0; m < 2; ++m) {
                const int mine = blocks_of(m);
                if (j < mine) {
                    if (!(CLEARED || j + 1 < mine ? products(std::true_type{}, m, j) : products(std::false_type{}, m, j))) return;
                }
                if (m == 1) {
                    if (elect_one()) umma_commit(&sh.vfree[v_buf(j)]);
                    __syncwarp();
                }
                if (j + 1 < mine) {
                    if (NK == 1 && !wait(&sh.k[0], k_phase(j + 1))) return;
                    scores(m, j + 1);
                }
                if (m == 1 && more) {
                    if (elect_one()) umma_commit(&sh.kfree[k_buf(j + 1)]);
                    __syncwarp();
                }
            }
        }
    }

    // ---- copies, by a converged warp.  load_k(blk, dst, bar), load_v(blk, dst, bar): tell the barrier the bytes and start the
    // copies.  The first ones start when the barriers are set up, while the other warps bring in the queries.
    template <class LoadK, class LoadV> __device__ __forceinline__ void first_copies(LoadK load_k, LoadV load_v) {
        load_k(0, k, &sh.k[0]);
        load_v(0, v, &sh.v[0]);
        if (NK > 1 && blocks() > 1) load_k(1, k + k_chunks * kTile, &sh.k[1]);
    }
    template <class LoadK, class LoadV> __device__ __forceinline__ void copy(LoadK load_k, LoadV load_v) {
        const int n = blocks();
        int k_issued = n < NK ? n : NK, v_issued = 1;
        bool alive = true;
        for (int j = 0; j < n && alive; ++j) {
            // V over that of block j - nv, then K of block j + NK over that of block j
            if (j > 0) {
                alive = j < nv || mbar_wait_all(&sh.vfree[v_buf(j)], v_phase(j) ^ 1u, &sh.abort);
                if (!alive) break;
                load_v(j, v + v_buf(j) * kVBuf, &sh.v[v_buf(j)]);
                ++v_issued;
            }
            if (j + NK < n) {
                alive = mbar_wait_all(&sh.kfree[k_buf(j)], k_phase(j), &sh.abort);
                if (!alive) break;
                load_k(k_issued, k + k_buf(k_issued) * k_chunks * kTile, &sh.k[k_buf(k_issued)]);
                ++k_issued;
            }
        }
        if (!alive) {                                    // the copies in flight still write shared memory
            volatile int never = 0;
            for (int i = k_issued > NK ? k_issued - NK : 0; i < k_issued; ++i) mbar_wait(&sh.k[k_buf(i)], k_phase(i), &never);
            for (int i = v_issued > nv ? v_issued - nv : 0; i < v_issued; ++i) mbar_wait(&sh.v[v_buf(i)], v_phase(i), &never);
        }
    }

    // ---- softmax of tile m, by its four warps (thread `row`).  prepare(s, j): the scores of block j, masked ones -inf; returns
    // whether form(x, y) is still to be applied to every pair of them.  The exponents are s f (FIXED: s) against m_ref.
    // clear(j): rows of V(j) that hold no key.  Returns whether O is complete.
    //
    // The reference is the larger of the sink and the first block's maximum, and stays while no half block's sum passes 2^8 (or is
    // infinite); then it is that half's maximum.  So no other block's maximum has to be searched, which cost 500 of a block's 3400
    // cycles.  A weight of 2^8 or more becomes 1, which bf16 holds exactly: the row of a key that outweighs all others is that
    // key's value.  And |O| <= 2^8 max|V| per 64 keys: 8192 keys leave |V| 2^113 (1e34) of the range of fp32.
    // The halves of a block are handed over one by one: the prompt of 8192 tokens and 32 heads takes 521 us without that, 498 with
    // it (two builds of one comparison).
    template <bool FIXED, class Prepare, class Form, class Clear>
    __device__ __forceinline__ bool softmax(int m, float f, float& m_ref, float& l_run, Prepare prepare, Form form, Clear clear) {
        const int warp = (threadIdx.x >> 5) & 3, lane = threadIdx.x & 31;
        const uint32_t my = sh.tmem + ((uint32_t)(warp * 32) << 16), s_at = my + m * 128, o_at = my + kFlColO + m * 128;
        const uint64_t f2 = pack2(f, f);
        const int mine = blocks_of(m);
        for (int j = 0; j < mine; ++j) {
            if (!mbar_wait_all(&sh.s[m], j & 1, &sh.abort)) return false;
            tc_fence_after();
            float s[KEYS];
            tmem_load(s_at, s);
            const bool raw = prepare(s, j);
            float base = FIXED ? 0.0f : -reference_or_zero(m_ref);
            uint32_t packed[kHalf / 2];
            uint64_t sum[2] = {0, 0};
            auto pair = [&](int from, int c, bool formed) {
                float x = s[from + 2 * c], y = s[from + 2 * c + 1];
                if (formed) form(x, y);
                if (!FIXED) unpack2(fma2(pack2(x, y), f2, pack2(base, base)), x, y);
                x = ex2(x);
                y = ex2(y);
                sum[c & 1] = add2(sum[c & 1], pack2(x, y));
                packed[c] = pack_bf16(x, y);
            };
            auto half = [&](int from) {
                sum[0] = sum[1] = 0;
                if (FIXED && raw) {
#pragma unroll
                    for (int c = 0; c < kHalf / 2; ++c) pair(from, c, true);
                } else {
#pragma unroll
                    for (int c = 0; c < kHalf / 2; ++c) pair(from, c, false);
                }
            };
            auto total = [&] {
                float a, b;
                unpack2(add2(sum[0], sum[1]), a, b);
                return a + b;
            };
            auto hand_over = [&](int from, uint64_t* bar) {
                tmem_st32_u32(s_at + from / 2, packed);
                l_run += total();
                tmem_st_wait();
                if (from == 0) clear(j);
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(bar);
            };
            // another reference, no lower than the exponents of columns from ..: O and the sum so far follow it
            auto move = [&](int from, bool mine_moves, bool has_o) {
                float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
                for (int c = 0; c < KEYS; c += 8)
                    if (c >= from)
#pragma unroll
                        for (int i = 0; i < 4; ++i) mx[i] = max3(mx[i], s[c + i], s[c + 4 + i]);
                const float top = max3(fmaxf(mx[0], mx[1]), mx[2], mx[3]) * f;
                const bool moves = mine_moves && top > m_ref;
                const float alpha = moves ? ex2(m_ref - top) : 1.0f;
                if (moves) m_ref = top;
                base = -reference_or_zero(m_ref);
                l_run *= alpha;
                if (has_o) {
#pragma unroll
                    for (int c = 0; c < VC * 64; c += 16) {
                        float o[16];
                        tmem_ld16(o_at + c, o);
#pragma unroll
                        for (int i = 0; i < 16; ++i) o[i] *= alpha;
                        tmem_st16(o_at + c, o);
                    }
                }
            };
            // the votes: tensor memory is read and written by whole warps
            // Rows that have seen no key hold an O of zeros.
            if (!FIXED && (j == 0 || __any_sync(0xffffffffu, m_ref == -INFINITY))) move(0, j == 0 || m_ref == -INFINITY, false);
            half(0);
            if (!FIXED) {
                const bool over = total() > kFlMost;
                if (__any_sync(0xffffffffu, over)) { move(0, over, j > 0); half(0); }
            }
            hand_over(0, &sh.p[m]);
            half(kHalf);
            if (!FIXED) {
                const bool over = total() > kFlMost;
                if (__any_sync(0xffffffffu, over)) {
                    if (!mbar_wait_all(&sh.o_half[m], j & 1, &sh.abort)) return false;
                    tc_fence_after();
                    move(kHalf, over, true);
                    half(kHalf);
                }
            }
            hand_over(kHalf, &sh.p_rest[m]);
        }
        if (mine > 0 && !mbar_wait_all(&sh.o[m], 0, &sh.abort)) return false;
        tc_fence_after();
        return true;
    }

    // Zeros over the rows of V(j) without a key (has_key(row)), by the first tile that sees the block
    template <class HasKey> __device__ __forceinline__ void clear_rows(int m, int j, HasKey has_key) {
        if (m != (j < blocks0 ? 0 : 1)) return;
        const int r = threadIdx.x & (kUmRows - 1);
        if (r < KEYS && !has_key(r)) {
            mbar_wait_fast(&sh.v[v_buf(j)], v_phase(j), &sh.abort);          // a wait that ran out ends the next block
#pragma unroll
            for (int c = 0; c < VC * 8; ++c)
                *reinterpret_cast<uint4*>(v + v_buf(j) * kVBuf + (c >> 3) * kTile + swz(r, c & 7)) = make_uint4(0u, 0u, 0u, 0u);
        }
        fence_proxy_async();
    }
};

}  // namespace ktk
