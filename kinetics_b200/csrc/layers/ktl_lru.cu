// A linear recurrence with real gates behind a short causal convolution, per channel (see ktk_layers.h), over a
// sequence's next tokens or one token of every sequence.  State, gates and decays are fp32.
//
// The convolution keeps its newest `taps` inputs in a ring by position: a step writes the place of the input that has
// just left the window, which nobody reads.  The prompt's scan is one pass over its inputs: the CTAs of a cluster take
// consecutive tiles of tokens and exchange the tiles' products and end states through distributed shared memory.
#include "../ktk_umma.cuh"
#include "ktl_common.cuh"

namespace ktk {

constexpr int kLcThreads = 64;
constexpr int kLcChunk = 16;            // tokens per thread of the convolution
constexpr int kLsWarps = 8, kLsRun = 8;  // warps of a scan CTA, tokens of a warp
constexpr int kLsThreads = kLsWarps * 32, kLsTile = kLsWarps * kLsRun, kLsMaxCluster = 8;
constexpr int kLdThreads = 128;

// what a sequence runs now: rows [row0, row0 + n), of positions base ..; false if the table or the slot is malformed
struct Run { int64_t row0; int n, base, slot; };
__device__ __forceinline__ bool run_of(const ktk_paged& t, const int32_t* new_indptr, const int32_t* slots, int64_t num_slots,
                                       int b, int32_t* status, Run& r) {
    const Span s = span_of(t, b);
    r.row0 = new_indptr ? new_indptr[b] : b;
    r.n = new_indptr ? new_indptr[b + 1] - new_indptr[b] : 1;
    r.base = s.total - r.n;
    r.slot = slots[b];
    const bool ok = !s.bad && r.base >= 0 && r.slot >= 0 && r.slot < num_slots;
    if (!ok && threadIdx.x == 0) report(status, KTK_STATUS_BAD_TABLE);
    return ok;
}

// Thread: 8 channels of `chunk` tokens.  TAPS > 0: the window stays in registers; 0: any number of taps.
template <typename T, int TAPS>
__global__ void __launch_bounds__(kLcThreads)
lru_conv_kernel(const T* __restrict__ x, int64_t row_stride, const int32_t* __restrict__ new_indptr,
                const int32_t* __restrict__ slots, int64_t num_slots, const float* __restrict__ w, const float* __restrict__ bias,
                T* ring, T* __restrict__ u, const ktk_paged t, int width, int taps_any, int chunk, int32_t* status) {
    Run r;
    if (!run_of(t, new_indptr, slots, num_slots, blockIdx.z, status, r)) return;
    const int taps = TAPS > 0 ? TAPS : taps_any;
    const int c = (blockIdx.x * kLcThreads + threadIdx.x) * 8;
    const int t0 = blockIdx.y * chunk, t1 = t0 + chunk < r.n ? t0 + chunk : r.n;
    if (c >= width || t0 >= r.n) return;
    T* mine = ring + (int64_t)r.slot * taps * width + c;
    auto input = [&](int i, float (&v)[8]) {              // input of token i of the run (i < 0: an earlier one)
        if (i >= 0) Vec8<T>::load(x + (r.row0 + i) * row_stride + c, v);
        else if (r.base + i >= 0) Vec8<T>::load(mine + (int64_t)((r.base + i) % taps) * width, v);
        else {
#pragma unroll
            for (int e = 0; e < 8; ++e) v[e] = 0.0f;
        }
    };
    float b8[8];
    load8(bias + c, b8);
    if (TAPS > 0) {
        float win[TAPS > 0 ? TAPS : 1][8], wt[TAPS > 0 ? TAPS : 1][8];
#pragma unroll
        for (int k = 0; k < TAPS; ++k) {
            load8(w + (int64_t)k * width + c, wt[k]);
            if (k + 1 < TAPS) input(t0 - (TAPS - 1) + k, win[k]);
        }
#pragma unroll 4
        for (int i = t0; i < t1; ++i) {
            input(i, win[TAPS > 0 ? TAPS - 1 : 0]);
            float o[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) o[e] = b8[e];
#pragma unroll
            for (int k = 0; k < TAPS; ++k)
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                    o[e] = fmaf(wt[k][e], win[k][e], o[e]);
                    if (k > 0) win[k - 1][e] = win[k][e];
                }
            Vec8<T>::store(u + (r.row0 + i) * width + c, o);
        }
    } else {
        for (int i = t0; i < t1; ++i) {
            float o[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) o[e] = b8[e];
            for (int k = 0; k < taps; ++k) {
                float v[8], wk[8];
                input(i - (taps - 1) + k, v);
                load8(w + (int64_t)k * width + c, wk);
#pragma unroll
                for (int e = 0; e < 8; ++e) o[e] = fmaf(wk[e], v[e], o[e]);
            }
            Vec8<T>::store(u + (r.row0 + i) * width + c, o);
        }
    }
    // the first chunk's thread is the only one that reads this ring (a chunk has at least `taps` tokens): it also writes
    if (t0 == 0)
        for (int i = r.n > taps ? r.n - taps : 0; i < r.n; ++i) {
            float v[8];
            Vec8<T>::load(x + (r.row0 + i) * row_stride + c, v);
            Vec8<T>::store(mine + (int64_t)((r.base + i) % taps) * width, v);
        }
}

// ---- gates and the recurrence ----
// v into the place of *p in CTA `cta` of the cluster
__device__ __forceinline__ void put_peer_f32(const float* p, float v, uint32_t cta) {
    uint32_t at;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at) : "r"(smem_u32(p)), "r"(cta));
    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(at), "f"(v) : "memory");
}
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ float sqrt_approx(float x) {
    float y;
    asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
// FAST (bf16): the approximate instructions themselves, without the scaling for results below 2^-126 that the functions add;
// what is flushed there is no part of a sigmoid that bf16 could show.  A scan spends 8 of them per token and channel.
constexpr float kLog2e = 1.4426950408889634f;
__device__ __forceinline__ float rcp_approx(float x) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
template <bool FAST> __device__ __forceinline__ float sigmoid_of(float x) {
    return FAST ? rcp_approx(1.0f + ex2(-kLog2e * x)) : 1.0f / (1.0f + expf(-x));
}
// 1 - exp(-x), x >= 0: the series where the difference would cancel
__device__ __forceinline__ float one_minus_exp(float x, float e) {
    const float s = x * (1.0f + x * (-0.5f + x * (1.0f / 6.0f + x * (-1.0f / 24.0f + x * (1.0f / 120.0f - x * (1.0f / 720.0f))))));
    return x < 0.3f ? s : 1.0f - e;
}
// one token of one channel: S <- a S + g
template <bool FAST>
__device__ __forceinline__ void gates(float zr, float zi, float u, float rb, float ib, float decay, float& a, float& g) {
    const float x = sigmoid_of<FAST>(zr + rb) * decay;                    // -log a
    a = FAST ? ex2(-kLog2e * x) : expf(-x);
    g = (FAST ? sqrt_approx(one_minus_exp(2.0f * x, a * a)) : sqrtf(-expm1f(-2.0f * x))) * sigmoid_of<FAST>(zi + ib) * u;
}
// 0.5 y (1 + tanh z) = y / (1 + exp(-2 z)),  z = sqrt(2 / pi) (y + 0.044715 y^3)
template <bool FAST> __device__ __forceinline__ float gelu_tanh(float y) {
    const float z2 = 2.0f * 0.7978845608028654f * (y + 0.044715f * y * y * y);
    return FAST ? y * rcp_approx(1.0f + ex2(fminf(-kLog2e * z2, 115.0f))) : y / (1.0f + expf(-z2));
}

struct LruParams {
    ktk_lru a;
    ktk_paged t;
    const float* z;
    const void *u, *y;
    int64_t row_stride;
    const int32_t *new_indptr, *slots;
    int64_t num_slots, rows;
    int max_new;
    const float *rb, *ib, *decay;
    float* state;
    void* out;
    int32_t* status;
};

// 32 channels of one sequence: lane = channel, a warp runs 8 consecutive tokens, a CTA 64, the CTAs of a cluster consecutive
// tiles of 64.  Per round of the cluster: local products and end states, joined over the CTA's warps in shared memory and
// over the cluster's CTAs through theirs; then every warp replays its tokens from the state in front of them.
// Bound by what it issues and by the rounds' barriers (8192 tokens of 2048 channels: 2.6 instructions a clock and SM, DRAM at a third of
// its rate), eight special functions per token and channel first; the bytes, 14 of each, take half the time.  So a warp's
// next round is on its way into shared memory while it computes this one, the output gate is worked out between the two
// halves of the cluster's barrier, and a CTA writes its totals into its peers' memory, where each warp folds them by itself.
// 8192 tokens of 4096 channels, bf16: 139 us (3.4 TB/s; the output gate's functions 16 of them), with loads into registers at
// the head of each round and totals read from the peers 205.  Three CTAs per SM that compute a round ahead of the barrier: 170.
constexpr int kLsGateBytes = 2 * kLsRun * 32 * 4;                      // zr, zi of a warp's round
template <typename T> constexpr int kLsStage = kLsGateBytes + 2 * kLsRun * 32 * (int)sizeof(T);      // and u, y
template <typename T> constexpr int kLsSmem = 2 * kLsWarps * kLsStage<T>;
template <typename T> constexpr int kLsResident = sizeof(T) == 2 ? 4 : 3;                          // CTAs per SM, by shared memory
// ONE: a single stage per warp and four CTAs per SM, for fp32 portions of one round, which have nothing to bring ahead.
// 200 sequences of 9 tokens, 2048 channels: 191 us, 232 with two stages and three CTAs.

template <typename T, bool ALIGNED, bool ONE>
__global__ void __launch_bounds__(kLsThreads, ONE ? 4 : kLsResident<T>) lru_scan_kernel(const LruParams p) {
    constexpr bool FAST = sizeof(T) == 2;
    extern __shared__ __align__(16) uint8_t ls_raw[];
    // by parity of the round, so that a round needs no barrier behind its last reads
    __shared__ float warp_a[2][kLsWarps][32], warp_s[2][kLsWarps][32], tile_a[2][kLsMaxCluster][32], tile_s[2][kLsMaxCluster][32];
    Run r;
    if (!run_of(p.t, p.new_indptr, p.slots, p.num_slots, blockIdx.z, p.status, r)) return;      // uniform for the cluster
    const int ctas = gridDim.x, rank = blockIdx.x;
    const int bs = p.a.block_stride, width = p.a.blocks * bs;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int c0 = blockIdx.y * 32, c = c0 + lane;
    const bool on = c < width;
    const T* u = (const T*)p.u + r.row0 * width;
    const T* y = (const T*)p.y + r.row0 * p.row_stride;
    T* out = (T*)p.out + r.row0 * width + c;
    uint8_t* stages = ls_raw + warp * (ONE ? 1 : 2) * kLsStage<T>;
    const auto gate_row = [&](int ch) {                                // zr of channel ch, token 0; zi lies bs behind it
        const int blk = ch / bs;
        return p.z + ((int64_t)blk * p.rows + r.row0) * (2 * bs) + (ch - blk * bs);
    };
    // a lane copies 16 bytes of one row of each copy; 8 channels never cross a block's or the width's end
    constexpr int kT = 16 / (int)sizeof(T), kTRows = kT, kTLanes = 32 / kT;      // channels of a piece of T, rows a copy takes
    const int zc = c0 + (lane & 7) * 4, tc = c0 + (lane % kTLanes) * kT;
    const float* zsrc = gate_row(zc < width ? zc : 0);
    const float* mine = gate_row(on ? c : 0);
    const auto fill = [&](int it) {
        const int i0 = (it * ctas + rank) * kLsTile + warp * kLsRun;
        uint8_t* st = stages + (ONE ? 0 : it & 1) * kLsStage<T>;
        if (ALIGNED) {
            const uint32_t at = smem_u32(st) + lane * 16;
#pragma unroll
            for (int k = 0; k < kLsRun; k += 4) {
                const int i = i0 + k + (lane >> 3);
                const bool have = zc < width && i < r.n;
                const float* src = zsrc + (have ? (int64_t)i : 0) * (2 * bs);
                cp_async16(at + k * 128, src, have ? 16u : 0u);
                cp_async16(at + kLsGateBytes / 2 + k * 128, src + bs, have ? 16u : 0u);
            }
#pragma unroll
            for (int k = 0; k < kLsRun; k += kTRows) {
                const int i = i0 + k + lane / kTLanes;
                const bool have = tc < width && i < r.n;
                const int64_t row = have ? i : 0;
                const int ch = have ? tc : 0;
                cp_async16(at + kLsGateBytes + k * 32 * sizeof(T), u + row * width + ch, have ? 16u : 0u);
                cp_async16(at + kLsGateBytes + (kLsRun + k) * 32 * sizeof(T), y + row * p.row_stride + ch, have ? 16u : 0u);
            }
            cp_async_commit();
        } else {
            float* z = reinterpret_cast<float*>(st) + lane;
            T* ty = reinterpret_cast<T*>(st + kLsGateBytes) + lane;
#pragma unroll 2
            for (int k = 0; k < kLsRun; ++k) {
                const bool have = on && i0 + k < r.n;
                const int64_t row = have ? i0 + k : 0;
                z[k * 32] = have ? mine[row * (2 * bs)] : 0.0f;
                z[(kLsRun + k) * 32] = have ? mine[row * (2 * bs) + bs] : 0.0f;
                ty[k * 32] = u[row * width + (have ? c : 0)];
                ty[(kLsRun + k) * 32] = y[row * p.row_stride + (have ? c : 0)];
            }
        }
    };
    const int rounds = (r.n + ctas * kLsTile - 1) / (ctas * kLsTile);
    if (rounds > 0) fill(0);
    const float rb = on ? p.rb[c] : 0.0f, ib = on ? p.ib[c] : 0.0f, decay = on ? p.decay[c] : 0.0f;
    float carry = on && r.base > 0 ? p.state[(int64_t)r.slot * width + c] : 0.0f;      // behind the previous round
    if (ctas > 1) cluster_sync();                          // the peers have begun: their shared memory may be written
    for (int it = 0; it < rounds; ++it) {
        const int par = it & 1, i0 = (it * ctas + rank) * kLsTile + warp * kLsRun;
        __syncwarp();                                      // the other stage, the warp's own, has been read
        if (ONE ? it > 0 : it + 1 < rounds) fill(ONE ? it : it + 1);
        if (ALIGNED) {
            if (!ONE && it + 1 < rounds) cp_async_wait<1>();
            else cp_async_wait<0>();
        }
        __syncwarp();
        const float* z = reinterpret_cast<const float*>(stages + (ONE ? 0 : par) * kLsStage<T>) + lane;
        const T* ty = reinterpret_cast<const T*>(stages + (ONE ? 0 : par) * kLsStage<T> + kLsGateBytes) + lane;
        const int have = !on ? 0 : r.n - i0 < kLsRun ? r.n - i0 : kLsRun;      // tokens of the lane
        float a[kLsRun], g[kLsRun], A = 1.0f, S = 0.0f;
#pragma unroll
        for (int k = 0; k < kLsRun; ++k) {
            gates<FAST>(z[k * 32], z[(kLsRun + k) * 32], to_f32(ty[k * 32]), rb, ib, decay, a[k], g[k]);
            if (k >= have) { a[k] = 1.0f; g[k] = 0.0f; }
            A *= a[k];
            S = fmaf(a[k], S, g[k]);
        }
        warp_a[par][warp][lane] = A;
        warp_s[par][warp][lane] = S;
        __syncthreads();
        if (warp < ctas) {                                 // warp w tells CTA w
            A = 1.0f; S = 0.0f;
#pragma unroll
            for (int w = 0; w < kLsWarps; ++w) {
                const float wa = warp_a[par][w][lane];
                S = fmaf(wa, S, warp_s[par][w][lane]);
                A *= wa;
            }
            put_peer_f32(&tile_a[par][rank][lane], A, warp);
            put_peer_f32(&tile_s[par][rank][lane], S, warp);
        }
        cluster_arrive();
        float gate[kLsRun];
#pragma unroll
        for (int k = 0; k < kLsRun; ++k) gate[k] = gelu_tanh<FAST>(to_f32(ty[(kLsRun + k) * 32]));
        cluster_wait();
        for (int k = 0; k < ctas; ++k) {
            if (k == rank) S = carry;
            carry = fmaf(tile_a[par][k][lane], carry, tile_s[par][k][lane]);
        }
        for (int w = 0; w < warp; ++w) S = fmaf(warp_a[par][w][lane], S, warp_s[par][w][lane]);
        T* o = out + (int64_t)i0 * width;
#pragma unroll
        for (int k = 0; k < kLsRun; ++k) {
            S = fmaf(a[k], S, g[k]);
            if (k < have) *o = from_f32<T>(S * gate[k]);
            o += width;
        }
    }
    // every write into this CTA's memory came before the last round's barrier
    if (warp == 0 && rank == 0 && on) p.state[(int64_t)r.slot * width + c] = carry;
}

// One token of every sequence: a thread per channel.
template <typename T>
__global__ void __launch_bounds__(kLdThreads) lru_step_kernel(const LruParams p) {
    constexpr bool FAST = sizeof(T) == 2;
    Run r;
    if (!run_of(p.t, nullptr, p.slots, p.num_slots, blockIdx.y, p.status, r)) return;
    const int bs = p.a.block_stride, width = p.a.blocks * bs;
    const int c = blockIdx.x * kLdThreads + threadIdx.x;
    if (c >= width) return;
    const int blk = c / bs, cc = c - blk * bs;
    const float* z = p.z + ((int64_t)blk * p.rows + r.row0) * (2 * bs) + cc;
    float* state = p.state + (int64_t)r.slot * width + c;
    float a, g;
    gates<FAST>(z[0], z[bs], to_f32(((const T*)p.u)[r.row0 * width + c]), p.rb[c], p.ib[c], p.decay[c], a, g);
    const float S = fmaf(a, r.base > 0 ? *state : 0.0f, g);
    *state = S;
    ((T*)p.out)[r.row0 * width + c] = from_f32<T>(S * gelu_tanh<FAST>(to_f32(((const T*)p.y)[r.row0 * p.row_stride + c])));
}

// ---- one token of every sequence in one launch: convolution, gate products on the tensor cores, recurrence, output gate ----
// A CTA takes CHAN channels of a block and up to 32 rows.  It convolves all channels of the block (the products need them;
// their inputs lie in L2), multiplies u [32 x block] with the CHAN + CHAN gate rows by mma.m16n8k16, and finishes its channels.
// The ring's place that a step writes is read by no other CTA.  Bound by latency: a chain of loads (slot, window and state), the
// products, the stores; so a thread keeps to one piece of the channels and loads a tap's weights once, the state and the gate are on their
// way before the products, and CHAN is what leaves the shorter rounds of CTAs (lf_wide).
constexpr int kLfRows = 32, kLfThreads = 256, kLfMaxBlock = 512;

__host__ __device__ inline int lf_ld(int block_stride) { return (block_stride + 15) / 16 * 16 + 8; }      // padded: no bank conflicts
__host__ __device__ inline int lf_smem(int block_stride, int chan) { return (kLfRows + 2 * chan) * lf_ld(block_stride) * 2 + kLfRows * (2 * chan + 1) * 4; }

// 64 channels per CTA instead of 32: where two such CTAs share an SM as two of the others do (blocks of up to 288 channels), and their
// rounds, of 5/4 the length, are fewer by more than that.  16 blocks of 256 channels, 128 rows: 29 us with an element per access, 22.8
// with 32 channels in two rounds, 16.8 with 64 in one.  us of 32 / 64 channels elsewhere: 40 x 64, 256 rows 19.4 / 18.3, 64 x 96, 128 rows
// 22.7 / 21.8, 20 x 200, 256 rows 41.7 / 38.1; but 20 x 200, 128 rows 22.8 / 24.9 (two rounds either way), blocks of one slice 64 x 32,
// 256 rows 14.5 / 18.6 and 128 x 24 24.5 / 32.3, one CTA per SM 8 x 512, 256 rows 59.9 / 64.6 and 12 x 304 55.4 / 60.0.
static bool lf_wide(const ktk_lru& a, int64_t groups) {
    const auto rounds = [&](int chan) {
        const int64_t ctas = groups * a.blocks * ((a.block_stride + chan - 1) / chan), slots = 2 * (int64_t)sm_count();
        return (ctas + slots - 1) / slots;
    };
    return 2 * (lf_smem(a.block_stride, 64) + 2048) <= 228 * 1024 && 5 * rounds(64) < 4 * rounds(32);
}

// neighbouring channels of a lane, one access
template <typename T, int N> struct alignas(N * sizeof(T)) Lanes { T x[N]; };

struct LruDecodeParams {
    LruParams p;
    const __nv_bfloat16 *x, *gates;
    const float *conv_w, *conv_b;
    __nv_bfloat16* ring;
};

template <int TAPS, int CHAN> __global__ void __launch_bounds__(kLfThreads, 2) lru_decode_kernel(const LruDecodeParams q) {
    extern __shared__ __align__(16) uint8_t lf_raw[];
    __shared__ int row_slot[kLfRows], row_pos[kLfRows];
    const LruParams& p = q.p;
    const int bs = p.a.block_stride, taps = p.a.taps, width = p.a.blocks * bs, ld = lf_ld(bs);
    __nv_bfloat16* su = reinterpret_cast<__nv_bfloat16*>(lf_raw);       // [rows][ld]
    __nv_bfloat16* sw = su + kLfRows * ld;                              // [CHAN rows of r, CHAN of i][ld]
    float* sz = reinterpret_cast<float*>(sw + 2 * CHAN * ld);               // [rows][CHAN zr | CHAN zi | pad]
    constexpr int kZ = 2 * CHAN + 1;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int slices = (bs + CHAN - 1) / CHAN, blk = blockIdx.x / slices, n0 = (blockIdx.x - blk * slices) * CHAN;
    const int64_t r0 = (int64_t)blockIdx.y * kLfRows;
    const int rows = p.rows - r0 < kLfRows ? (int)(p.rows - r0) : kLfRows;
    const int c0 = blk * bs, pieces = (ld - 8) / 8;                     // 16-byte pieces of a row
    if (tid < kLfRows) {
        int slot = -1, pos = 0;
        if (tid < rows) {
            const Span s = span_of(p.t, (int)(r0 + tid));
            slot = p.slots[r0 + tid];
            pos = s.total - 1;
            if (s.bad || pos < 0 || slot < 0 || slot >= p.num_slots) {
                report(p.status, KTK_STATUS_BAD_TABLE);
                slot = -1;
            }
        }
        row_slot[tid] = slot;
        row_pos[tid] = pos;
    }
    // thread: piece k of rows first_row, + row_step, ...
    int per = 8, shift = 3;                                             // threads of a row: the next power of two
    while (per < pieces) { per *= 2; ++shift; }
    const int k = tid & (per - 1), first_row = tid >> shift, row_step = kLfThreads >> shift, c_mine = c0 + k * 8;
    const bool mine_on = k * 8 < bs;
    // gate weights on their way; rows and columns outside are zero
    if (k < pieces) {
        const __nv_bfloat16* src = q.gates + ((int64_t)2 * blk * bs + n0) * bs + k * 8;
        const uint32_t dst = smem_u32(sw + k * 8);
#pragma unroll 4
        for (int n = first_row; n < 2 * CHAN; n += row_step) {
            const int c = n & (CHAN - 1);
            const bool on = mine_on && n0 + c < bs;
            cp_async16(dst + n * ld * 2, on ? src + (n < CHAN ? c : bs + c) * bs : q.gates, on ? 16u : 0u);
        }
    }
    constexpr int kTaps = TAPS > 0 ? TAPS : 1, kBatch = TAPS > 0 ? 2 : 1;
    __syncthreads();
    // this CTA's channels, CHAN / 32 neighbours per lane: state and gate of rows warp, + 8, ...
    constexpr int kCols = CHAN / 32, kMine = kLfRows / (kLfThreads / 32);
    using Floats = Lanes<float, kCols>;
    using Halves = Lanes<__nv_bfloat16, kCols>;
    const int n = n0 + lane * kCols, c = c0 + n;                        // a block's channels are a multiple of 8
    Floats state0[kMine];
    Halves gate[kMine];
#pragma unroll
    for (int i = 0; i < kMine; ++i) {
        const int r = warp + i * (kLfThreads / 32), slot = n < bs ? row_slot[r] : -1;
#pragma unroll
        for (int h = 0; h < kCols; ++h) { state0[i].x[h] = 0.0f; gate[i].x[h] = __float2bfloat16(0.0f); }
        if (slot >= 0) {
            if (row_pos[r] > 0) state0[i] = *reinterpret_cast<const Floats*>(p.state + (int64_t)slot * width + c);
            gate[i] = *reinterpret_cast<const Halves*>((const __nv_bfloat16*)p.y + (r0 + r) * p.row_stride + c);
        }
    }
    // u of every channel of the block: kBatch rows per thread with all their loads in flight
    if (k < pieces)
        for (int rb = first_row; rb < kLfRows; rb += row_step * kBatch) {
            uint4 raw[kBatch][kTaps];
#pragma unroll
            for (int b = 0; b < kBatch; ++b) {
                const int r = rb + b * row_step;
                const int slot = r < kLfRows && mine_on ? row_slot[r & (kLfRows - 1)] : -1, pos = slot >= 0 ? row_pos[r] : 0;
                const __nv_bfloat16* mine = q.ring + (int64_t)(slot >= 0 ? slot : 0) * taps * width + c_mine;
#pragma unroll
                for (int t = 0; t < kTaps; ++t) {                       // the last is the token's own
                    const int at = pos - (kTaps - 1) + t;
                    raw[b][t] = make_uint4(0u, 0u, 0u, 0u);             // zeros before the sequence
                    if (t == kTaps - 1) { if (slot >= 0) raw[b][t] = *reinterpret_cast<const uint4*>(q.x + (r0 + r) * p.row_stride + c_mine); }
                    else if (slot >= 0 && at >= 0) raw[b][t] = *reinterpret_cast<const uint4*>(mine + (int64_t)(at % taps) * width);
                }
            }
            float o[kBatch][8], w[8];
#pragma unroll
            for (int b = 0; b < kBatch; ++b)
#pragma unroll
                for (int e = 0; e < 8; ++e) o[b][e] = 0.0f;
            if (mine_on) {                                              // a tap's weights serve the batch
                load8(q.conv_b + c_mine, w);
#pragma unroll
                for (int b = 0; b < kBatch; ++b)
#pragma unroll
                    for (int e = 0; e < 8; ++e) o[b][e] = w[e];
                if (TAPS == 0)
                    for (int t = 0; t + 1 < taps; ++t) {
                        const int slot = rb < kLfRows ? row_slot[rb] : -1, at = slot >= 0 ? row_pos[rb] - (taps - 1) + t : -1;
                        if (at < 0) continue;
                        float v[8];
                        Vec8<__nv_bfloat16>::load(q.ring + ((int64_t)slot * taps + at % taps) * width + c_mine, v);
                        load8(q.conv_w + (int64_t)t * width + c_mine, w);
#pragma unroll
                        for (int e = 0; e < 8; ++e) o[0][e] = fmaf(w[e], v[e], o[0][e]);
                    }
#pragma unroll
                for (int t = 0; t < kTaps; ++t) {
                    load8(q.conv_w + (int64_t)(taps - kTaps + t) * width + c_mine, w);
#pragma unroll
                    for (int b = 0; b < kBatch; ++b) {
                        float v[8];
                        unpack8(raw[b][t], v);
#pragma unroll
                        for (int e = 0; e < 8; ++e) o[b][e] = fmaf(w[e], v[e], o[b][e]);
                    }
                }
            }
#pragma unroll
            for (int b = 0; b < kBatch; ++b) {
                const int r = rb + b * row_step;
                if (r >= kLfRows) continue;
                const int slot = mine_on ? row_slot[r] : -1;
                if (slot >= 0 && k * 8 >= n0 && k * 8 < n0 + CHAN)      // this CTA's channels
                    *reinterpret_cast<uint4*>(q.ring + ((int64_t)slot * taps + row_pos[r] % taps) * width + c_mine) = raw[b][kTaps - 1];
                if (slot < 0)
#pragma unroll
                    for (int e = 0; e < 8; ++e) o[b][e] = 0.0f;
                Vec8<__nv_bfloat16>::store(su + r * ld + k * 8, o[b]);
            }
        }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    {
        // warp: 16 rows, CHAN / 2 of the 2 CHAN columns
        constexpr int kTiles = CHAN / 16;
        const int gid = lane >> 2, tig = lane & 3, m0 = (warp & 1) * 16, g0 = (warp >> 1) * (CHAN / 2);
        float acc[kTiles][4] = {};
        const __nv_bfloat16* a0 = su + (m0 + gid) * ld + 2 * tig;
        const __nv_bfloat16* b0 = sw + (g0 + gid) * ld + 2 * tig;
#pragma unroll 4
        for (int kk = 0; kk < ld - 8; kk += 16) {
            uint32_t a[4];
            a[0] = *reinterpret_cast<const uint32_t*>(a0 + kk);
            a[1] = *reinterpret_cast<const uint32_t*>(a0 + 8 * ld + kk);
            a[2] = *reinterpret_cast<const uint32_t*>(a0 + kk + 8);
            a[3] = *reinterpret_cast<const uint32_t*>(a0 + 8 * ld + kk + 8);
#pragma unroll
            for (int t = 0; t < kTiles; ++t)
                mma_bf16(acc[t], a, *reinterpret_cast<const uint32_t*>(b0 + t * 8 * ld + kk),
                         *reinterpret_cast<const uint32_t*>(b0 + t * 8 * ld + kk + 8));
        }
#pragma unroll
        for (int t = 0; t < kTiles; ++t)
#pragma unroll
            for (int e = 0; e < 4; ++e) sz[(m0 + gid + (e >= 2 ? 8 : 0)) * kZ + g0 + t * 8 + 2 * tig + (e & 1)] = acc[t][e];
    }
    __syncthreads();
    if (n >= bs) return;
    const Floats rb = *reinterpret_cast<const Floats*>(p.rb + c), ib = *reinterpret_cast<const Floats*>(p.ib + c),
                 decay = *reinterpret_cast<const Floats*>(p.decay + c);
#pragma unroll
    for (int i = 0; i < kMine; ++i) {
        const int r = warp + i * (kLfThreads / 32), slot = row_slot[r];
        if (slot < 0) continue;
        Floats S;
        Halves out;
#pragma unroll
        for (int h = 0; h < kCols; ++h) {
            const int at = lane * kCols + h;
            float a, g;
            gates<true>(sz[r * kZ + at], sz[r * kZ + CHAN + at], __bfloat162float(su[r * ld + n + h]), rb.x[h], ib.x[h], decay.x[h], a, g);
            S.x[h] = fmaf(a, state0[i].x[h], g);
            out.x[h] = __float2bfloat16_rn(S.x[h] * gelu_tanh<true>(__bfloat162float(gate[i].x[h])));
        }
        *reinterpret_cast<Floats*>(p.state + (int64_t)slot * width + c) = S;
        *reinterpret_cast<Halves*>((__nv_bfloat16*)p.out + (r0 + r) * width + c) = out;
    }
}

static int check_lru(const ktk_lru* a, const ktk_paged* t, const int32_t* new_indptr, int64_t rows, int32_t max_new,
                     int64_t row_stride, int64_t col, int64_t num_slots, const char* who) {
    if (a == nullptr || t == nullptr || a->blocks <= 0 || a->block <= 0 || a->block_stride < a->block ||
        a->block_stride % 8 != 0 || a->taps <= 0 || a->taps > 1024 || (a->dtype != KTK_F32 && a->dtype != KTK_BF16) ||
        (int64_t)a->blocks * a->block_stride > (1 << 20) || t->page_size <= 0 || t->batch < 0 || t->batch > 65535) {
        set_error("%s: bad sizes", who);
        return KTK_ERR_ARG;
    }
    const int width = a->blocks * a->block_stride;
    if (rows < 0 || rows > 2147483647LL || (!new_indptr && rows != t->batch) || (new_indptr && max_new < 0) || row_stride % 8 != 0 ||
        col % 8 != 0 || col < 0 || col + width > row_stride || num_slots < 0) {
        set_error("%s: %lld rows for %d sequences, columns %lld of %lld", who, (long long)rows, t->batch, (long long)col,
                  (long long)row_stride);
        return KTK_ERR_ARG;
    }
    return KTK_OK;
}

template <typename T>
static int conv_launch(const void* x, int64_t row_stride, const int32_t* ni, int max_new, const int32_t* slots, int64_t num_slots,
                       const float* w, const float* b, void* ring, void* u, const ktk_paged& t, const ktk_lru& a,
                       int32_t* status, cudaStream_t st) {
    const int width = a.blocks * a.block_stride, chunk = a.taps > kLcChunk ? a.taps : kLcChunk;
    const int n = ni ? max_new : 1;
    const dim3 grid((unsigned)((width / 8 + kLcThreads - 1) / kLcThreads), (unsigned)((n + chunk - 1) / chunk), (unsigned)t.batch);
    if (grid.y > 65535) { set_error("ktk_lru_conv: %d tokens in one call", n); return KTK_ERR_TOO_LARGE; }
    auto kernel = a.taps == 4 ? lru_conv_kernel<T, 4> : lru_conv_kernel<T, 0>;
    kernel<<<grid, kLcThreads, 0, st>>>((const T*)x, row_stride, ni, slots, num_slots, w, b, (T*)ring, (T*)u, t, width, a.taps,
                                        chunk, status);
    KTK_CUDA_TRY(cudaGetLastError(), "ktk_lru_conv");
    return KTK_OK;
}

template <typename T> static int scan_launch(const LruParams& p, cudaStream_t st) {
    const int width = p.a.blocks * p.a.block_stride;
    if (p.new_indptr) {
        // as many CTAs along the sequence as stay resident together and have tokens
        const int64_t groups = (width + 31) / 32, tiles = (p.max_new + kLsTile - 1) / kLsTile;
        int ctas = kLsMaxCluster;
        while (ctas > 1 && (ctas > tiles || groups * p.t.batch * ctas > (int64_t)sm_count() * kLsResident<T>)) ctas /= 2;
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3((unsigned)ctas, (unsigned)groups, (unsigned)p.t.batch);
        cfg.blockDim = dim3(kLsThreads);
        cfg.dynamicSmemBytes = kLsSmem<T>;
        cfg.stream = st;
        cudaLaunchAttribute attr{};
        attr.id = cudaLaunchAttributeClusterDimension;
        attr.val.clusterDim.x = ctas;
        attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
        cfg.attrs = &attr;
        cfg.numAttrs = 1;
        // copies of 16 bytes: strides and columns are multiples of 8 elements, so only the buffers' addresses can forbid them
        const bool aligned = (((uintptr_t)p.z | (uintptr_t)p.u | (uintptr_t)p.y) & 15u) == 0;
        constexpr bool kHasOne = sizeof(T) == 4;
        const bool one = kHasOne && tiles <= 1;
        const auto kernel = one ? (aligned ? lru_scan_kernel<T, true, kHasOne> : lru_scan_kernel<T, false, kHasOne>)
                                : (aligned ? lru_scan_kernel<T, true, false> : lru_scan_kernel<T, false, false>);
        if (one) cfg.dynamicSmemBytes /= 2;
        KTK_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)cfg.dynamicSmemBytes), "ktk_lru_scan");
        KTK_CUDA_TRY(cudaLaunchKernelEx(&cfg, kernel, p), "ktk_lru_scan");
    }
    else
        lru_step_kernel<T><<<dim3((unsigned)((width + kLdThreads - 1) / kLdThreads), (unsigned)p.t.batch), kLdThreads, 0, st>>>(p);
    KTK_CUDA_TRY(cudaGetLastError(), "ktk_lru_scan");
    return KTK_OK;
}

}  // namespace ktk

using namespace ktk;

extern "C" int ktk_lru_conv(const void* proj, int64_t row_stride, int64_t x_col, const int32_t* new_indptr, int64_t rows,
                            int32_t max_new, const int32_t* slots, int64_t num_slots, const float* conv_w,
                            const float* conv_b, void* ring, void* u, const ktk_paged* table, const ktk_lru* shape,
                            int32_t* status, void* stream) {
    const char* who = "ktk_lru_conv";
    const int rc = check_lru(shape, table, new_indptr, rows, max_new, row_stride, x_col, num_slots, who);
    if (rc != KTK_OK) return rc;
    if (rows == 0 || max_new == 0) return KTK_OK;
    if (!proj || !slots || !conv_w || !conv_b || !ring || !u || !table->kv_indptr || !table->kv_last_page_len ||
        (((uintptr_t)proj | (uintptr_t)conv_w | (uintptr_t)conv_b | (uintptr_t)ring | (uintptr_t)u) & 15u) != 0) {
        set_error("%s: null or misaligned pointer", who);
        return KTK_ERR_ARG;
    }
    cudaStream_t st = (cudaStream_t)stream;
    if (shape->dtype == KTK_F32)
        return conv_launch<float>((const float*)proj + x_col, row_stride, new_indptr, max_new, slots, num_slots, conv_w, conv_b,
                                  ring, u, *table, *shape, status, st);
    return conv_launch<__nv_bfloat16>((const __nv_bfloat16*)proj + x_col, row_stride, new_indptr, max_new, slots, num_slots,
                                      conv_w, conv_b, ring, u, *table, *shape, status, st);
}

extern "C" int ktk_lru_scan(const float* z, const void* u, const void* proj, int64_t row_stride, int64_t y_col,
                            const int32_t* new_indptr, int64_t rows, int32_t max_new, const int32_t* slots,
                            int64_t num_slots, const float* rb, const float* ib, const float* decay, float* state,
                            void* out, const ktk_paged* table, const ktk_lru* shape, int32_t* status, void* stream) {
    const char* who = "ktk_lru_scan";
    const int rc = check_lru(shape, table, new_indptr, rows, max_new, row_stride, y_col, num_slots, who);
    if (rc != KTK_OK) return rc;
    if (rows == 0 || max_new == 0) return KTK_OK;
    if (!z || !u || !proj || !slots || !rb || !ib || !decay || !state || !out || !table->kv_indptr || !table->kv_last_page_len) {
        set_error("%s: null pointer", who);
        return KTK_ERR_ARG;
    }
    const size_t size = shape->dtype == KTK_F32 ? 4 : 2;
    const LruParams p{*shape, *table, z, u, (const char*)proj + y_col * size, row_stride, new_indptr, slots, num_slots, rows,
                      max_new, rb, ib, decay, state, out, status};
    return shape->dtype == KTK_F32 ? scan_launch<float>(p, (cudaStream_t)stream) : scan_launch<__nv_bfloat16>(p, (cudaStream_t)stream);
}

extern "C" int ktk_lru_decode_supported(const ktk_lru* shape) {
    return shape && shape->dtype == KTK_BF16 && shape->block_stride > 0 && shape->block_stride <= kLfMaxBlock ? 1 : 0;
}

extern "C" int ktk_lru_decode(const void* proj, int64_t row_stride, int64_t y_col, int64_t x_col, int64_t rows,
                              const int32_t* slots, int64_t num_slots, const float* conv_w, const float* conv_b,
                              const void* gates, const float* rb, const float* ib, const float* decay, void* ring, float* state,
                              void* out, const ktk_paged* table, const ktk_lru* shape, int32_t* status, void* stream) {
    const char* who = "ktk_lru_decode";
    int rc = check_lru(shape, table, nullptr, rows, 1, row_stride, x_col, num_slots, who);
    if (rc == KTK_OK) rc = check_lru(shape, table, nullptr, rows, 1, row_stride, y_col, num_slots, who);
    if (rc != KTK_OK) return rc;
    if (!ktk_lru_decode_supported(shape)) { set_error("%s: bf16, blocks of at most %d channels", who, kLfMaxBlock); return KTK_ERR_UNSUPPORTED; }
    if (rows == 0) return KTK_OK;
    if (!proj || !slots || !conv_w || !conv_b || !gates || !rb || !ib || !decay || !ring || !state || !out || !table->kv_indptr ||
        !table->kv_last_page_len ||
        (((uintptr_t)proj | (uintptr_t)conv_w | (uintptr_t)conv_b | (uintptr_t)gates | (uintptr_t)ring) & 15u) != 0) {
        set_error("%s: null or misaligned pointer", who);
        return KTK_ERR_ARG;
    }
    const LruParams p{*shape, *table, nullptr, nullptr, (const __nv_bfloat16*)proj + y_col, row_stride, nullptr, slots, num_slots,
                      rows, 1, rb, ib, decay, state, out, status};
    const LruDecodeParams q{p, (const __nv_bfloat16*)proj + x_col, (const __nv_bfloat16*)gates, conv_w, conv_b, (__nv_bfloat16*)ring};
    const int64_t groups = (rows + kLfRows - 1) / kLfRows;
    const bool pairs = ((uintptr_t)state & 7u) == 0 && (((uintptr_t)rb | (uintptr_t)ib | (uintptr_t)decay) & 7u) == 0 && ((uintptr_t)out & 3u) == 0;
    const bool narrow = !pairs || !lf_wide(*shape, groups);
    const int chan = narrow ? 32 : 64, smem = lf_smem(shape->block_stride, chan), slices = (shape->block_stride + chan - 1) / chan;
    auto kernel = shape->taps == 4 ? (narrow ? lru_decode_kernel<4, 32> : lru_decode_kernel<4, 64>)
                                   : (narrow ? lru_decode_kernel<0, 32> : lru_decode_kernel<0, 64>);
    KTK_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem), who);
    kernel<<<dim3((unsigned)(shape->blocks * slices), (unsigned)groups), kLfThreads, smem, (cudaStream_t)stream>>>(q);
    KTK_CUDA_TRY(cudaGetLastError(), who);
    return KTK_OK;
}
