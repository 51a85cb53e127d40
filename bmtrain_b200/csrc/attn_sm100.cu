// Fused attention for sm_100a (B200): softmax(scale * Q K^T + mask) V without the score matrix ever leaving the SM.
//
// Forward, backward and the packing of dense masks; the kernels' comments say how each is organised and what bounds it.
// Masks: causal (key j visible to query i iff j <= i + sk - sq), per-sample key counts, dense boolean (b, sq, sk).
// Grouped-query attention: kv head = head / (h / hk).  Head dims up to 128 (multiples of 16); tiles are padded with
// zeros by TMA.  Every mbarrier wait is bounded; on expiry a status word is set and the CTA winds down.
//
// The reference example materialises (b, h, s, s) scores and probabilities in HBM with two bmm calls
// (example/layers/attention.py:78-104).
#include <cuda.h>
#include <math.h>
#include <string.h>

#include <type_traits>

#include "api.h"
#include "common.cuh"
#include "tcgen05.cuh"
#include "tma_host.h"

namespace {

using namespace bmt_tc;

constexpr int FWD_THREADS = 384;                 // two groups of four softmax warps, producer, MMA issuer (a warpgroup of their own)
constexpr int TILE = 128;                        // query rows per CTA and keys per step
constexpr uint32_t CHUNK = TILE * 64 * 2;        // one [128 rows][64 columns] swizzled chunk of 16-bit elements: 16 KiB

__device__ int g_attn_status = 0;                // 0, or (code << 16) | blockIdx.x of the first CTA whose wait ran out

struct AttnParams {
    int64_t sq, sk;
    int h, hk, d;
    float sl2;                  // scale * log2(e)
    int causal;
    int64_t causal_off;         // sk - sq
    const uint32_t* bits;       // packed mask (b, sq, key tiles, 4 words) or null; a set bit = attend
    const uint8_t* cls;         // its summary (b, query tiles, key tiles): 0 nothing visible, 1 mixed, 2 everything visible
    const int32_t* kv_lens;     // (b) or null
    void* o;                    // (b, sq, h, d) by strides
    int64_t o_tok, o_head, o_batch;
    float* lse;                 // (b, h, sq), natural log; -inf for rows without a visible key
    uint32_t idesc_s, idesc_pv;
    int q_tiles, k_tiles;       // 128-row tiles of the queries / keys
    int per_cta;                // query tiles per CTA: 2, or 1 when there are too few to fill the GPU with pairs
};

struct AttnShared {
    uint64_t q_full, k_full[2], v_full[2], k_empty[2], v_empty[2];
    uint64_t s_full[2], p_half[2], p_ready[2], o_full[2];
    uint32_t tmem_base;
    int failed;
};

__device__ __forceinline__ float ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
using bmt::add_f2;
using bmt::fma_f2;
using bmt::mul_f2;
using bmt::pack2;
using bmt::pack_f2;
using bmt::unpack_f2;
// A from tensor memory: lane = row, every column holds two consecutive 16-bit elements of the reduction dimension.
__device__ __forceinline__ void umma_f16_ts(uint32_t tmem_c, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(tmem_c), "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}

__device__ __forceinline__ void fail(AttnShared* sh, int code) {
    sh->failed = 1;
    atomicCAS(&g_attn_status, 0, (code << 16) | (int)(blockIdx.x & 0xffff));
}

// Register split: a warpgroup hands registers back or takes more.  The shares of all warpgroups stay within what the block was
// launched with.
template <int N> __device__ __forceinline__ void regs_down() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N)); }
template <int N> __device__ __forceinline__ void regs_up() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N)); }


// The lowest `n` of 32 bits (n may be outside [0, 32]).
__device__ __forceinline__ uint32_t low_bits(int64_t n) { return n >= 32 ? 0xffffffffu : n <= 0 ? 0u : ((1u << (int)n) - 1u); }

// Packs a dense mask (b, sq, sk) of bytes into bits, once per call instead of once per head: one block per 128 x 128 tile.
//   bits   (b, sq, key tiles, 4 words): the 128 keys of a tile as seen by one query (forward)
//   bits_t (b, sk, query tiles, 4 words): the 128 queries of a tile as seen by one key (backward)
//   cls    (b, query tiles, key tiles): 0 nothing visible, 1 mixed, 2 everything visible -- tiles of class 0 are skipped
// Read per head and row, the bytes of a 437-key mask (rows not 16-byte aligned) took 3/4 of the attention kernel's time.
// A warp packs 32 queries x 32 keys with all its bytes in flight: a lane its query's keys from two 16-byte pieces, where the rows are
// made of such, or else its key's queries; the other direction is the same 32 x 32 bits transposed in five shuffles.  Latency bounds
// it up to some 500 tokens, then the bytes (1.8 - 2.1 TB/s).  With a vote per word and per key, and stores of single words:
// 2 x 512 x 512 10.4 us, now 2.9; 3 x 437 x 437 10.4, now 3.8; 4096 x 4096 39, now 9.1; 8 x 2048 x 2048 71, now 16.
constexpr int MASK_THREADS = 512;
// Bit i of lane l <-> bit l of lane i.
__device__ __forceinline__ uint32_t transpose_bits(uint32_t x, int lane) {
#pragma unroll
    for (int j = 16; j; j >>= 1) {
        const uint32_t low = j == 16 ? 0x0000ffffu : j == 8 ? 0x00ff00ffu : j == 4 ? 0x0f0f0f0fu : j == 2 ? 0x33333333u : 0x55555555u;
        const uint32_t y = __shfl_xor_sync(0xffffffffu, x, j);
        x = lane & j ? (x & ~low) | ((y & ~low) >> j) : (x & low) | ((y & low) << j);
    }
    return x;
}
__global__ void __launch_bounds__(MASK_THREADS)
attn_mask_pack_kernel(const uint8_t* mask, int64_t sq, int64_t sk, uint32_t* bits, uint32_t* bits_t, uint8_t* cls) {
    bmt::after_previous();
    __shared__ __align__(16) uint32_t w[TILE][4], wt[TILE][4];      // of a query, of a key
    const int kt = blockIdx.x, qt = blockIdx.y, b = blockIdx.z, n_kt = gridDim.x, n_qt = gridDim.y;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, qw = warp >> 2, kw = warp & 3;
    const int rows = (int)min((int64_t)TILE, sq - (int64_t)qt * TILE), keys = (int)min((int64_t)TILE, sk - (int64_t)kt * TILE);
    const uint8_t* tile = mask + ((int64_t)b * sq + (int64_t)qt * TILE) * sk + (int64_t)kt * TILE;
    // warp (qw, kw): 32 queries x 32 keys
    uint32_t by_query, by_key;
    if (sk % 16 == 0 && (reinterpret_cast<uintptr_t>(mask) & 15) == 0) {
        const int row = qw * 32 + lane, key = kw * 32;
        uint4 v[2];
#pragma unroll
        for (int u = 0; u < 2; ++u)
            v[u] = row < rows && key + u * 16 < keys ? *reinterpret_cast<const uint4*>(tile + row * sk + key + u * 16) : make_uint4(0, 0, 0, 0);
        // one bit per byte that is not 0: the product moves the lowest bits of the four bytes next to one another, without carries
        const auto nibble = [](uint32_t x) { return ((__vcmpne4(x, 0u) & 0x01010101u) * 0x10204080u) >> 28; };
        by_query = 0;
#pragma unroll
        for (int u = 0; u < 2; ++u)
            by_query |= (nibble(v[u].x) | nibble(v[u].y) << 4 | nibble(v[u].z) << 8 | nibble(v[u].w) << 12) << (16 * u);
        by_key = transpose_bits(by_query, lane);
    } else {
        const int row = qw * 32, key = kw * 32 + lane;
        uint8_t byte[32];
#pragma unroll
        for (int i = 0; i < 32; ++i) byte[i] = row + i < rows && key < keys ? tile[(row + i) * sk + key] : 0;
        by_key = 0;
#pragma unroll
        for (int i = 0; i < 32; ++i) by_key |= (byte[i] ? 1u : 0u) << i;
        by_query = transpose_bits(by_key, lane);
    }
    w[qw * 32 + lane][kw] = by_query;
    wt[kw * 32 + lane][qw] = by_key;
    const bool any = __syncthreads_or(by_query != 0);
    const bool full = __syncthreads_and(qw * 32 + lane >= rows || by_query == low_bits(keys - kw * 32));
    if (threadIdx.x == 0) cls[((int64_t)b * n_qt + qt) * n_kt + kt] = (uint8_t)(!any ? 0 : full ? 2 : 1);
    const int i = threadIdx.x;
    if (i < rows)
        *reinterpret_cast<uint4*>(bits + ((((int64_t)b * sq + (int64_t)qt * TILE + i) * n_kt) + kt) * 4) = *reinterpret_cast<const uint4*>(w[i]);
    else if (i >= TILE && i - TILE < keys)
        *reinterpret_cast<uint4*>(bits_t + ((((int64_t)b * sk + (int64_t)kt * TILE + i - TILE) * n_qt) + qt) * 4) = *reinterpret_cast<const uint4*>(wt[i - TILE]);
}

// Forward.  A CTA works on two tiles of 128 query rows (one when the grid would not fill the GPU) with a group of four
// softmax warps each, so that the tensor core multiplies for one tile while the other one is in its softmax:
//   warps 0..3 / 4..7   softmax of tile 0 / 1 (below)
//   warp 8      TMA producer: both Q tiles once, then K and V tiles of 128 keys through two-stage rings (shared by both)
//   warp 9      MMA issuer: S_t = Q_t K^T into tensor memory, O_t += P_t V with P_t read from tensor memory
//   softmax     one thread per query row reads its row of S from tensor memory, applies the
//               masks, and writes the probabilities back over it as packed 16-bit pairs, where the MMA takes them from.
// What bounds it: a 128 x 128 tile at head dim 128 is 1024 clocks of MMA and 1024 clocks of ex2 (16 per clock and SM); with
// one tile per CTA, and P going through shared memory, the two and everything in between took turns (about 4500 clocks).
// Now a group's tile takes about 3500 clocks (two groups: 1750 a tile): 550 for reading the row and its maximum, 1600 for the
// exponentials of both groups (2048 clocks of ex2 between them), 1200 from handing over P to the next scores, of which the MMAs are 770:
// P lies over the scores, and with two accumulators there is no tensor memory for a second set at head dim 128.
// The commit behind S_t(j) also covers P V of the tile before (the tensor pipe works in issue order), so a softmax group that
// has seen S_t(j) may rescale O_t without another wait.
template <int HD, typename T>
__global__ void __launch_bounds__(FWD_THREADS, 1)
flash_fwd_kernel(const __grid_constant__ CUtensorMap tq, const __grid_constant__ CUtensorMap tk, const __grid_constant__ CUtensorMap tv,
                 const AttnParams p) {
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    constexpr int DC = HD / 64;                     // 64-column chunks of the (padded) head dim
    constexpr uint32_t TB = DC * CHUNK;             // bytes of one Q / K / V tile
    const uint32_t sQ = smem_u32(smem), sK = sQ + 2 * TB, sV = sK + 2 * TB;
    AttnShared* sh = (AttnShared*)(smem + 6 * TB);

    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        mbar_init(&sh->q_full, 1);
        for (int i = 0; i < 2; ++i) {
            mbar_init(&sh->k_full[i], 1); mbar_init(&sh->v_full[i], 1); mbar_init(&sh->k_empty[i], 1); mbar_init(&sh->v_empty[i], 1);
            mbar_init(&sh->s_full[i], 1); mbar_init(&sh->p_half[i], 4); mbar_init(&sh->p_ready[i], 4); mbar_init(&sh->o_full[i], 1);
        }
        sh->failed = 0;
        fence_barrier_init();
    }
    if (warp == 9) { tmem_alloc(&sh->tmem_base, 512); tmem_relinquish(); }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    bmt::after_previous();
    const int head = blockIdx.x % p.h, b = blockIdx.x / p.h, kvh = head / (p.h / p.hk);
    const int qt0 = ((int)gridDim.y - 1 - (int)blockIdx.y) * p.per_cta;   // under a causal mask the long rows start first
    int64_t kv_lim = p.sk;
    if (p.kv_lens && p.kv_lens[b] < kv_lim) kv_lim = p.kv_lens[b];
    if (kv_lim < 0) kv_lim = 0;
    int J[2];                                       // key tiles that query tile t can see
#pragma unroll
    for (int t = 0; t < 2; ++t) {
        const int64_t q_end = (int64_t)(qt0 + t + 1) * TILE;
        int64_t end = kv_lim;
        if (p.causal && q_end + p.causal_off < end) end = q_end + p.causal_off;
        if (end < 0 || t >= p.per_cta || qt0 + t >= p.q_tiles) end = 0;
        J[t] = (int)((end + TILE - 1) / TILE);
    }
    const int J_max = J[0] > J[1] ? J[0] : J[1];
    const uint8_t* cls0 = p.cls ? p.cls + ((int64_t)b * p.q_tiles + qt0) * p.k_tiles : nullptr;
    auto active = [&](int t, int j) -> bool { return j < J[t] && (!cls0 || cls0[t * p.k_tiles + j] != 0); };
    auto next_step = [&](int j) -> int {
        do ++j; while (j < J_max && !active(0, j) && !active(1, j));
        return j;
    };

    const uint32_t tmem = sh->tmem_base;            // S_0 / P_0 [0,128), S_1 / P_1 [128,256), O_0 [256,384), O_1 [384,512)
    const int first = next_step(-1);

    if (warp >= 8) {
    regs_down<56>();             // 128 x 56 + 256 x 216 of the 384 x 168 registers at launch
    if (warp == 8) {
        // ------------------------------------------------------------------------------------------ TMA producer
        if (first < J_max) {
            const uint32_t qbar = smem_u32(&sh->q_full);
            if (elect_one()) {
                mbar_expect_tx_u32(qbar, (J[0] > 0 ? TB : 0) + (J[1] > 0 ? TB : 0));
#pragma unroll
                for (int t = 0; t < 2; ++t)
                    if (J[t] > 0) {
#pragma unroll
                        for (int c = 0; c < DC; ++c) tma_load_4d_u32(&tq, qbar, sQ + t * TB + c * CHUNK, c * 64, (qt0 + t) * TILE, head, b);
                    }
            }
            __syncwarp();
            int n = 0;
            for (int j = first; j < J_max; j = next_step(j), ++n) {
                const int st = n & 1;
                const uint32_t ph = (uint32_t)((n >> 1) & 1);
                if (!mbar_wait_warp(smem_u32(&sh->k_empty[st]), ph ^ 1)) { if (lane == 0) fail(sh, 1); break; }
                const uint32_t kbar = smem_u32(&sh->k_full[st]), vbar = smem_u32(&sh->v_full[st]);
                if (elect_one()) {
                    mbar_expect_tx_u32(kbar, TB);
#pragma unroll
                    for (int c = 0; c < DC; ++c) tma_load_4d_u32(&tk, kbar, sK + st * TB + c * CHUNK, c * 64, j * TILE, kvh, b);
                }
                __syncwarp();
                if (!mbar_wait_warp(smem_u32(&sh->v_empty[st]), ph ^ 1)) { if (lane == 0) fail(sh, 2); break; }
                if (elect_one()) {
                    mbar_expect_tx_u32(vbar, TB);
#pragma unroll
                    for (int c = 0; c < DC; ++c) tma_load_4d_u32(&tv, vbar, sV + st * TB + c * CHUNK, c * 64, j * TILE, kvh, b);
                }
                __syncwarp();
            }
        }
    } else if (warp == 9) {
        // ------------------------------------------------------------------------------------------ MMA issuer
        // the warp stays converged and one elected lane issues (operands in uniform registers)
        if (first < J_max) {
            const uint32_t hi = desc_hi(1024);
            const int ks_s = p.d / 16;                   // 16-deep steps of the Q K^T contraction
            bool ok = mbar_wait_warp(smem_u32(&sh->q_full), 0);
            if (!ok && lane == 0) fail(sh, 3);
            uint32_t done[2] = {0u, 0u};                 // tiles of P V issued per query tile
            int last[2] = {J[0] - 1, J[1] - 1};          // its last key tile
#pragma unroll
            for (int t = 0; t < 2; ++t)
                while (last[t] >= 0 && !active(t, last[t])) --last[t];
            auto issue_s = [&](int t, int st) {          // S_t = Q_t K^T
                // unrolled: a loop of unknown length took 70 clocks an instruction, more than its 64 of multiplying
                const uint32_t qd = desc_lo(sQ + t * TB, 0), kd = desc_lo(sK + st * TB, 0);
#pragma unroll
                for (int ks = 0; ks < HD / 16; ++ks) {
                    const uint32_t off = (uint32_t)((ks >> 2) * CHUNK + (ks & 3) * 32) >> 4;
                    if (ks < ks_s) umma_f16(tmem + t * TILE, pack_desc(qd + off, hi), pack_desc(kd + off, hi), p.idesc_s, ks != 0 ? 1u : 0u);
                }
                umma_commit(&sh->s_full[t]);
            };
            int j = first, n = 0;
            if (ok && !mbar_wait_warp(smem_u32(&sh->k_full[0]), 0)) { if (lane == 0) fail(sh, 4); ok = false; }
            if (ok) {
                tc_fence_after();
                if (elect_one()) {
                    if (active(0, j)) issue_s(0, 0);
                    if (active(1, j)) issue_s(1, 0);
                    umma_commit(&sh->k_empty[0]);
                }
                __syncwarp();
            }
            while (ok && j < J_max) {
                const int jn = next_step(j), st = n & 1, sn = (n + 1) & 1;
                const uint32_t ph = (uint32_t)((n >> 1) & 1), phn = (uint32_t)(((n + 1) >> 1) & 1);
                if (!mbar_wait_warp(smem_u32(&sh->v_full[st]), ph)) { if (lane == 0) fail(sh, 5); ok = false; break; }
                if (jn < J_max && !mbar_wait_warp(smem_u32(&sh->k_full[sn]), phn)) { if (lane == 0) fail(sh, 7); ok = false; break; }
                const uint32_t vd = desc_lo(sV + st * TB, CHUNK);
                // P V: B = V (128 keys x head dim, head dim contiguous = MN-major), 16 key rows per step, 64-column chunks CHUNK apart
                auto issue_pv = [&](int t, int half) {
#pragma unroll
                    for (int ks = half * 4; ks < half * 4 + 4; ++ks)
                        umma_f16_ts(tmem + 256 + t * TILE, tmem + t * TILE + ks * 8, pack_desc(vd + ks * 128, hi), p.idesc_pv, (done[t] | ks) != 0 ? 1u : 0u);
                };
#pragma unroll
                for (int t = 0; t < 2; ++t) {
                    const bool now = active(t, j), next = jn < J_max && active(t, jn);
                    if (now) {
                        // the first 64 keys of P_t are in tensor memory and, if row maxima moved, O_t has been rescaled by its
                        // owners; the second half of the softmax runs under the first half of the MMAs
                        if (!mbar_wait_warp(smem_u32(&sh->p_half[t]), done[t] & 1u)) { if (lane == 0) fail(sh, 6); ok = false; break; }
                        tc_fence_after();
                        if (elect_one()) issue_pv(t, 0);
                        __syncwarp();
                        if (!mbar_wait_warp(smem_u32(&sh->p_ready[t]), done[t] & 1u)) { if (lane == 0) fail(sh, 6); ok = false; break; }
                    }
                    tc_fence_after();
                    if (elect_one()) {
                        if (now) {
                            issue_pv(t, 1);
                            if (j == last[t]) umma_commit(&sh->o_full[t]);
                        }
                        if (next) issue_s(t, sn);
                    }
                    __syncwarp();
                    if (now) ++done[t];
                }
                if (!ok) break;
                if (elect_one()) {
                    umma_commit(&sh->v_empty[st]);
                    if (jn < J_max) umma_commit(&sh->k_empty[sn]);
                }
                __syncwarp();
                j = jn;
                ++n;
            }
        }
    }
    } else {
        // ------------------------------------------------------------------------------------------ softmax + epilogue
        regs_up<216>();
        const int t = warp >> 2, quarter = warp & 3;      // TMEM lanes [32 * quarter, 32 * quarter + 32) belong to this warp
        const int row = quarter * 32 + lane;
        const int64_t q0 = (int64_t)(qt0 + t) * TILE, qi = q0 + row;
        const bool row_ok = qi < p.sq;
        const uint32_t lane_addr = (uint32_t)(quarter * 32) << 16;
        const uint32_t s_addr = tmem + lane_addr + t * TILE, o_addr = tmem + lane_addr + 256 + t * TILE;
        const uint4* brow = (p.bits && row_ok) ? reinterpret_cast<const uint4*>(p.bits) + ((int64_t)b * p.sq + qi) * p.k_tiles : nullptr;
        const uint8_t* crow = cls0 ? cls0 + t * p.k_tiles : nullptr;
        const int64_t limit = p.causal && qi + p.causal_off + 1 < kv_lim ? qi + p.causal_off + 1 : kv_lim;   // keys below it are visible
        // m_ref: the maximum the exponents are taken against.  It follows the running maximum lazily: only when that
        // has grown by more than 8 (in base-2 exponent units) is the accumulator in tensor memory rescaled -- probabilities
        // stay below 2^8, sums are fp32 -- so that after the first few tiles a tile costs one round trip to tensor memory.
        float m_ref = -INFINITY, l_run = 0.f;
        uint32_t n = 0;
        bool ok = true;
        for (int j = 0; j < J[t] && ok; ++j) {
            const int kind = crow ? crow[j] : 2;
            if (kind == 0) continue;
            const int64_t kv0 = (int64_t)j * TILE;
            const bool need_mask = kind == 1 || kv0 + TILE > kv_lim || (p.causal && kv0 + TILE - 1 > q0 + p.causal_off);
            uint32_t vis[TILE / 32];
            if (need_mask) {
                uint4 w = make_uint4(0xffffffffu, 0xffffffffu, 0xffffffffu, 0xffffffffu);
                if (kind == 1 && brow) w = brow[j];
                vis[0] = w.x & low_bits(limit - kv0); vis[1] = w.y & low_bits(limit - kv0 - 32);
                vis[2] = w.z & low_bits(limit - kv0 - 64); vis[3] = w.w & low_bits(limit - kv0 - 96);
            }
            if (!mbar_wait_warp(smem_u32(&sh->s_full[t]), n & 1u)) { if (lane == 0) fail(sh, 9); ok = false; break; }
            tc_fence_after();
            uint32_t r[TILE / 32][32];
            tmem_ld32(s_addr, r[0]);
            tmem_ld32(s_addr + 32, r[1]);
            tmem_ld_wait_for(r[0]);
            tmem_ld_wait_for(r[1]);
            tmem_ld32(s_addr + 64, r[2]);        // on its way while the maximum of the first half is taken
            tmem_ld32(s_addr + 96, r[3]);
            // tiles away from the diagonal and the ragged edge (the common case) skip the per-element visibility tests
            float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
            if (need_mask) {
#pragma unroll
                for (int c4 = 0; c4 < TILE / 32; ++c4) {
                    if (c4 == 2) { tmem_ld_wait_for(r[2]); tmem_ld_wait_for(r[3]); }
#pragma unroll
                    for (int i = 0; i < 32; ++i)
                        if ((vis[c4] >> i) & 1u) mx[i & 3] = fmaxf(mx[i & 3], __uint_as_float(r[c4][i]));
                }
            } else {
#pragma unroll
                for (int c4 = 0; c4 < TILE / 32; ++c4) {
                    if (c4 == 2) { tmem_ld_wait_for(r[2]); tmem_ld_wait_for(r[3]); }
#pragma unroll
                    for (int i = 0; i < 32; i += 2)
                        mx[(i >> 1) & 3] = fmaxf(fmaxf(mx[(i >> 1) & 3], __uint_as_float(r[c4][i])), __uint_as_float(r[c4][i + 1]));
                }
            }
            const float mt = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3]));
            // move the reference maximum?  (first visible score of the row, or growth beyond the threshold)
            const bool fresh = m_ref == -INFINITY;                        // nothing accumulated yet: O and l are zero
            const bool move = !fresh && mt != -INFINITY && (mt - m_ref) * p.sl2 > 8.f;
            if (__any_sync(0xffffffffu, move)) {
                // rescale this warp's 32 rows of the accumulator (lanes whose maximum did not move multiply by one)
                const float alpha = move ? ex2((m_ref - mt) * p.sl2) : 1.f;
                l_run *= alpha;
#pragma unroll
                for (int c8 = 0; c8 < HD / 8; ++c8) {
                    if (c8 * 8 < p.d) {
                        uint32_t o[8];
                        tmem_ld8(o_addr + c8 * 8, o);
                        tmem_ld_wait();
#pragma unroll
                        for (int i = 0; i < 8; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
                        tmem_st8(o_addr + c8 * 8, o);
                    }
                }
            }
            if (fresh || move) m_ref = mt;
            const float neg_m = m_ref == -INFINITY ? 0.f : -m_ref * p.sl2;
            const uint64_t sl2_2 = pack_f2(p.sl2, p.sl2), neg_2 = pack_f2(neg_m, neg_m);
            uint64_t sum2[2] = {0ull, 0ull};
            // compiled with and without masks: tests that are predicated off still take an issue slot each
            auto exps = [&](auto masked) {
#pragma unroll
                for (int half = 0; half < 2; ++half) {
                    uint32_t pk[32];
#pragma unroll
                    for (int i = 0; i < 32; ++i) {
                        const int e = half * 64 + 2 * i, c4 = e >> 5, k = e & 31;
                        float x, y;
                        unpack_f2(fma_f2(pack_f2(__uint_as_float(r[c4][k]), __uint_as_float(r[c4][k + 1])), sl2_2, neg_2), x, y);
                        x = ex2(x);
                        y = ex2(y);
                        if constexpr (decltype(masked)::value) {
                            if (!((vis[c4] >> k) & 1u)) x = 0.f;
                            if (!((vis[c4] >> (k + 1)) & 1u)) y = 0.f;
                        }
                        sum2[i & 1] = add_f2(sum2[i & 1], pack_f2(x, y));
                        pk[i] = pack2<T>(x, y);
                    }
                    tmem_st32(s_addr + half * 32, pk);     // over the scores: this thread's row, already in registers
                    tmem_st_wait();
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(half ? &sh->p_ready[t] : &sh->p_half[t]);
                }
            };
            if (need_mask) exps(std::true_type{}); else exps(std::false_type{});
            float s0, s1;
            unpack_f2(add_f2(sum2[0], sum2[1]), s0, s1);
            l_run += s0 + s1;
            ++n;
        }
        if (ok && n > 0) {
            if (!mbar_wait_warp(smem_u32(&sh->o_full[t]), 0u)) { if (lane == 0) fail(sh, 12); ok = false; }
        }
        if (ok && t < p.per_cta && qt0 + t < p.q_tiles) {
            // normalise and store the row (the tensor-memory loads are warp-wide; only the stores depend on the row)
            const float inv = l_run > 0.f ? 1.f / l_run : 0.f;
            T* orow = (T*)p.o + (int64_t)b * p.o_batch + qi * p.o_tok + (int64_t)head * p.o_head;
            tc_fence_after();
#pragma unroll
            for (int c4 = 0; c4 < HD / 32; ++c4) {
                uint32_t o[32];
                if (n > 0) {
                    tmem_ld32(o_addr + c4 * 32, o);
                    tmem_ld_wait();
                } else {
#pragma unroll
                    for (int i = 0; i < 32; ++i) o[i] = 0u;
                }
                if (row_ok) {
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        if (c4 * 32 + q * 8 < p.d) {
                            bmt::Vec16<T> ov;
#pragma unroll
                            for (int i = 0; i < 8; ++i) ov.v[i] = bmt::Cvt<T>::from_f(__uint_as_float(o[q * 8 + i]) * inv);
                            bmt::st16(orow + c4 * 32 + q * 8, ov);
                        }
                    }
                }
            }
            tc_fence_before();
            if (row_ok && p.lse)
                p.lse[((int64_t)b * p.h + head) * p.sq + qi] = l_run > 0.f ? (m_ref * p.sl2 + log2f(l_run)) * 0.6931471805599453f : -INFINITY;
        }
    }

    // ---------------------------------------------------------------------------------------------- teardown
    __syncthreads();
    if (sh->failed) {
        // a wait ran out: give copies that are still in flight time to land before the shared memory goes away
        const uint64_t t0 = global_ns();
        while (global_ns() - t0 < 2000000ull) __nanosleep(1000);
        __syncthreads();
    }
    tc_fence_after();
    if (warp == 9) tmem_dealloc(tmem, 512);
}

template <int HD, typename T>
int launch_fwd(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, AttnParams& p, int64_t batch, cudaStream_t stream) {
    constexpr uint32_t TB = (HD / 64) * CHUNK;
    const size_t smem = 6 * TB + sizeof(AttnShared) + 1024;
    static bool configured = false;
    if (!configured) {
        if (cudaFuncSetAttribute(flash_fwd_kernel<HD, T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) return -30;
        configured = true;
    }
    // pairs of query tiles unless single tiles still find an SM each: a pair shares its K / V loads and hides one tile's
    // softmax behind the other's MMAs, two SMs are faster still
    p.per_cta = (int64_t)p.q_tiles * p.h * batch > bmt::sm_count() ? 2 : 1;
    dim3 grid((unsigned)(p.h * batch), (unsigned)((p.q_tiles + p.per_cta - 1) / p.per_cta));
    bmt::launch(flash_fwd_kernel<HD, T>, grid, FWD_THREADS, smem, stream, 1, tq, tk, tv, p);
    bmt_count_launch(1);
    return cudaGetLastError() == cudaSuccess ? 0 : -31;
}

// ================================================================================================ backward
// One CTA per (128 keys, kv head, sample).  K and V tiles stay in shared memory; the CTA walks over the query heads that
// share the kv head and over the query tiles that can see its keys.  Scores are held transposed (lane = key, column =
// query), so that P^T and dS^T are the A operands of dV += P^T dO and dK += dS^T Q as they stand.  Per (query, key) tile:
//   MMA   S^T = K Q^T and dP^T = V dO^T into tensor memory
//   softmax warps (8, two per 32 keys, 64 queries each): P = exp2(S * scale * log2e - lse * log2e) (masked) back into
//         tensor memory as packed 16-bit pairs, over S^T; dS = P * (dP - delta) * scale as 16 bits into shared memory,
//         [key][query] swizzled: K-major A for dK and, read "transposed", MN-major A for dQ = dS K
//   MMA   dV += P^T dO (P from tensor memory), dK += dS^T Q, dQ = dS K
//   one warp fetches lse and delta of the tiles to come
//   dQ warps (4): add the tile of dQ to an fp32 accumulator in global memory (bulk reductions out of shared memory, 32 columns
//         at a time through two buffers a warp: with one, waiting for it to be read made a tile 4065 clocks of their time; vector
//         reductions by the threads themselves took 4300); a small kernel converts it
// delta = rowsum(dO * O) comes from a pre-pass.  dK / dV are written once at the end, already summed over the group.
// Order on the tensor pipe, which bounds a tile at 5 x 512 clocks (head dim 128): dP(i), dV(i), S(i+1), dK(i), dQ(i), dP(i+1):
// while the softmax warps turn dP(i) into dS(i) the pipe has dV(i) and S(i+1) to do, and while it does dK(i) and dQ(i) they
// exponentiate S(i+1).  dQ(i) shares its columns with dP, so dP(i+1) waits until the dQ warps have read them; with head
// dims up to 80 dQ has columns of its own.  All five products in turn with one group of four warps doing everything in
// between took 13 600 clocks a tile.
struct AttnBwdParams {
    int64_t sq, sk;
    int h, hk, d;
    float sl2, scale;
    int causal;
    int64_t causal_off;
    const uint32_t* bits_t;     // packed mask by key (b, sk, query tiles, 4 words) or null
    const uint8_t* cls;         // (b, query tiles, key tiles), see the forward kernel
    const int32_t* kv_lens;
    const float* lse;
    const float* delta;
    float* dq_acc;              // (b, h, sq, d) fp32, zero on entry
    void* dk; void* dv;         // (b, sk, hk, d) by strides {token, head, batch}
    int64_t dk_tok, dk_head, dk_batch, dv_tok, dv_head, dv_batch;
    uint32_t idesc_s, idesc_dv, idesc_dq;
    int q_tiles, k_tiles;
    int splits;                 // CTAs that share the query heads of one kv head; above 1 they leave fp32 parts in dkv_part
    float* dkv_part;            // (splits, 2: dK / dV, b, sk, hk, d)
    int64_t part_elems;         // b * sk * hk * d
};

constexpr uint32_t DQ_BUF = 32 * 128;            // exchange buffer of a dQ warp: 32 rows x 32 floats; each warp has two
constexpr int BWD_THREADS = 512;                 // 8 softmax warps, 4 dQ warps, producer and MMA issuer (a warpgroup of their own)

struct BwdShared {
    alignas(16) uint64_t kv_full; uint64_t q_full[2], q_empty[2], do_full, do_empty, s_full, dp_full, p_ready, ds_ready, dq_full, dq_empty, all_done;
    uint64_t row_full[2], row_empty[2];
    float nlse[2][TILE], ndelta[2][TILE];        // per query of a tile: -lse * log2(e) (0 for rows that take no part), -delta * scale
    uint32_t live[2][4];                         // queries of the tile that exist and see at least one key
    uint32_t tmem_base;
    int failed;
};

__device__ __forceinline__ void fail_bwd(BwdShared* sh, int code) {
    sh->failed = 1;
    atomicCAS(&g_attn_status, 0, ((0x40 | code) << 16) | (int)(blockIdx.x & 0xffff));
}

// Walks the (head, query tile) pairs of a CTA in order, leaving out tiles without a visible pair.
struct BwdWalk {
    int head, qt, head_end, qt_first, q_tiles, k_tiles;
    const uint8_t* cls;        // class of (query tile, this key tile), row pitch k_tiles; or null
    __device__ __forceinline__ void settle() {
        while (head < head_end) {
            while (qt < q_tiles && cls && cls[(int64_t)qt * k_tiles] == 0) ++qt;
            if (qt < q_tiles) return;
            ++head;
            qt = qt_first;
        }
    }
    __device__ __forceinline__ bool more() const { return head < head_end; }
    __device__ __forceinline__ void next() { ++qt; settle(); }
};

template <int HD, typename T>
__global__ void __launch_bounds__(BWD_THREADS, 1)
flash_bwd_kernel(const __grid_constant__ CUtensorMap tq, const __grid_constant__ CUtensorMap tk, const __grid_constant__ CUtensorMap tv,
                 const __grid_constant__ CUtensorMap tdo, const __grid_constant__ CUtensorMap tdq, const AttnBwdParams p) {
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t* smem = smem_raw;         // swizzled tiles want 1024-byte alignment, there is no room to round up: launch_bwd looks after it
    constexpr int DC = HD / 64;
    constexpr uint32_t TB = DC * CHUNK;
    const uint32_t sK = smem_u32(smem), sV = sK + TB, sQ = sV + TB, sdO = sQ + 2 * TB, sdS = sdO + TB, sX = sdS + 2 * CHUNK;
    BwdShared* sh = (BwdShared*)(smem + 5 * TB + 2 * CHUNK + 8 * DQ_BUF);
    // tensor memory columns: S^T / P^T [0,128), dP^T [128,256), dV, dK, dQ each of d columns; above head dim 80 dQ takes dP's
    const uint32_t C_DP = 128, C_DV = 256, C_DK = C_DV + p.d, C_DQ = p.d <= 80 ? C_DK + p.d : C_DP;
    const bool dq_shared = p.d > 80;
    // Registers of the producer / issuer warpgroup and of the other three, of the 512 x 128 at launch.  The unrolled issue of 8-step
    // products wants more than 48 (2x4096, 20 x 128 causal: 505 us with 48 / 152, 493 with 72 / 144); with 4 steps 48 do, and the
    // softmax has use for the rest (1x8192, 16 x 64 causal: 460 against 464).
    constexpr int FEW = HD == 128 ? 72 : 48, MANY = HD == 128 ? 144 : 152;
    static_assert(128 * FEW + 384 * MANY <= 512 * 128, "registers of a block");

    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        mbar_init(&sh->kv_full, 1); mbar_init(&sh->do_full, 1); mbar_init(&sh->do_empty, 1);
        for (int i = 0; i < 2; ++i) { mbar_init(&sh->q_full[i], 1); mbar_init(&sh->q_empty[i], 1); mbar_init(&sh->row_full[i], 1); mbar_init(&sh->row_empty[i], 8); }
        mbar_init(&sh->s_full, 1); mbar_init(&sh->dp_full, 1); mbar_init(&sh->p_ready, 8); mbar_init(&sh->ds_ready, 8);
        mbar_init(&sh->dq_full, 1); mbar_init(&sh->dq_empty, 4); mbar_init(&sh->all_done, 1);
        sh->failed = 0;
        fence_barrier_init();
    }
    if (warp == 13) { tmem_alloc(&sh->tmem_base, 512); tmem_relinquish(); }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    bmt::after_previous();
    const int kvh = blockIdx.x % p.hk, b = blockIdx.x / p.hk, kt = blockIdx.y;   // under a causal mask the long columns start first
    const int group = p.h / p.hk / p.splits;     // query heads of this CTA
    const int64_t kv0 = (int64_t)kt * TILE;
    int64_t kv_valid = p.sk;
    if (p.kv_lens && p.kv_lens[b] < kv_valid) kv_valid = p.kv_lens[b];
    BwdWalk walk;
    walk.qt_first = 0;
    if (p.causal && kv0 - p.causal_off > 0) walk.qt_first = (int)((kv0 - p.causal_off) / TILE);
    walk.qt = walk.qt_first; walk.q_tiles = p.q_tiles; walk.k_tiles = p.k_tiles;
    walk.head = (kvh * p.splits + (int)blockIdx.z) * group; walk.head_end = kv0 < kv_valid ? walk.head + group : walk.head;
    walk.cls = p.cls ? p.cls + (int64_t)b * p.q_tiles * p.k_tiles + kt : nullptr;
    walk.settle();
    const bool work = walk.more();

    const uint32_t tmem = sh->tmem_base;

    if (warp >= 12) {
    regs_down<FEW>();
    if (warp == 12) {
        // ------------------------------------------------------------------------------------------ TMA producer
        if (work) {
            const uint32_t kvbar = smem_u32(&sh->kv_full);
            if (elect_one()) {
                mbar_expect_tx_u32(kvbar, 2 * TB);
#pragma unroll
                for (int c = 0; c < DC; ++c) {
                    tma_load_4d_u32(&tk, kvbar, sK + c * CHUNK, c * 64, (int)kv0, kvh, b);
                    tma_load_4d_u32(&tv, kvbar, sV + c * CHUNK, c * 64, (int)kv0, kvh, b);
                }
            }
            __syncwarp();
            for (uint32_t it = 0; walk.more(); walk.next(), ++it) {
                const uint32_t st = it & 1, ph = (it >> 1) & 1;
                if (!mbar_wait_warp(smem_u32(&sh->q_empty[st]), ph ^ 1)) { if (lane == 0) fail_bwd(sh, 1); break; }
                if (elect_one()) {
                    const uint32_t bar = smem_u32(&sh->q_full[st]);
                    mbar_expect_tx_u32(bar, TB);
#pragma unroll
                    for (int c = 0; c < DC; ++c) tma_load_4d_u32(&tq, bar, sQ + st * TB + c * CHUNK, c * 64, walk.qt * TILE, walk.head, b);
                }
                __syncwarp();
                if (!mbar_wait_warp(smem_u32(&sh->do_empty), (it & 1) ^ 1)) { if (lane == 0) fail_bwd(sh, 2); break; }
                if (elect_one()) {
                    const uint32_t bar = smem_u32(&sh->do_full);
                    mbar_expect_tx_u32(bar, TB);
#pragma unroll
                    for (int c = 0; c < DC; ++c) tma_load_4d_u32(&tdo, bar, sdO + c * CHUNK, c * 64, walk.qt * TILE, walk.head, b);
                }
                __syncwarp();
            }
        }
    } else if (warp == 13) {
        // ------------------------------------------------------------------------------------------ MMA issuer
        if (work) {
            const uint32_t hi = desc_hi(1024);
            const int ks_d = p.d / 16;
            bool ok = mbar_wait_warp(smem_u32(&sh->kv_full), 0);
            if (!ok && lane == 0) fail_bwd(sh, 3);
            auto issue_s = [&](uint32_t it) -> bool {       // S^T = K Q^T of tile `it`
                const uint32_t st = it & 1;
                if (!mbar_wait_warp(smem_u32(&sh->q_full[st]), (it >> 1) & 1)) { if (lane == 0) fail_bwd(sh, 4); return false; }
                tc_fence_after();
                if (elect_one()) {
                    const uint32_t kd = desc_lo(sK, 0), qd = desc_lo(sQ + st * TB, 0);
#pragma unroll
                    for (int ks = 0; ks < HD / 16; ++ks) {       // unrolled, see the forward kernel
                        const uint32_t off = (uint32_t)((ks >> 2) * CHUNK + (ks & 3) * 32) >> 4;
                        if (ks < ks_d) umma_f16(tmem, pack_desc(kd + off, hi), pack_desc(qd + off, hi), p.idesc_s, ks != 0 ? 1u : 0u);
                    }
                    umma_commit(&sh->s_full);
                }
                __syncwarp();
                return true;
            };
            ok = ok && issue_s(0);
            for (uint32_t it = 0; ok && walk.more(); ++it) {
                const uint32_t ph = it & 1, st = it & 1;
                walk.next();
                if (!mbar_wait_warp(smem_u32(&sh->do_full), ph)) { if (lane == 0) fail_bwd(sh, 5); break; }
                // dP's columns: dS(it-1) was computed from them before dK(it-1) could be issued; dQ(it-1) has to be out of them
                if (dq_shared && !mbar_wait_warp(smem_u32(&sh->dq_empty), ph ^ 1)) { if (lane == 0) fail_bwd(sh, 6); break; }
                tc_fence_after();
                if (elect_one()) {
                    const uint32_t vd = desc_lo(sV, 0), od = desc_lo(sdO, 0);
#pragma unroll
                    for (int ks = 0; ks < HD / 16; ++ks) {
                        const uint32_t off = (uint32_t)((ks >> 2) * CHUNK + (ks & 3) * 32) >> 4;
                        if (ks < ks_d) umma_f16(tmem + C_DP, pack_desc(vd + off, hi), pack_desc(od + off, hi), p.idesc_s, ks != 0 ? 1u : 0u);
                    }
                    umma_commit(&sh->dp_full);
                }
                __syncwarp();
                if (!mbar_wait_warp(smem_u32(&sh->p_ready), ph)) { if (lane == 0) fail_bwd(sh, 7); break; }
                tc_fence_after();
                if (elect_one()) {
#pragma unroll
                    for (int ks = 0; ks < TILE / 16; ++ks)      // dV += P^T dO: 16 queries per step, dO MN-major
                        umma_f16_ts(tmem + C_DV, tmem + (ks >> 2) * 64 + (ks & 3) * 8, pack_desc(desc_lo(sdO + ks * 2048, CHUNK), hi), p.idesc_dv, (it | (uint32_t)ks) != 0 ? 1u : 0u);
                    umma_commit(&sh->do_empty);
                }
                __syncwarp();
                if (walk.more() && !issue_s(it + 1)) break;
                if (!mbar_wait_warp(smem_u32(&sh->ds_ready), ph)) { if (lane == 0) fail_bwd(sh, 8); break; }
                if (!dq_shared && !mbar_wait_warp(smem_u32(&sh->dq_empty), ph ^ 1)) { if (lane == 0) fail_bwd(sh, 9); break; }
                tc_fence_after();
                if (elect_one()) {
#pragma unroll
                    for (int ks = 0; ks < TILE / 16; ++ks)      // dQ = dS K: 16 keys per step, both operands MN-major
                        umma_f16(tmem + C_DQ, pack_desc(desc_lo(sdS + ks * 2048, CHUNK), hi), pack_desc(desc_lo(sK + ks * 2048, CHUNK), hi),
                                 p.idesc_dq, ks != 0 ? 1u : 0u);
                    umma_commit(&sh->dq_full);
#pragma unroll
                    for (int ks = 0; ks < TILE / 16; ++ks)      // dK += dS^T Q: 16 queries per step, A K-major, Q MN-major
                        umma_f16(tmem + C_DK, pack_desc(desc_lo(sdS + (ks >> 2) * CHUNK + (ks & 3) * 32, 0), hi),
                                 pack_desc(desc_lo(sQ + st * TB + ks * 2048, CHUNK), hi), p.idesc_dv, (it | (uint32_t)ks) != 0 ? 1u : 0u);
                    umma_commit(&sh->q_empty[st]);
                    if (!walk.more()) umma_commit(&sh->all_done);
                }
                __syncwarp();
            }
        }
    } else if (warp == 14) {
        // ------------------------------------------------------------------------------------------ row statistics, up to two tiles ahead
        for (uint32_t it = 0; walk.more(); walk.next(), ++it) {
            const uint32_t st = it & 1;
            if (!mbar_wait_warp(smem_u32(&sh->row_empty[st]), ((it >> 1) & 1) ^ 1)) { if (lane == 0) fail_bwd(sh, 15); break; }
            const int64_t q0 = (int64_t)walk.qt * TILE + lane, at = ((int64_t)b * p.h + walk.head) * p.sq + q0;
            float l[4], dl[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const bool in = q0 + i * 32 < p.sq;
                l[i] = in ? p.lse[at + i * 32] : -INFINITY;
                dl[i] = in ? p.delta[at + i * 32] : 0.f;
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const bool alive = l[i] != -INFINITY;
                sh->nlse[st][i * 32 + lane] = alive ? -l[i] * 1.4426950408889634f : 0.f;
                sh->ndelta[st][i * 32 + lane] = -dl[i] * p.scale;
                const uint32_t bits = __ballot_sync(0xffffffffu, alive);
                if (lane == 0) sh->live[st][i] = bits;
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&sh->row_full[st]);
        }
    }
    } else if (warp < 8) {
        // ------------------------------------------------------------------------------------------ softmax: P and dS
        regs_up<MANY>();
        const int quarter = warp & 3, part = warp >> 2;             // 32 keys, 64 queries of the tile
        const int row = quarter * 32 + lane;
        const int64_t kj = kv0 + row;                                // this thread's key
        const uint32_t lane_addr = (uint32_t)(quarter * 32) << 16;
        const uint4* brow = (p.bits_t && kj < p.sk) ? reinterpret_cast<const uint4*>(p.bits_t) + ((int64_t)b * p.sk + kj) * p.q_tiles : nullptr;
        const uint64_t sl2_2 = pack_f2(p.sl2, p.sl2), scale_2 = pack_f2(p.scale, p.scale);
        bool ok = true;
        uint32_t it = 0;
        for (; walk.more() && ok; walk.next(), ++it) {
            const uint32_t ph = it & 1, st = it & 1;
            const int64_t q0 = (int64_t)walk.qt * TILE;
            const int kind = walk.cls ? walk.cls[(int64_t)walk.qt * p.k_tiles] : 2;
            if (!mbar_wait_warp(smem_u32(&sh->row_full[st]), (it >> 1) & 1)) { if (lane == 0) fail_bwd(sh, 10); ok = false; break; }
            uint32_t vis[2];
            vis[0] = sh->live[st][part * 2]; vis[1] = sh->live[st][part * 2 + 1];
            bool need_mask = kind == 1 || kv0 + TILE > kv_valid || (p.causal && kv0 + TILE - 1 > q0 + p.causal_off) ||
                             (vis[0] & vis[1]) != 0xffffffffu;
            if (need_mask) {
                if (kj >= kv_valid) vis[0] = vis[1] = 0u;
                if (p.causal) {          // query q0 + c sees this key from c = kj - causal_off - q0 on
                    const int64_t c0 = kj - p.causal_off - q0 - part * 64;
                    vis[0] &= ~low_bits(c0);
                    vis[1] &= ~low_bits(c0 - 32);
                }
                if (kind == 1 && brow) {
                    const uint4 w = brow[walk.qt];
                    vis[0] &= part ? w.z : w.x;
                    vis[1] &= part ? w.w : w.y;
                }
            }
            if (!mbar_wait_warp(smem_u32(&sh->s_full), ph)) { if (lane == 0) fail_bwd(sh, 11); ok = false; break; }
            tc_fence_after();
            uint32_t s[2][32];
            tmem_ld32(tmem + lane_addr + part * 64, s[0]);
            tmem_ld32(tmem + lane_addr + part * 64 + 32, s[1]);
            tmem_ld_wait();
            float pr[64];
            uint32_t pk[32];
#pragma unroll
            for (int i = 0; i < 16; ++i) {
                const int u = i >> 3, k = (4 * i) & 31;
                const float4 nl = *reinterpret_cast<const float4*>(&sh->nlse[st][part * 64 + 4 * i]);
                float x[4];
                unpack_f2(fma_f2(pack_f2(__uint_as_float(s[u][k]), __uint_as_float(s[u][k + 1])), sl2_2, pack_f2(nl.x, nl.y)), x[0], x[1]);
                unpack_f2(fma_f2(pack_f2(__uint_as_float(s[u][k + 2]), __uint_as_float(s[u][k + 3])), sl2_2, pack_f2(nl.z, nl.w)), x[2], x[3]);
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    x[e] = ex2(x[e]);
                    if (need_mask && !((vis[u] >> (k + e)) & 1u)) x[e] = 0.f;
                    pr[4 * i + e] = x[e];
                }
                pk[2 * i] = pack2<T>(x[0], x[1]);
                pk[2 * i + 1] = pack2<T>(x[2], x[3]);
            }
            // over this warp's own half of the scores: queries [0,64) go to columns [0,32), queries [64,128) to [64,96)
            tmem_st32(tmem + lane_addr + part * 64, pk);
            tmem_st_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&sh->p_ready);
            if (!mbar_wait_warp(smem_u32(&sh->dp_full), ph)) { if (lane == 0) fail_bwd(sh, 12); ok = false; break; }
            tc_fence_after();
            tmem_ld32(tmem + lane_addr + C_DP + part * 64, s[0]);
            // dS(it-1) in shared memory may still be read by dQ / dK(it-1): wait for the commit behind both
            if (it > 0 && !mbar_wait_warp(smem_u32(&sh->q_empty[st ^ 1]), ((it - 1) >> 1) & 1)) { if (lane == 0) fail_bwd(sh, 13); ok = false; break; }
            const uint32_t base = sdS + (uint32_t)part * CHUNK + (uint32_t)row * 128;
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                tmem_ld_wait_for(s[0]);
#pragma unroll
                for (int t = 0; t < 4; ++t) {
                    uint32_t w[4];
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        const int k = t * 8 + 4 * i, e = u * 32 + k;
                        const float4 nd = *reinterpret_cast<const float4*>(&sh->ndelta[st][part * 64 + e]);
                        float a, c;
                        // dS = P * (dP * scale - delta * scale)
                        unpack_f2(mul_f2(pack_f2(pr[e], pr[e + 1]), fma_f2(pack_f2(__uint_as_float(s[0][k]), __uint_as_float(s[0][k + 1])), scale_2, pack_f2(nd.x, nd.y))), a, c);
                        w[2 * i] = pack2<T>(a, c);
                        unpack_f2(mul_f2(pack_f2(pr[e + 2], pr[e + 3]), fma_f2(pack_f2(__uint_as_float(s[0][k + 2]), __uint_as_float(s[0][k + 3])), scale_2, pack_f2(nd.z, nd.w))), a, c);
                        w[2 * i + 1] = pack2<T>(a, c);
                    }
                    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(base + (uint32_t)(((u * 4 + t) ^ (row & 7)) << 4)), "r"(w[0]),
                                 "r"(w[1]), "r"(w[2]), "r"(w[3]) : "memory");
                }
                if (u == 0) tmem_ld32(tmem + lane_addr + C_DP + part * 64 + 32, s[0]);
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            tc_fence_before();
            __syncwarp();
            if (lane == 0) { mbar_arrive(&sh->ds_ready); mbar_arrive(&sh->row_empty[st]); }
        }
        // dK, dV rows of this CTA's keys (zeros when no query sees them): part 0 writes dK, part 1 dV.  The tensor-memory
        // loads are warp-wide, so every lane takes part in them; only the stores depend on the row.
        if (ok && it > 0 && !mbar_wait_warp(smem_u32(&sh->all_done), 0)) { if (lane == 0) fail_bwd(sh, 14); ok = false; }
        if (ok) {
            tc_fence_after();
            T* dst = part == 0 ? (T*)p.dk + (int64_t)b * p.dk_batch + kj * p.dk_tok + (int64_t)kvh * p.dk_head
                               : (T*)p.dv + (int64_t)b * p.dv_batch + kj * p.dv_tok + (int64_t)kvh * p.dv_head;
            const uint32_t src = tmem + lane_addr + (part == 0 ? C_DK : C_DV);
#pragma unroll
            for (int c16 = 0; c16 < HD / 16; ++c16) {
                if (c16 * 16 < p.d) {
                    uint32_t r[16];
                    if (it > 0) {
                        tmem_ld16(src + c16 * 16, r);
                        tmem_ld_wait();
                    } else {
#pragma unroll
                        for (int i = 0; i < 16; ++i) r[i] = 0u;
                    }
                    if (kj < p.sk && p.splits > 1) {
                        float* part_dst = p.dkv_part + ((int64_t)blockIdx.z * 2 + part) * p.part_elems + (((int64_t)b * p.sk + kj) * p.hk + kvh) * p.d + c16 * 16;
#pragma unroll
                        for (int q = 0; q < 4; ++q)
                            reinterpret_cast<float4*>(part_dst)[q] = make_float4(__uint_as_float(r[4 * q]), __uint_as_float(r[4 * q + 1]),
                                                                                 __uint_as_float(r[4 * q + 2]), __uint_as_float(r[4 * q + 3]));
                    } else if (kj < p.sk) {
#pragma unroll
                        for (int q = 0; q < 2; ++q) {
                            bmt::Vec16<T> ov;
#pragma unroll
                            for (int i = 0; i < 8; ++i) ov.v[i] = bmt::Cvt<T>::from_f(__uint_as_float(r[q * 8 + i]));
                            bmt::st16(dst + c16 * 16 + q * 8, ov);
                        }
                    }
                }
            }
            tc_fence_before();
        }
    } else {
        // ------------------------------------------------------------------------------------------ dQ
        regs_up<MANY>();
        const int quarter = warp & 3, r0 = quarter * 32;
        const uint32_t lane_addr = (uint32_t)r0 << 16, xbufs = sX + (uint32_t)(warp - 8) * 2 * DQ_BUF;
        bool ok = true;
        for (uint32_t it = 0; walk.more() && ok; walk.next(), ++it) {
            if (!mbar_wait_warp(smem_u32(&sh->dq_full), it & 1)) { if (lane == 0) fail_bwd(sh, 16); ok = false; break; }
            tc_fence_after();
            uint32_t r[HD / 32][32];
#pragma unroll
            for (int c4 = 0; c4 < HD / 32; ++c4)
                if (c4 * 32 < p.d) tmem_ld32(tmem + lane_addr + C_DQ + c4 * 32, r[c4]);
            tmem_ld_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&sh->dq_empty);
            // 32 columns at a time into the buffer (16-byte units swizzled as the tensor map says), one bulk reduction each
#pragma unroll
            for (int c4 = 0; c4 < HD / 32; ++c4) {
                if (c4 * 32 >= p.d) break;
                const uint32_t xbuf = xbufs + (c4 & 1) * DQ_BUF;
                // the buffers in turn: all of the previous tile have been read by now, from the third on the last but one has
                if (lane == 0 && c4 == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
                if (lane == 0 && c4 >= 2) asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
                __syncwarp();
                const uint32_t srow = xbuf + (uint32_t)lane * 128;
#pragma unroll
                for (int q = 0; q < 8; ++q)
                    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(srow + (uint32_t)((q ^ (lane & 7)) << 4)), "r"(r[c4][4 * q]),
                                 "r"(r[c4][4 * q + 1]), "r"(r[c4][4 * q + 2]), "r"(r[c4][4 * q + 3]) : "memory");
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncwarp();
                if (lane == 0) {
                    asm volatile("cp.reduce.async.bulk.tensor.3d.global.shared::cta.add.tile.bulk_group [%0, {%2, %3, %4}], [%1];"
                                 ::"l"(&tdq), "r"(xbuf), "r"(c4 * 32), "r"(walk.qt * TILE + r0), "r"(b * p.h + walk.head) : "memory");
                    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
                }
            }
        }
        if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");   // the reductions read this CTA's shared memory
    }

    __syncthreads();
    if (sh->failed) {
        const uint64_t t0 = global_ns();
        while (global_ns() - t0 < 2000000ull) __nanosleep(1000);
        __syncthreads();
    }
    tc_fence_after();
    if (warp == 13) tmem_dealloc(tmem, 512);
}

// Row `w` of all (sample, token, head); divisions of 32 bits where they do (a 64-bit one is a hundred instructions, for 16 bytes a thread).
struct Place { int64_t b, q; int head; };
__device__ __forceinline__ Place place_of(int64_t w, int64_t rows, int64_t sq, int h) {
    if (rows <= 0x7fffffff) {
        const uint32_t n = (uint32_t)w, tok = n / (uint32_t)h, b = tok / (uint32_t)sq;
        return {b, tok - b * (uint32_t)sq, (int)(n - tok * (uint32_t)h)};
    }
    const int64_t tok = w / h, b = tok / sq;
    return {b, tok - b * sq, (int)(w - tok * h)};
}

// delta[b, h, q] = sum_d dO[b, q, h, d] * O[b, q, h, d], and zeros in the same row of the dQ accumulator (b, h, sq, d); 16
// lanes per row (head dims up to 128 are 16 vectors of 8), two rows per warp.
template <typename T>
__global__ void attn_delta_kernel(const T* o, int64_t o_tok, int64_t o_head, int64_t o_batch, const T* dout, int64_t g_tok, int64_t g_head,
                                  int64_t g_batch, float* delta, float* dq_acc, int64_t rows, int64_t sq, int h, int d) {
    bmt::after_previous();
    const int64_t w = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 4;
    const int c = (threadIdx.x & 15) * 8;
    const bool ok = w < rows;
    const Place at = place_of(ok ? w : 0, rows, sq, h);
    const int head = at.head;
    const int64_t bb = at.b, qi = at.q, row = (bb * h + head) * sq + qi;
    float acc = 0.f;
    if (ok && c < d) {
        const bmt::Vec16<T> a = bmt::ld16(o + bb * o_batch + qi * o_tok + head * o_head + c), g = bmt::ld16(dout + bb * g_batch + qi * g_tok + head * g_head + c);
#pragma unroll
        for (int i = 0; i < 8; ++i) acc += bmt::Cvt<T>::to_f(a.v[i]) * bmt::Cvt<T>::to_f(g.v[i]);
        float4* z = reinterpret_cast<float4*>(dq_acc + row * d + c);
        z[0] = z[1] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
#pragma unroll
    for (int s = 8; s > 0; s >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, s);
    if (ok && c == 0) delta[row] = acc;
}

// dq[b, q, h, :] (strided, T) <- dq_acc (b, h, sq, d) fp32
template <typename T>
__global__ void attn_dq_convert_kernel(const float* acc, T* dq, int64_t q_tok, int64_t q_head, int64_t q_batch, int64_t rows, int64_t sq,
                                       int h, int d) {
    bmt::after_previous();
    const int64_t w = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 4;
    const int c = (threadIdx.x & 15) * 8;
    if (w >= rows || c >= d) return;
    const Place at = place_of(w, rows, sq, h);
    const int head = at.head;
    const int64_t bb = at.b, qi = at.q;
    const float4* src = reinterpret_cast<const float4*>(acc + ((bb * h + head) * sq + qi) * d + c);
    const float4 a0 = src[0], a1 = src[1];
    bmt::Vec16<T> o;
    o.v[0] = bmt::Cvt<T>::from_f(a0.x); o.v[1] = bmt::Cvt<T>::from_f(a0.y); o.v[2] = bmt::Cvt<T>::from_f(a0.z); o.v[3] = bmt::Cvt<T>::from_f(a0.w);
    o.v[4] = bmt::Cvt<T>::from_f(a1.x); o.v[5] = bmt::Cvt<T>::from_f(a1.y); o.v[6] = bmt::Cvt<T>::from_f(a1.z); o.v[7] = bmt::Cvt<T>::from_f(a1.w);
    bmt::st16(dq + bb * q_batch + qi * q_tok + head * q_head + c, o);
}

// dk / dv (strided, T) <- sum of the parts in split order; one 8-element vector per thread, dK in the first half of the grid
template <typename T>
__global__ void attn_dkv_sum_kernel(const float* part, int splits, int64_t elems, int64_t sk, int hk, int d, T* dk, int64_t k_tok, int64_t k_head,
                                    int64_t k_batch, T* dv, int64_t v_tok, int64_t v_head, int64_t v_batch) {
    bmt::after_previous();
    const int64_t vecs = elems / 8;
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= 2 * vecs) return;
    const int which = i >= vecs ? 1 : 0;
    i -= which * vecs;
    float acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    for (int sp = 0; sp < splits; ++sp) {
        const float4* src = reinterpret_cast<const float4*>(part + ((int64_t)sp * 2 + which) * elems + i * 8);
        const float4 a = src[0], c = src[1];
        acc[0] += a.x; acc[1] += a.y; acc[2] += a.z; acc[3] += a.w; acc[4] += c.x; acc[5] += c.y; acc[6] += c.z; acc[7] += c.w;
    }
    const int per = d / 8;
    const int64_t row = i / per, tok = row / hk;
    const int col = (int)(i - row * per) * 8, head = (int)(row - tok * hk);
    const int64_t bb = tok / sk, kj = tok - bb * sk;
    bmt::Vec16<T> o;
#pragma unroll
    for (int e = 0; e < 8; ++e) o.v[e] = bmt::Cvt<T>::from_f(acc[e]);
    T* dst = which ? dv + bb * v_batch + kj * v_tok + head * v_head : dk + bb * k_batch + kj * k_tok + head * k_head;
    bmt::st16(dst + col, o);
}

// CTAs that share the query heads of a kv head.  Without a split there is a CTA per key tile, kv head and sample, which walks
// over all query heads of the group: one kv head leaves most SMs idle, and under a causal mask the CTA of the first keys sets
// the pace (1x2048, 64 / 8 heads x 128: 128 CTAs, 408 us).  The heads are shared out until there are two CTAs per SM.
int bwd_splits(int64_t batch, int64_t sk, int h, int hk) {
    const int group = h / hk;
    const int64_t ctas = (sk + TILE - 1) / TILE * hk * batch;
    for (int s = 1; s < group; ++s)
        if (group % s == 0 && ctas * s >= 2 * bmt::sm_count()) return s;
    return group;
}

template <int HD, typename T>
int launch_bwd(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const CUtensorMap& tdo, const CUtensorMap& tdq, const AttnBwdParams& p,
               int64_t batch, cudaStream_t stream) {
    constexpr uint32_t TB = (HD / 64) * CHUNK;
    const size_t smem = 5 * TB + 2 * CHUNK + 8 * DQ_BUF + sizeof(BwdShared);
    static_assert(5 * 2 * CHUNK + 2 * CHUNK + 8 * DQ_BUF + sizeof(BwdShared) <= 227 * 1024, "shared memory of a block");
    static bool configured = false;
    if (!configured) {
        // what lies in front of the kernel's own shared memory: the system's share and static arrays
        int dev = 0, reserved = 0;
        cudaFuncAttributes attr;
        if (cudaGetDevice(&dev) != cudaSuccess || cudaFuncGetAttributes(&attr, flash_bwd_kernel<HD, T>) != cudaSuccess ||
            cudaDeviceGetAttribute(&reserved, cudaDevAttrReservedSharedMemoryPerBlock, dev) != cudaSuccess) return -30;
        if ((reserved + attr.sharedSizeBytes) % 1024 != 0) return -34;
        if (cudaFuncSetAttribute(flash_bwd_kernel<HD, T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) return -30;
        configured = true;
    }
    dim3 grid((unsigned)(p.hk * batch), (unsigned)p.k_tiles, (unsigned)p.splits);
    bmt::launch(flash_bwd_kernel<HD, T>, grid, BWD_THREADS, smem, stream, 1, tq, tk, tv, tdo, tdq, p);
    bmt_count_launch(1);
    return cudaGetLastError() == cudaSuccess ? 0 : -31;
}

template <typename T>
int run_bwd(int64_t batch, int64_t sq, int64_t sk, int h, int hk, int d, const void* q, const int64_t* qs, const void* k, const int64_t* ks,
            const void* v, const int64_t* vs, const void* o, const int64_t* os, const void* dout, const int64_t* gs, const void* lse,
            void* dq, const int64_t* dqs, void* dk, const int64_t* dks, void* dv, const int64_t* dvs, void* dq_acc, void* delta, float scale,
            int causal, const void* mask_bits_t, const void* mask_cls, const void* kv_lens, void* dkv_part, int dtype, cudaStream_t st) {
    const int hd = d <= 64 ? 64 : 128;
    CUtensorMap tq, tk, tv, tdo, tdq;
    int rc;
    if ((rc = bmt_tma_map_4d(&tq, q, dtype, d, sq, qs[0], h, qs[1], batch, qs[2], 64, TILE)) != 0) return rc;
    if ((rc = bmt_tma_map_4d(&tk, k, dtype, d, sk, ks[0], hk, ks[1], batch, ks[2], 64, TILE)) != 0) return rc;
    if ((rc = bmt_tma_map_4d(&tv, v, dtype, d, sk, vs[0], hk, vs[1], batch, vs[2], 64, TILE)) != 0) return rc;
    if ((rc = bmt_tma_map_4d(&tdo, dout, dtype, d, sq, gs[0], h, gs[1], batch, gs[2], 64, TILE)) != 0) return rc;
    if ((rc = bmt_tma_map_f32_3d(&tdq, dq_acc, d, sq, batch * h, 32, 32)) != 0) return rc;
    const int64_t rows = batch * sq * h;
    const unsigned row_blocks = (unsigned)((rows * 16 + 255) / 256);
    bmt::launch(attn_delta_kernel<T>, row_blocks, 256, 0, st, 1, (const T*)o, os[0], os[1], os[2], (const T*)dout, gs[0], gs[1], gs[2], (float*)delta,
                                                     (float*)dq_acc, rows, sq, h, d);
    AttnBwdParams p;
    memset(&p, 0, sizeof(p));
    p.sq = sq; p.sk = sk; p.h = h; p.hk = hk; p.d = d;
    p.scale = scale; p.sl2 = scale * 1.4426950408889634f;
    p.causal = causal; p.causal_off = sk - sq;
    p.bits_t = (const uint32_t*)mask_bits_t; p.cls = (const uint8_t*)mask_cls; p.kv_lens = (const int32_t*)kv_lens;
    p.q_tiles = (int)((sq + TILE - 1) / TILE); p.k_tiles = (int)((sk + TILE - 1) / TILE);
    p.splits = dkv_part ? bwd_splits(batch, sk, h, hk) : 1; p.dkv_part = (float*)dkv_part; p.part_elems = batch * sk * hk * d;
    p.lse = (const float*)lse; p.delta = (const float*)delta; p.dq_acc = (float*)dq_acc;
    p.dk = dk; p.dk_tok = dks[0]; p.dk_head = dks[1]; p.dk_batch = dks[2];
    p.dv = dv; p.dv_tok = dvs[0]; p.dv_head = dvs[1]; p.dv_batch = dvs[2];
    const uint32_t fmt = dtype == BMT_DT_F16 ? 0u : 1u;
    const uint32_t common = (1u << 4) | (fmt << 7) | (fmt << 10) | ((uint32_t)(TILE >> 4) << 24);
    p.idesc_s = common | ((uint32_t)(TILE >> 3) << 17);
    p.idesc_dv = common | (1u << 16) | ((uint32_t)(d >> 3) << 17);              // A K-major (or tensor memory), B MN-major, N = head dim
    p.idesc_dq = common | (1u << 15) | (1u << 16) | ((uint32_t)(d >> 3) << 17);  // A and B MN-major
    rc = hd == 64 ? launch_bwd<64, T>(tq, tk, tv, tdo, tdq, p, batch, st) : launch_bwd<128, T>(tq, tk, tv, tdo, tdq, p, batch, st);
    if (rc != 0) return rc;
    if (p.splits > 1) {
        const int64_t vecs = p.part_elems / 4;   // 8-element vectors of dK and dV
        bmt::launch(attn_dkv_sum_kernel<T>, (unsigned)((vecs + 255) / 256), 256, 0, st, 1, p.dkv_part, p.splits, p.part_elems, sk, hk, d, (T*)dk, dks[0], dks[1],
                                                                              dks[2], (T*)dv, dvs[0], dvs[1], dvs[2]);
        bmt_count_launch(1);
    }
    // Long grids wait for the kernel before them to end instead of for its last CTAs to begin: the backward of 2x4096, 20 x 128
    // causal 473 us so, 486 with blocks that sit on the SMs early; 2x512, 32 x 80 (2048 blocks) 41.4 and 40.1.
    if (row_blocks > 4u * 8u * (unsigned)bmt::sm_count())
        attn_dq_convert_kernel<T><<<row_blocks, 256, 0, st>>>((const float*)dq_acc, (T*)dq, dqs[0], dqs[1], dqs[2], rows, sq, h, d);
    else
        bmt::launch(attn_dq_convert_kernel<T>, row_blocks, 256, 0, st, 1, (const float*)dq_acc, (T*)dq, dqs[0], dqs[1], dqs[2], rows, sq, h, d);
    bmt_count_launch(2);
    return cudaGetLastError() == cudaSuccess ? 0 : -33;
}

}  // namespace

// q (b, sq, h, d), k / v (b, sk, hk, d), o (b, sq, h, d): element strides given per tensor as {token, head, batch}, the
// head dim is contiguous.  d: multiple of 16, at most 128; every stride a multiple of 8, pointers 16-byte aligned.
// lse (b, h, sq) fp32 or NULL.  mask_bits, mask_cls: a dense mask as bmt_attn_mask_pack wrote it, or NULL; kv_lens: (b) int32
// or NULL.
extern "C" int bmt_flash_attn_fwd(int64_t batch, int64_t sq, int64_t sk, int h, int hk, int d, const void* q, const int64_t* q_strides,
                                  const void* k, const int64_t* k_strides, const void* v, const int64_t* v_strides, void* o,
                                  const int64_t* o_strides, void* lse, float scale, int causal, const void* mask_bits,
                                  const void* mask_cls, const void* kv_lens, int dtype, void* stream) {
    if (d <= 0 || d > 128 || (d & 15) || h % hk || batch <= 0 || sq <= 0 || sk <= 0) return -1;
    if (((uintptr_t)o & 15) || (o_strides[0] & 7) || (o_strides[1] & 7) || (o_strides[2] & 7)) return -2;
    const int hd = d <= 64 ? 64 : 128;
    CUtensorMap tq, tk, tv;
    int rc;
    if ((rc = bmt_tma_map_4d(&tq, q, dtype, d, sq, q_strides[0], h, q_strides[1], batch, q_strides[2], 64, TILE)) != 0) return rc;
    if ((rc = bmt_tma_map_4d(&tk, k, dtype, d, sk, k_strides[0], hk, k_strides[1], batch, k_strides[2], 64, TILE)) != 0) return rc;
    if ((rc = bmt_tma_map_4d(&tv, v, dtype, d, sk, v_strides[0], hk, v_strides[1], batch, v_strides[2], 64, TILE)) != 0) return rc;
    AttnParams p;
    memset(&p, 0, sizeof(p));
    p.sq = sq; p.sk = sk; p.h = h; p.hk = hk; p.d = d;
    p.sl2 = scale * 1.4426950408889634f;
    p.causal = causal; p.causal_off = sk - sq;
    p.bits = (const uint32_t*)mask_bits; p.cls = (const uint8_t*)mask_cls; p.kv_lens = (const int32_t*)kv_lens;
    p.q_tiles = (int)((sq + TILE - 1) / TILE); p.k_tiles = (int)((sk + TILE - 1) / TILE);
    p.o = o; p.o_tok = o_strides[0]; p.o_head = o_strides[1]; p.o_batch = o_strides[2];
    p.lse = (float*)lse;
    const uint32_t fmt = dtype == BMT_DT_F16 ? 0u : 1u;
    const uint32_t common = (1u << 4) | (fmt << 7) | (fmt << 10) | ((uint32_t)(TILE >> 4) << 24);
    p.idesc_s = common | ((uint32_t)(TILE >> 3) << 17);                       // A, B K-major; N = 128 keys
    p.idesc_pv = common | (1u << 16) | ((uint32_t)(d >> 3) << 17);            // B (V) MN-major; N = head dim
    cudaStream_t st = (cudaStream_t)stream;
    if (dtype == BMT_DT_F16) return hd == 64 ? launch_fwd<64, __half>(tq, tk, tv, p, batch, st) : launch_fwd<128, __half>(tq, tk, tv, p, batch, st);
    if (dtype == BMT_DT_BF16) return hd == 64 ? launch_fwd<64, __nv_bfloat16>(tq, tk, tv, p, batch, st) : launch_fwd<128, __nv_bfloat16>(tq, tk, tv, p, batch, st);
    return -3;
}

// Bytes of a packed mask, and where its three parts start: bits at 0, bits_t and cls at the returned offsets.
extern "C" int64_t bmt_attn_mask_layout(int64_t batch, int64_t sq, int64_t sk, int64_t* bits_t_off, int64_t* cls_off) {
    const int64_t qt = (sq + TILE - 1) / TILE, kt = (sk + TILE - 1) / TILE;
    const int64_t t_off = batch * sq * kt * 16, c_off = t_off + batch * sk * qt * 16;
    if (bits_t_off) *bits_t_off = t_off;
    if (cls_off) *cls_off = c_off;
    return c_off + batch * qt * kt;
}

// Packs a dense mask (batch, sq, sk) of bytes (non-zero = attend) for the attention kernels; `packed` is 16-byte aligned and
// has the size that bmt_attn_mask_layout gives.
extern "C" int bmt_attn_mask_pack(int64_t batch, int64_t sq, int64_t sk, const void* mask, void* packed, void* stream) {
    if (batch <= 0 || sq <= 0 || sk <= 0 || ((uintptr_t)packed & 15)) return -1;
    const int64_t qt = (sq + TILE - 1) / TILE, kt = (sk + TILE - 1) / TILE;
    if (qt > 65535 || batch > 65535) return -2;
    int64_t t_off, c_off;
    bmt_attn_mask_layout(batch, sq, sk, &t_off, &c_off);
    bmt::launch(attn_mask_pack_kernel, dim3((unsigned)kt, (unsigned)qt, (unsigned)batch), MASK_THREADS, 0, (cudaStream_t)stream, 1, 
        (const uint8_t*)mask, sq, sk, (uint32_t*)packed, (uint32_t*)((char*)packed + t_off), (uint8_t*)packed + c_off);
    bmt_count_launch(1);
    return cudaGetLastError() == cudaSuccess ? 0 : -31;
}

// status of the attention kernels: 0, or (wait code << 16 | CTA) of the first CTA that gave up; reading clears it
extern "C" int bmt_attn_status(void) {
    int v = 0, zero = 0;
    if (cudaMemcpyFromSymbol(&v, g_attn_status, sizeof(int)) != cudaSuccess) return -1;
    if (v != 0) cudaMemcpyToSymbol(g_attn_status, &zero, sizeof(int));
    return v;
}

// Floats of dkv_part that the backward takes for this problem; 0: none needed.
extern "C" int64_t bmt_flash_attn_bwd_parts(int64_t batch, int64_t sk, int h, int hk, int d) {
    const int splits = bwd_splits(batch, sk, h, hk);
    return splits > 1 ? (int64_t)splits * 2 * batch * sk * hk * d : 0;
}

// Backward of bmt_flash_attn_fwd.  o / lse are the forward's results, dout the gradient of o; dq, dk, dv receive the
// gradients (strided like their operands).  dq_acc: scratch of batch * sq * h * d floats, delta: batch * h * sq floats,
// dkv_part: bmt_flash_attn_bwd_parts floats, or NULL (the query heads of a kv head then share one CTA).
// All tensors follow the forward's stride and alignment rules.
extern "C" int bmt_flash_attn_bwd(int64_t batch, int64_t sq, int64_t sk, int h, int hk, int d, const void* q, const int64_t* q_strides,
                                  const void* k, const int64_t* k_strides, const void* v, const int64_t* v_strides, const void* o,
                                  const int64_t* o_strides, const void* dout, const int64_t* do_strides, const void* lse, void* dq,
                                  const int64_t* dq_strides, void* dk, const int64_t* dk_strides, void* dv, const int64_t* dv_strides,
                                  void* dq_acc, void* delta, float scale, int causal, const void* mask_bits_t,
                                  const void* mask_cls, const void* kv_lens, void* dkv_part, int dtype, void* stream) {
    if (d <= 0 || d > 128 || (d & 15) || h % hk || batch <= 0 || sq <= 0 || sk <= 0) return -1;
    const int64_t* all[] = {o_strides, dq_strides, dk_strides, dv_strides};
    for (const int64_t* s3 : all)
        if ((s3[0] & 7) || (s3[1] & 7) || (s3[2] & 7)) return -2;
    if (((uintptr_t)o | (uintptr_t)dq | (uintptr_t)dk | (uintptr_t)dv | (uintptr_t)dq_acc | (uintptr_t)dkv_part) & 15) return -2;
    cudaStream_t st = (cudaStream_t)stream;
    if (dtype == BMT_DT_F16)
        return run_bwd<__half>(batch, sq, sk, h, hk, d, q, q_strides, k, k_strides, v, v_strides, o, o_strides, dout, do_strides, lse, dq,
                               dq_strides, dk, dk_strides, dv, dv_strides, dq_acc, delta, scale, causal, mask_bits_t, mask_cls, kv_lens, dkv_part, dtype, st);
    if (dtype == BMT_DT_BF16)
        return run_bwd<__nv_bfloat16>(batch, sq, sk, h, hk, d, q, q_strides, k, k_strides, v, v_strides, o, o_strides, dout, do_strides, lse,
                                      dq, dq_strides, dk, dk_strides, dv, dv_strides, dq_acc, delta, scale, causal, mask_bits_t, mask_cls, kv_lens, dkv_part, dtype, st);
    return -3;
}
