// Persistent tcgen05 GEMM for sm_100a (B200).
//
//   C[b][M,N] (+)= alpha * op(A[b]) * op(B[b]) (+ bias[N]) , optional ReLU / GELU
//
// * fp16 / bf16 operands, fp32 accumulation in tensor memory (TMEM), output fp16 / bf16 / fp32.
// * Each operand may be "K-major" (reduction dim contiguous) or "MN-major" (output dim contiguous), so
//   forward (NT), dgrad (NN) and wgrad (TN) of a linear layer all run here without any transpose pass.
// * One CTA per SM, static persistent tile loop.  Warp roles:
//       warp 0      TMA producer  (cp.async.bulk.tensor, 128-byte swizzle, S-stage mbarrier pipeline)
//       warp 1      MMA issuer    (tcgen05.mma cta_group::1 kind::f16, 128 x BN x 16, one elected thread)
//       warps 2..9  epilogue      (tcgen05.ld 32x32b -> shared memory -> alpha/bias/activation -> global)
//   Two TMEM accumulator buffers let the epilogue of tile i overlap the main loop of tile i+1.
// * BN (16..256) is picked per problem to minimise wave quantisation on 148 SMs.
// * Every wait on an mbarrier is bounded (about two seconds of polling); on expiry the kernel records a code in a
//   device status word, lets in-flight copies land, frees its TMEM and returns.  Nothing traps.
// * No TMA multicast is used anywhere (every CTA loads its own tiles).
//
// The reference has no GEMM kernel: all matmuls go through cuBLAS (bmtrain/nn/linear.py:10-24).
#include <cuda.h>
#include <atomic>
#include <mutex>
#include <unordered_map>
#include <vector>
#include <stdio.h>
#include <string.h>

#include "api.h"
#include "common.cuh"
#include "tcgen05.cuh"

namespace {

using namespace bmt_tc;

constexpr int BM = 128;
constexpr int BK = 64;          // 64 halves = 128 bytes = one swizzle row
constexpr int UMMA_K = 16;
constexpr int NUM_THREADS = 192;                      // GEMM -> reduce-scatter kernel: producer, MMA issuer, 4 epilogue warps
constexpr int epilogue_warps(int fused) { return fused == 1 ? 4 : 8; }
constexpr int num_threads(int fused) { return 64 + 32 * epilogue_warps(fused); }
constexpr int MAX_STAGES = 8;
constexpr uint32_t SMEM_MAX = 227 * 1024;     // dynamic shared memory a CTA can ask for
constexpr uint32_t SMEM_FIXED = 3 * 1024;     // header, alignment slack, small static arrays of the fused kernels

__device__ int g_gemm_status = 0;  // 0 = fine; otherwise (code << 16) | blockIdx of the first CTA that gave up
// Timing of the fused compute+collective kernels since the last read (nanoseconds of %globaltimer):
// [0] sum over the compute CTAs of the time their producer spent waiting for remote data, [1] longest pusher CTA,
// [2] longest CTA of any kind (main phase), [3] longest producer wait of one CTA, [4] kernels counted,
// [5] GEMM -> reduce-scatter: longest wait for the other ranks' deliveries, [6] longest CTA including its reduce phase,
// [7] sum over CTAs of that wait.
__device__ unsigned long long g_fused_stats[8] = {0, 0, 0, 0, 0, 0, 0, 0};

struct GemmParams {
    int64_t M, N, K;
    int bn;           // tile N
    int stages;
    uint32_t hdr_off;      // byte offset of the barrier header behind the tile stages (pusher CTAs need room for their ring)
    uint32_t out_stage_off;  // byte offset of the epilogue's buffers: 4 KiB per warp, or 128 rows x OUT_PITCH when rows go out as bulk copies
    int a_mn, b_mn;   // 1 = MN-major operand
    int a_mn5, b_mn5; // the MN-major operand's tensor map has the 64-element chunks as a dimension of their own: one copy per
                      // stage brings all chunks of the tile (instead of one copy per chunk)
    int m_blocks, n_blocks;
    int64_t batch_inner, batch_outer, b_inner_div;
    void* c;
    int64_t ldc, c_bs0, c_bs1;
    int c_dtype;
    const void* bias;
    int bias_dtype;
    int act;
    int accumulate;
    int epi;          // form of the epilogue: EXTRA of epilogue_rows, or -1: epilogue_rows_any
    float alpha;
    uint32_t idesc;
    const void* residual;  // optional (M x N, operand dtype, row pitch ldr): added after bias / activation
    int64_t ldr;
    int round_first;       // the product is rounded to C's type before the residual is added, as two operators do it
    const void* aux;       // optional (M x N, operand dtype, row pitch ld_aux) for the multiplicative epilogues
    int64_t ld_aux;
    int aux_mode;          // 0 none, 1: out *= (aux > 0)  (ReLU backward), 2: out *= gelu'(aux)
    int group_m;           // tile raster: consecutive tiles walk down `group_m` row blocks before moving to the next column block
    // Split tiles: the first `sk_tiles` tiles of the raster are cut along K over the first `sk_workers` CTAs (or CTA pairs), see Work.
    int sk_tiles, sk_workers, sk_snap;
    uint32_t sk_tag;       // what a flag holds when the partial sums behind it are complete (another one for each launch)
    uint32_t* sk_flags;    // SK_WARPS words per CTA, zero between launches
    float4* sk_part;       // sk_slot 16-byte units per CTA
    uint32_t sk_slot;
    int* host_status;      // pinned host memory, see gave_up
};

// A bounded wait has run out: what the CTA was to compute is missing.  Plain GEMMs report to the host as well, where the next launch finds it
// without waiting for the device (fused ones have a status of their own, and their callers decide).
template <bool FUSED> __device__ __forceinline__ void gave_up(int what, int* host_status) {
    const int code = (what << 16) | (int)(blockIdx.x & 0xffff);
    atomicCAS(&g_gemm_status, 0, code);
    if (!FUSED) {
        *reinterpret_cast<volatile int*>(host_status) = code;
        __threadfence_system();
    }
}

template <typename T> __device__ __forceinline__ void store8(T* dst, const float* v) {
    bmt::Vec16<T> o;
#pragma unroll
    for (int i = 0; i < 8; ++i) o.v[i] = bmt::Cvt<T>::from_f(v[i]);
    bmt::st16(dst, o);
}
template <typename T> __device__ __forceinline__ void load8(const T* src, float* v) {
    bmt::Vec16<T> o = bmt::ld16(src);
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = bmt::Cvt<T>::to_f(o.v[i]);
}

// Sum of `world` inbox slots (+ bias) for the vectors [v0, v0 + U * stride) step stride: all U * world loads are issued
// before the first add so that enough bytes are in flight to stream from HBM.
template <typename T, int U, int WMAX>
__device__ __forceinline__ void rs_reduce_vectors(const T* inbox, int64_t slot_elems, int world, const T* bias, int64_t N, T* out,
                                                  int64_t v0, int64_t stride, int64_t nvec) {
    bmt::Vec16<T> t[U][WMAX];
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const int64_t v = v0 + u * stride;
        if (v < nvec) {
#pragma unroll
            for (int j = 0; j < WMAX; ++j)
                if (j < world) t[u][j] = bmt::ld16(inbox + j * slot_elems + v * 8);
        }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const int64_t v = v0 + u * stride;
        if (v >= nvec) continue;
        float acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll
        for (int j = 0; j < WMAX; ++j)
            if (j < world) {
#pragma unroll
                for (int i = 0; i < 8; ++i) acc[i] += bmt::Cvt<T>::to_f(t[u][j].v[i]);
            }
        if (bias) {
            float b[8];
            load8(bias + (v * 8) % N, b);
#pragma unroll
            for (int i = 0; i < 8; ++i) acc[i] += b[i];
        }
        store8(out + v * 8, acc);
    }
}

template <typename T>
__device__ __forceinline__ void rs_reduce_all(const void* inbox, int64_t slot_elems, int world, const void* bias, int64_t N, void* out,
                                              int64_t nvec) {
    const int64_t stride = (int64_t)gridDim.x * NUM_THREADS;
    const int64_t first = (int64_t)blockIdx.x * NUM_THREADS + threadIdx.x;
    if (world <= 2) {
        for (int64_t v = first; v < nvec; v += stride * 8)
            rs_reduce_vectors<T, 8, 2>((const T*)inbox, slot_elems, world, (const T*)bias, N, (T*)out, v, stride, nvec);
    } else if (world <= 4) {
        for (int64_t v = first; v < nvec; v += stride * 4)
            rs_reduce_vectors<T, 4, 4>((const T*)inbox, slot_elems, world, (const T*)bias, N, (T*)out, v, stride, nvec);
    } else {
        for (int64_t v = first; v < nvec; v += stride * 2)
            rs_reduce_vectors<T, 2, 8>((const T*)inbox, slot_elems, world, (const T*)bias, N, (T*)out, v, stride, nvec);
    }
}

// Grouped raster: the CTAs that run at the same time cover a compact (group_m x ~#SM/group_m) patch of output tiles, so
// every k-slice of A and B that one of them pulls from DRAM is found in L2 by the others.
__device__ __forceinline__ void tile_coords(const GemmParams& p, int rem, int& m_blk, int& n_blk) {
    const int per_group = p.group_m * p.n_blocks;
    const int group = rem / per_group, in_group = rem - group * per_group;
    const int first_m = group * p.group_m;
    const int rows = p.m_blocks - first_m < p.group_m ? p.m_blocks - first_m : p.group_m;
    n_blk = in_group / rows;
    m_blk = first_m + in_group - n_blk * rows;
}

struct SharedHeader {
    uint64_t full[MAX_STAGES];
    uint64_t empty[MAX_STAGES];
    uint64_t tmem_full[2];
    uint64_t tmem_empty[2];
    uint32_t tmem_base;
    int failed;
};

// Eight consecutive elements of a row (the first `n` of them exist) as floats; one 16-byte load when `vec`.
template <typename T> __device__ __forceinline__ void load_row8(const T* src, int n, bool vec, float (&v)[8]) {
    if (vec && n >= 8) {
        load8(src, v);
    } else {
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] = i < n ? bmt::Cvt<T>::to_f(src[i]) : 0.f;
    }
}
__device__ __forceinline__ void load_row8_dt(const void* src, int dtype, int64_t idx, int n, bool vec, float (&v)[8]) {
    if (dtype == BMT_DT_F16) load_row8((const __half*)src + idx, n, vec, v);
    else if (dtype == BMT_DT_BF16) load_row8((const __nv_bfloat16*)src + idx, n, vec, v);
    else load_row8((const float*)src + idx, n, false, v);
}
template <typename T> __device__ __forceinline__ void unpack8(const uint4& q, float (&v)[8]) {
    bmt::Vec16<T> o;
    *reinterpret_cast<uint4*>(&o) = q;
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = bmt::Cvt<T>::to_f(o.v[i]);
}
__device__ __forceinline__ uint4 ld_global_16(const void* p) { return *reinterpret_cast<const uint4*>(p); }

// ---- split tiles --------------------------------------------------------------------------------------------------------
// Whole tiles leave SMs idle when their number is not a multiple of the CTAs: outputs of 1024 x 2560 are 40 tiles of 256 x 256 for 74
// pairs, and smaller tiles pay in bytes from L2 per multiplication.  So the tiles of the last, partial wave (and of the wave before, when
// there is one) are laid end to end along K and cut into equal ranges, one per CTA (pair).  After its whole tiles a CTA works on the
// part of its range that ends inside a tile and leaves the fp32 accumulators in its slot of the scratch; last, the CTA whose range
// holds the end of a tile adds the slots of the others to its own accumulators, in a fixed order, and stores the tile.  It waits only
// for CTAs with a lower index, which have been given an SM before it and wait for nobody before they deliver.
constexpr int SK_WARPS = 8;
struct Item { int tile, kb0, kb1, kind; };        // kind: 0 whole tile, 1 leaves partial sums, 2 adds the others' and stores
struct Work {
    int begin, end, k_blocks, phase, whole, whole_end, tile, step, tiles;
    __host__ __device__ __forceinline__ static int bound(const GemmParams& p, int worker, int k_blocks) {
        const int total = p.sk_tiles * k_blocks;
        if (worker >= p.sk_workers) return total;
        int at = (int)((int64_t)worker * total / p.sk_workers);
        const int in = at % k_blocks;             // no slivers of a tile
        if (in < p.sk_snap) at -= in;
        else if (k_blocks - in < p.sk_snap) at += k_blocks - in;
        return at;
    }
    // First of the workers whose ranges reach into the tile that `worker` finishes; it and those up to worker - 1 leave sums of it.
    __host__ __device__ __forceinline__ static int first_of(const GemmParams& p, int worker, int tile, int k_blocks) {
        int low = worker - 1;
        while (low > 0 && bound(p, low, k_blocks) > tile * k_blocks) --low;
        return low;
    }
    // `worker` takes the whole tiles sk_tiles + worker, + step, ... and the range [bound(worker), bound(worker + 1)) of the split ones
    __host__ __device__ __forceinline__ Work(const GemmParams& p, int worker, int step_, int tiles_, int k_blocks_, bool split)
        : begin(0), end(0), k_blocks(k_blocks_), phase(3), whole(0), whole_end(0), tile(worker), step(step_), tiles(tiles_) {
        if (!split) return;
        tile += p.sk_tiles;
        if (worker >= p.sk_workers) return;
        begin = bound(p, worker, k_blocks);
        end = bound(p, worker + 1, k_blocks);
        whole = (begin + k_blocks - 1) / k_blocks;
        whole_end = end / k_blocks;
        phase = begin < end ? 1 : 3;
    }
    __host__ __device__ __forceinline__ bool next(Item& it) {
        if (tile < tiles) {
            it = Item{tile, 0, k_blocks, 0};
            tile += step;
            return true;
        }
        if (whole < whole_end) { it = Item{whole++, 0, k_blocks, 0}; return true; }
        if (phase == 1) {
            phase = 2;
            const int t = end / k_blocks, at = t * k_blocks;
            if (end > at) { it = Item{t, (begin > at ? begin : at) - at, end - at, 1}; return true; }
        }
        if (phase == 2) {
            phase = 3;
            const int t = begin / k_blocks, in = begin - t * k_blocks;
            if (in && (t + 1) * k_blocks <= end) { it = Item{t, in, k_blocks, 2}; return true; }
        }
        return false;
    }
};

// The next item of a whole warp, in a form that tells the compiler that it is the same in all lanes: the descriptors and coordinates
// that depend on it stay in uniform registers (without, a k-block of a single-CTA tile took 120 ns more).
__device__ __forceinline__ bool next_item(Work& work, Item& it) {
    const bool more = __all_sync(0xffffffffu, work.next(it)) != 0;
    if (more) {
        it.tile = __shfl_sync(0xffffffffu, it.tile, 0);
        it.kb0 = __shfl_sync(0xffffffffu, it.kb0, 0);
        it.kb1 = __shfl_sync(0xffffffffu, it.kb1, 0);
        it.kind = __shfl_sync(0xffffffffu, it.kind, 0);
    }
    return more;
}

// The slots a storing warp adds: `count` of them, from `at` down, `slot` units apart.  In a slot, piece c (32 columns) of the 32 rows of
// a quarter is 256 units of 16 bytes, unit q * 32 + r being the columns 4q .. 4q + 3 of row r: what a lane holds in registers, and 512
// consecutive bytes per access.  The tile is the CTA's last, so the pipeline's shared memory is free: the units are fetched SK_AHEAD
// pieces ahead (every lane its own, so nobody has to be waited for); read when needed, a piece took 1 us.
constexpr int SK_AHEAD = 4;
struct Partials {
    const float4* at;
    int64_t slot;
    int count;
    uint32_t ring;                    // this lane's first unit of SK_AHEAD buffers of 4 KiB
    int c, i, step, n_chunks;         // next piece to fetch
    uint32_t put, get;

    __device__ __forceinline__ void fetch() {
        if (c < n_chunks) {
            const float4* src = at - i * slot + c * 256;
#pragma unroll
            for (int q = 0; q < 8; ++q)
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(ring + put * 4096 + q * 512), "l"(src + q * 32) : "memory");
            if (++put == SK_AHEAD) put = 0;
            if (++i == count) { i = 0; c += step; }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    __device__ __forceinline__ void start(uint32_t ring_, int first, int step_, int n_chunks_) {
        ring = ring_; c = first; i = 0; step = step_; n_chunks = n_chunks_; put = get = 0;
#pragma unroll
        for (int k = 0; k < SK_AHEAD; ++k) fetch();
    }
    // r += the next piece of all slots.  count < 0: they did not all arrive, and every row gets a NaN in the first column of the piece (whole tiles of
    // them, stored here or in the epilogue, cost the kernel registers, and 2 % of its time).
    __device__ __forceinline__ void add(uint32_t (&r)[32]) {
        if (count < 0) r[0] = 0x7fffffffu;
        for (int k = 0; k < count; ++k) {
            float4 v[8];
            asm volatile("cp.async.wait_group %0;" ::"n"(SK_AHEAD - 1) : "memory");
#pragma unroll
            for (int q = 0; q < 8; ++q)
                asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v[q].x), "=f"(v[q].y), "=f"(v[q].z), "=f"(v[q].w)
                             : "r"(ring + get * 4096 + q * 512) : "memory");
            if (++get == SK_AHEAD) get = 0;
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                r[4 * q] = __float_as_uint(__uint_as_float(r[4 * q]) + v[q].x);
                r[4 * q + 1] = __float_as_uint(__uint_as_float(r[4 * q + 1]) + v[q].y);
                r[4 * q + 2] = __float_as_uint(__uint_as_float(r[4 * q + 2]) + v[q].z);
                r[4 * q + 3] = __float_as_uint(__uint_as_float(r[4 * q + 3]) + v[q].w);
            }
            fetch();
        }
    }
};

// This warp's pieces of the accumulator into the slot, then its flag.
template <typename Release>
__device__ __forceinline__ void store_partials(float4* slot, uint32_t* flag, uint32_t tag, int n_chunks, uint32_t taddr, int lane, int first,
                                               Release release) {
    if (first >= n_chunks) release();
    for (int c = first; c < n_chunks; c += 2) {
        uint32_t r[32];
        tmem_ld32(taddr + c * 32, r);
        tmem_ld_wait();
        if (c + 2 >= n_chunks) release();
#pragma unroll
        for (int q = 0; q < 8; ++q)
            __stcg(slot + c * 256 + q * 32, make_float4(__uint_as_float(r[4 * q]), __uint_as_float(r[4 * q + 1]),
                                                          __uint_as_float(r[4 * q + 2]), __uint_as_float(r[4 * q + 3])));
    }
    __syncwarp();       // the release of lane 0 covers what the others have stored
    if (lane == 0) asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(flag), "r"(tag) : "memory");
}

// Bounded wait for the same warp of `count` other CTAs; takes the flags back.
__device__ __forceinline__ bool wait_partials(uint32_t* flag, int64_t pitch, int count, uint32_t tag, int lane) {
    bool ok = true;
    if (lane == 0)
        for (int i = 0; i < count && ok; ++i, flag -= pitch) {
            uint64_t t0 = 0;
            for (uint32_t spin = 0;; ++spin) {
                uint32_t v;
                asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(flag) : "memory");
                if (v == tag) break;
                if ((spin & 255u) == 255u) {
                    const uint64_t now = global_ns();
                    if (t0 == 0) t0 = now;
                    else if (now - t0 > 2000000000ull) { ok = false; break; }
                }
            }
            asm volatile("st.relaxed.gpu.global.u32 [%0], 0;" ::"l"(flag) : "memory");
        }
    ok = __all_sync(0xffffffffu, ok) != 0;
    __syncwarp();       // what lane 0 has acquired is there for the others
    return ok;
}

// Epilogue of one warp's 32 rows of a tile: tensor memory -> (alpha, bias, activation, mask, residual, old C) -> global.
// tcgen05.ld hands every thread one row; written out that way, a store instruction touches 32 rows with 16 bytes each, which
// cost 5.5 to 8 us per 128 x 256 tile and made every weight gradient of a 1024-token block epilogue-bound (2560 x 8192 x 1024:
// 52.8 us, of which 16 us without the stores).  So 32 columns at a time go through a 4 KiB exchange buffer of the warp
// (fp32, 16-byte units XOR-swizzled by the row: no bank conflicts either way) and come back as 8 columns per thread,
// 4 threads per row: stores and the loads of residual / mask / old C move whole 32-byte sectors.  The next 32 columns are
// read from tensor memory, and the matching piece of the residual, mask or old C from global memory, while the current
// ones are worked on; `release` runs as soon as the last column has left tensor memory.  Two warps share 32 rows and take
// the pieces of 32 columns in turn (`first` = 0 or 1).
// Two warps per scheduler do this, so it is bound by their own instruction stream: the forms that the layers use are
// compiled without run-time choices (EXTRA: 0 none, 1 add a 16-bit matrix (residual or old C), 2 / 3 ReLU / GELU gradient
// mask; bias and ReLU stay run-time, they cost a few instructions), everything else takes epilogue_rows_any.
constexpr uint32_t EPI_BYTES_PER_WARP = 32 * 128;

__device__ __forceinline__ void epi_put(uint32_t sbuf, int lane, const uint32_t (&r)[32]) {
    const uint32_t srow = sbuf + (uint32_t)lane * 128;
#pragma unroll
    for (int q = 0; q < 8; ++q)
        asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(srow + (uint32_t)((q ^ (lane & 7)) << 4)), "r"(r[4 * q]),
                     "r"(r[4 * q + 1]), "r"(r[4 * q + 2]), "r"(r[4 * q + 3]) : "memory");
}
// columns 8 * (lane & 3) .. + 7 of row `rl` of the exchange buffer
__device__ __forceinline__ void epi_get(uint32_t sbuf, int lane, int rl, float (&v)[8]) {
#pragma unroll
    for (int h = 0; h < 2; ++h)
        asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v[4 * h]), "=f"(v[4 * h + 1]), "=f"(v[4 * h + 2]), "=f"(v[4 * h + 3])
                     : "r"(sbuf + (uint32_t)(rl * 128 + ((((lane & 3) * 2 + h) ^ (rl & 7)) << 4))) : "memory");
}

template <typename T, int EXTRA, typename Release>
__device__ __forceinline__ void epilogue_rows(const GemmParams& p, T* cbase, const T* ebase, int64_t e_ld, int64_t row0, int64_t n0,
                                              int64_t col_end, uint32_t taddr, uint32_t sbuf, int lane, int first, Partials& sk,
                                              Release release) {
    const int sub = lane >> 2, cq = (lane & 3) * 8;
    const int n_cols = (int)(col_end - n0), n_chunks = (n_cols + 31) / 32;
    const int rows = (int)(p.M - row0 < 32 ? p.M - row0 : 32);     // may be <= 0: nothing is stored then
    T* dst = cbase + (row0 + sub) * p.ldc + n0 + cq;
    const T* src = EXTRA ? ebase + (row0 + sub) * e_ld + n0 + cq : nullptr;
    const T* bias = p.bias ? (const T*)p.bias + n0 + cq : nullptr;
    const int64_t d_step = 8 * p.ldc, e_step = 8 * e_ld;
    const float alpha = p.alpha;
    const bool relu = p.act == 1;
    uint4 nx[4];
    auto fetch = [&](int c) {
        const bool col_ok = c * 32 + cq < n_cols;
#pragma unroll
        for (int it = 0; it < 4; ++it) {
            nx[it] = make_uint4(0u, 0u, 0u, 0u);
            if (col_ok && it * 8 + sub < rows) nx[it] = ld_global_16(src + it * e_step + c * 32);
        }
    };
    if (first >= n_chunks) { release(); return; }
    uint32_t r[32];
    tmem_ld32(taddr + first * 32, r);
    if (EXTRA) fetch(first);
    for (int c = first; c < n_chunks; c += 2) {
        const bool col_ok = c * 32 + cq < n_cols;
        float b[8] = {0, 0, 0, 0, 0, 0, 0, 0};
        if (bias && col_ok) load8(bias + c * 32, b);
        tmem_ld_wait();
        if (sk.count) sk.add(r);
        epi_put(sbuf, lane, r);
        if (c + 2 < n_chunks) tmem_ld32(taddr + (c + 2) * 32, r);
        else release();
        uint4 cur[4];
        if (EXTRA) {
#pragma unroll
            for (int it = 0; it < 4; ++it) cur[it] = nx[it];
            if (c + 2 < n_chunks) fetch(c + 2);
        }
        __syncwarp();
        float v[4][8];
#pragma unroll
        for (int it = 0; it < 4; ++it) epi_get(sbuf, lane, it * 8 + sub, v[it]);
        __syncwarp();    // the buffer has been read by all lanes
#pragma unroll
        for (int it = 0; it < 4; ++it) {
#pragma unroll
            for (int i = 0; i < 8; ++i) v[it][i] = v[it][i] * alpha + b[i];
            if (relu) {      // a branch, not a floor of -inf: fmaxf(NaN, -inf) is -inf
#pragma unroll
                for (int i = 0; i < 8; ++i) v[it][i] = fmaxf(v[it][i], 0.f);
            }
            if (EXTRA) {
                float e[8];
                unpack8<T>(cur[it], e);
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    if (EXTRA == 1) v[it][i] = (p.round_first ? bmt::Cvt<T>::to_f(bmt::Cvt<T>::from_f(v[it][i])) : v[it][i]) + e[i];
                    else if (EXTRA == 2) v[it][i] = e[i] > 0.f ? v[it][i] : 0.f;
                    else v[it][i] *= bmt::gelu_grad(e[i]);
                }
            }
            if (col_ok && it * 8 + sub < rows) store8(dst + it * d_step + c * 32, v[it]);
        }
    }
}

// All other forms: fp32 output, odd pitches and widths, unaligned pointers, GELU, several extras at once.
template <typename TC, typename Release>
__device__ __forceinline__ void epilogue_rows_any(const GemmParams& p, TC* cbase, int64_t row0, int64_t n0, int64_t col_end, uint32_t taddr,
                                               uint32_t sbuf, int lane, int first, Partials& sk, Release release) {
    const int sub = lane >> 2, cq = (lane & 3) * 8;
    const int n_chunks = (int)((col_end - n0 + 31) / 32);
    const bool c_vec = sizeof(TC) == 2 ? ((p.ldc & 7) == 0 && (((uintptr_t)cbase) & 15) == 0)
                                       : ((p.ldc & 3) == 0 && (((uintptr_t)cbase) & 15) == 0);
    const bool b_vec = (((uintptr_t)p.bias) & 15) == 0, r_vec = (p.ldr & 7) == 0 && (((uintptr_t)p.residual) & 15) == 0;
    const bool a_vec = (p.ld_aux & 7) == 0 && (((uintptr_t)p.aux) & 15) == 0;
    if (first >= n_chunks) { release(); return; }
    for (int c = first; c < n_chunks; c += 2) {
        uint32_t r[32];
        tmem_ld32(taddr + c * 32, r);
        tmem_ld_wait();
        if (sk.count) sk.add(r);
        epi_put(sbuf, lane, r);
        if (c + 2 >= n_chunks) release();
        __syncwarp();
        const int64_t col = n0 + c * 32 + cq;
        const int n_ok = col_end - col >= 8 ? 8 : (int)(col_end - col);       // columns of this thread that exist (may be <= 0)
        float bias[8] = {0, 0, 0, 0, 0, 0, 0, 0};
        if (p.bias && n_ok > 0) load_row8_dt(p.bias, p.bias_dtype, col, n_ok, b_vec, bias);
        for (int it = 0; it < 4; ++it) {
            const int64_t row = row0 + it * 8 + sub;
            if (row >= p.M || n_ok <= 0) continue;
            float v[8], e[8];
            epi_get(sbuf, lane, it * 8 + sub, v);
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                v[i] = v[i] * p.alpha + bias[i];
                if (p.act == 1) v[i] = fmaxf(v[i], 0.f);
                else if (p.act == 2) v[i] = bmt::gelu(v[i]);
            }
            if (p.aux_mode) {
                load_row8_dt(p.aux, p.bias_dtype, row * p.ld_aux + col, n_ok, a_vec, e);
#pragma unroll
                for (int i = 0; i < 8; ++i) v[i] = p.aux_mode == 1 ? (e[i] > 0.f ? v[i] : 0.f) : v[i] * bmt::gelu_grad(e[i]);
            }
            if (p.residual) {
                load_row8_dt(p.residual, p.bias_dtype, row * p.ldr + col, n_ok, r_vec, e);
#pragma unroll
                for (int i = 0; i < 8; ++i) v[i] = (p.round_first ? bmt::Cvt<TC>::to_f(bmt::Cvt<TC>::from_f(v[i])) : v[i]) + e[i];
            }
            TC* dst = cbase + row * p.ldc + col;
            if (p.accumulate) {
                if constexpr (sizeof(TC) == 2) {
                    load_row8(dst, n_ok, c_vec, e);
                } else {
#pragma unroll
                    for (int i = 0; i < 8; ++i) e[i] = i < n_ok ? dst[i] : 0.f;
                }
#pragma unroll
                for (int i = 0; i < 8; ++i) v[i] += e[i];
            }
            if (n_ok == 8 && c_vec) {
                if constexpr (sizeof(TC) == 2) {
                    store8(dst, v);
                } else {
                    reinterpret_cast<float4*>(dst)[0] = make_float4(v[0], v[1], v[2], v[3]);
                    reinterpret_cast<float4*>(dst)[1] = make_float4(v[4], v[5], v[6], v[7]);
                }
            } else {
#pragma unroll
                for (int i = 0; i < 8; ++i)
                    if (i < n_ok) dst[i] = bmt::Cvt<TC>::from_f(v[i]);
            }
        }
        __syncwarp();    // the buffer has been read by all lanes
    }
}

// Picks the form of the epilogue for a 16-bit output tile; `p.epi` is what launch_gemm found for the whole problem.
template <typename T, typename Release>
__device__ __forceinline__ void epilogue_tile(const GemmParams& p, T* cbase, int64_t row0, int64_t n0, int64_t col_end, uint32_t taddr,
                                              uint32_t sbuf, int lane, int first, Partials& sk, Release release) {
    if (p.epi == 0) epilogue_rows<T, 0>(p, cbase, nullptr, 0, row0, n0, col_end, taddr, sbuf, lane, first, sk, release);
    else if (p.epi == 1)
        epilogue_rows<T, 1>(p, cbase, p.accumulate ? cbase : (const T*)p.residual, p.accumulate ? p.ldc : p.ldr, row0, n0, col_end, taddr,
                            sbuf, lane, first, sk, release);
    else if (p.epi == 2) epilogue_rows<T, 2>(p, cbase, (const T*)p.aux, p.ld_aux, row0, n0, col_end, taddr, sbuf, lane, first, sk, release);
    else if (p.epi == 3) epilogue_rows<T, 3>(p, cbase, (const T*)p.aux, p.ld_aux, row0, n0, col_end, taddr, sbuf, lane, first, sk, release);
    else epilogue_rows_any(p, cbase, row0, n0, col_end, taddr, sbuf, lane, first, sk, release);
}

// ---- two-CTA (cta_group::2) helpers: the pair shares one 256 x BN accumulator tile, each CTA feeds its own
// 128 rows of A and its own half of the B tile, the leader CTA (rank 0) issues the MMAs for both.
__device__ __forceinline__ uint32_t cluster_ctarank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ uint32_t map_to_cta(uint32_t local_smem_addr, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(local_smem_addr), "r"(rank));
    return r;
}
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// Relaxed: what has to come before it is the warp's reading of tensor memory, which tcgen05.wait::ld and the fence have completed.  A
// release would also wait for the warp's stores to global memory, about 1000 clocks.
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
    asm volatile("mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
__device__ __forceinline__ void tmem_alloc_2cta(uint32_t* dst_smem, uint32_t ncols) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(dst_smem)), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tmem_relinquish_2cta() { asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_dealloc_2cta(uint32_t taddr, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void umma_f16_2cta(uint32_t tmem_c, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(tmem_c), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}
// arrives on the barrier at the same shared-memory offset in both CTAs of the pair
__device__ __forceinline__ void umma_commit_2cta(uint64_t* bar) {
    const uint16_t mask = 3;
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
                 ::"r"(smem_u32(bar)), "h"(mask) : "memory");
}

// ---- fused collectives over peer memory (NVLink) ----------------------------------------------------------------
// mode 1, GEMM -> reduce-scatter: the epilogue stores every output row straight into the inbox of the rank that owns
//         the row (own rank: local memory, other ranks: P2P stores).  When all CTAs of this rank are done, the last one
//         publishes "rank r delivered" to every peer; each CTA then waits (bounded) for all ranks and sums the inbox
//         slots of its share of the local rows (+ bias) into the output.
// mode 2, all-gather -> GEMM: the first `ag_ctas` CTAs do no math; they push this rank's rows of A into the gathered
//         buffer of every rank (own first) in pieces and bump a per-128-row-block counter on the destination.  The
//         TMA producers of the compute CTAs visit local row blocks first and wait (bounded) on the counter of a block
//         before loading it, so the transfer overlaps the math block by block.
// Flags: `flags[j]` is rank j's flag array, row `x` of it has one counter per rank.  free_row: "my inbox / gathered
// buffer may be overwritten for this epoch" (published at kernel start); done_row: "my contributions are delivered".
struct FusedComm {
    int mode;                 // 0 none, 1 GEMM -> reduce-scatter, 2 all-gather -> GEMM
    int world, rank;
    unsigned int* flags[8];
    int free_row, done_row;
    unsigned int epoch;
    int* status;
    uint64_t limit_ns;
    // mode 1
    void* rs_inbox[8];        // destination j: base of slot `rank` inside j's inbox (rs_rows x N, pitch N)
    const void* rs_inbox_local;  // this rank's inbox: world slots of rs_rows x N
    int64_t rs_rows;          // rows per rank
    unsigned int* rs_counter; // local, monotonic: [0] epilogue warps that finished the tiles with rows of other ranks (early
                              // mode) or CTAs that finished all tiles; [1] early mode: CTAs that finished all tiles
    int rs_split;             // the kernel ends after publishing "delivered": waiting for the other ranks and summing the inbox
                              // are left to later launches (a one-CTA wait kernel and rs_reduce_kernel), so that no CTA of this
                              // grid holds an SM while it waits for another rank or for the rest of its own grid
    int rs_early;             // tiles with other ranks' rows come first and "delivered" is published when they are done
    int rs_bpr;               // early mode: tile rows per rank
    int64_t rs_remote_tiles;  // early mode: number of tiles (in raster order) that hold rows of other ranks
    void* rs_out;             // rs_rows x N
    const void* rs_bias;
    // mode 2
    int skip_local;           // modes 2/3: this rank's own part is already in its gathered buffer (copied before the launch)
    int ag_ctas;
    const void* ag_src;       // this rank's rows (ag_rows x K, pitch ag_ld_src)
    int64_t ag_ld_src, ag_rows;
    void* ag_dst[8];          // every rank's gathered buffer (world * ag_rows x K, pitch K)
    unsigned int* ag_count[8];// every rank's per-row-block counters
    int ag_piece_bytes;       // bytes per pushed piece: divides the bytes of a 128-row block, at most PUSH_PIECE_BYTES
    int ag_pieces_per_block;  // pieces per 128-row block
    int ag_runs_per_block;    // a block is pushed as this many runs of consecutive pieces, each by one CTA, each ending with
                              // one bump of the block's counter on the destination (what the counter grows by per epoch)
    // mode 3 (ZeRO weight gather -> GEMM): the B operand (N x K, rows contiguous) is cut over the ranks as a flat element
    // range; every rank pushes its part to all ranks in pieces and the TMA producer waits for the 128-row chunks it needs
    const char* bg_src;       // this rank's part (local shard memory)
    int64_t bg_first, bg_count;   // flat element range [bg_first, bg_first + bg_count) of the N*K weight elements
    void* bg_dst[8];          // start of the weight inside every rank's gathered buffer
    unsigned int* bg_cnt[8];  // every rank's per-chunk counters (chunk = 128 rows)
    const unsigned int* bg_expected;  // pieces a chunk receives in total, per chunk
    int bg_first_block;       // n-block at which this rank's own rows start (tile order is rotated to begin there)
    int bg_split;             // a rank's part of one 128-row chunk is pushed as up to this many runs (one counter bump each)
};
constexpr int64_t BG_PIECE = 16384;  // elements per pushed piece (32 KiB = one stage of the push pipeline)

__device__ __forceinline__ void st_release_sys_u32(unsigned int* p, unsigned int v) {
    asm volatile("st.release.sys.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ unsigned int ld_acquire_sys_u32(const unsigned int* p) {
    unsigned int v;
    asm volatile("ld.acquire.sys.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
// Bounded poll until *p >= target (counters only grow).
__device__ __forceinline__ bool wait_counter(const unsigned int* p, unsigned int target, uint64_t limit_ns) {
    uint64_t t0 = 0;
    for (unsigned int spins = 0;; ++spins) {
        if ((int)(ld_acquire_sys_u32(p) - target) >= 0) return true;
        if ((spins & 255u) == 255u) {
            const uint64_t now = global_ns();
            if (t0 == 0) t0 = now;
            else if (now - t0 > limit_ns) return false;
        }
    }
}

// ---- push pipeline of a pusher CTA ---------------------------------------------------------------------------------
// One thread moves pieces of local global memory to a (peer or local) destination through a ring of shared-memory
// stages with bulk asynchronous copies: global -> shared completes on an mbarrier, shared -> global is tracked in bulk
// groups.  Up to PUSH_AHEAD loads and PUSH_PENDING + 1 stores are in flight at a time; a piece's counter on the
// destination is bumped only after its store has completed (full wait_group, proxy fence, system fence).
// Epilogue staging of the GEMM -> reduce-scatter kernel: every thread packs up to OUT_CHUNK columns of its row into shared
// memory and sends them with one bulk copy (256-byte writes keep NVLink packets full; 16-byte scattered stores do not).
// The 16 bytes of padding per row spread the rows of a warp over all banks.
constexpr int OUT_CHUNK = 128, OUT_PITCH = OUT_CHUNK * 2 + 16;
constexpr int PUSH_STAGES = 6, PUSH_AHEAD = 3, PUSH_PENDING = 3;
constexpr uint32_t PUSH_PIECE_BYTES = 32768;

struct PushMeta {
    char* dst[PUSH_STAGES];
    unsigned int* cnt[PUSH_STAGES];
    uint32_t bytes[PUSH_STAGES];
};

struct PushPipe {
    uint32_t buf0, bar0;     // shared addresses: first stage, first mbarrier (8 bytes apart)
    PushMeta* meta;          // in shared memory
    int64_t n_loaded, n_stored, n_sig;

    __device__ __forceinline__ void init(uint32_t buf, uint32_t bar, PushMeta* m) {
        buf0 = buf; bar0 = bar; meta = m; n_loaded = n_stored = n_sig = 0;
    }
    __device__ __forceinline__ void retire(int64_t upto) {
        bool fenced = false;
        for (; n_sig < upto; ++n_sig) {
            unsigned int* c = meta->cnt[n_sig % PUSH_STAGES];
            if (!c) continue;
            if (!fenced) {
                asm volatile("fence.proxy.async.global;" ::: "memory");  // the stores went through the async proxy
                __threadfence_system();
                fenced = true;
            }
            atomicAdd_system(c, 1u);
        }
    }
    // Issue the store of the oldest loaded piece (if any) and retire stores beyond the pending limit.
    __device__ __forceinline__ bool advance() {
        if (n_stored < n_loaded) {
            const int s = (int)(n_stored % PUSH_STAGES);
            if (!mbar_wait_u32(bar0 + 8 * s, (uint32_t)((n_stored / PUSH_STAGES) & 1))) return false;
            asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;"
                         ::"l"(meta->dst[s]), "r"(buf0 + s * PUSH_PIECE_BYTES), "r"(meta->bytes[s]) : "memory");
            asm volatile("cp.async.bulk.commit_group;" ::: "memory");
            ++n_stored;
        }
        if (n_stored - n_sig > PUSH_PENDING) {
            asm volatile("cp.async.bulk.wait_group %0;" ::"n"(PUSH_PENDING) : "memory");
            retire(n_stored - PUSH_PENDING);
        }
        return true;
    }
    // Queue one piece: bytes is a multiple of 16 and at most PUSH_PIECE_BYTES, both addresses are 16-byte aligned.
    __device__ __forceinline__ bool submit(const char* src, char* dst, unsigned int* cnt, uint32_t bytes) {
        while (n_loaded - n_sig >= PUSH_STAGES || n_loaded - n_stored >= PUSH_AHEAD) {
            if (!advance()) return false;
        }
        const int s = (int)(n_loaded % PUSH_STAGES);
        meta->dst[s] = dst; meta->cnt[s] = cnt; meta->bytes[s] = bytes;
        mbar_expect_tx_u32(bar0 + 8 * s, bytes);
        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                     ::"r"(buf0 + s * PUSH_PIECE_BYTES), "l"(src), "r"(bytes), "r"(bar0 + 8 * s) : "memory");
        ++n_loaded;
        return true;
    }
    // Store what is loaded, wait for every store, signal the rest.  On a failed load wait the stores already issued are
    // still waited for (they read this CTA's shared memory).
    __device__ __forceinline__ bool drain() {
        bool ok = true;
        while (ok && n_stored < n_loaded) ok = advance();
        asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
        retire(n_stored);
        return ok;
    }
};

template <bool CTA2, int FUSED>
__global__ void __launch_bounds__(num_threads(FUSED), 1)
gemm_tcgen05_kernel(const __grid_constant__ CUtensorMap tma_a, const __grid_constant__ CUtensorMap tma_b, const GemmParams p,
                    const FusedComm f) {
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    // tiles first (1024-byte aligned for the 128-byte swizzle), bookkeeping after them
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    constexpr int NCTA = CTA2 ? 2 : 1;
    const uint32_t rank = CTA2 ? cluster_ctarank() : 0u;          // position inside the CTA pair
    const uint32_t bn_local = (uint32_t)p.bn / NCTA;               // rows of the B tile this CTA loads
    const uint32_t a_bytes = BM * BK * 2;
    const uint32_t b_bytes = bn_local * BK * 2;
    const uint32_t stage_bytes = a_bytes + b_bytes;
    SharedHeader* hdr = (SharedHeader*)(smem + p.hdr_off);

    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
    const int k_blocks = (int)((p.K + BK - 1) / BK);
    const int tiles_per_batch = p.m_blocks * p.n_blocks;   // m_blocks counts (BM * NCTA)-row tiles
    const int num_tiles = tiles_per_batch * (int)(p.batch_inner * p.batch_outer);
    // The pusher CTAs are the first CTAs of the grid: CTAs are handed to SMs in index order, so when another kernel keeps
    // part of the GPU busy it is compute CTAs that wait for an SM, never the CTAs the other ranks depend on.
    const int comm_first = (FUSED == 2 || FUSED == 3) ? f.ag_ctas : 0;
    const int compute_ctas = (int)gridDim.x - comm_first;
    const bool comm_cta = (int)blockIdx.x < comm_first;
    const int first_tile = comm_cta ? num_tiles : ((int)blockIdx.x - comm_first) / NCTA, tile_step = compute_ctas / NCTA;
    const int blocks_per_rank = FUSED == 2 ? (int)(f.ag_rows / (BM * NCTA)) : 0;   // in tile rows (256 rows for a CTA pair)
    const int row_blocks_per_rank = FUSED == 2 ? (int)(f.ag_rows / BM) : 1;          // in 128-row blocks (counter granularity)
    const uint32_t tmem_cols = 2 * p.bn <= 32 ? 32 : 2 * p.bn <= 64 ? 64 : 2 * p.bn <= 128 ? 128 : 2 * p.bn <= 256 ? 256 : 512;

    if (threadIdx.x == 0) {
        for (int s = 0; s < MAX_STAGES; ++s) { mbar_init(&hdr->full[s], 1); mbar_init(&hdr->empty[s], 1); }
        for (int a = 0; a < 2; ++a) { mbar_init(&hdr->tmem_full[a], 1); mbar_init(&hdr->tmem_empty[a], epilogue_warps(FUSED) * NCTA); }
        hdr->failed = 0;
        fence_barrier_init();
    }
    if (warp == 1) {
        if (CTA2) { tmem_alloc_2cta(&hdr->tmem_base, tmem_cols); tmem_relinquish_2cta(); }
        else { tmem_alloc(&hdr->tmem_base, tmem_cols); tmem_relinquish(); }
    }
    tc_fence_before();
    __syncthreads();
    if (CTA2) cluster_sync();   // the peer's barriers must be initialised before anything is signalled across
    tc_fence_after();
    if (FUSED == 0) bmt::after_previous();
    const uint32_t tmem_base = hdr->tmem_base;

    const uint64_t t_kernel0 = (FUSED != 0 && threadIdx.x == 0) ? global_ns() : 0;
    if (FUSED != 0 && blockIdx.x == 0 && threadIdx.x == 0) atomicAdd(&g_fused_stats[4], 1ull);
    if (FUSED != 0 && blockIdx.x == 0 && threadIdx.x < (unsigned)f.world) {
        // everything this rank did earlier on the stream is complete: peers may write into its buffers for this epoch
        st_release_sys_u32(f.flags[threadIdx.x] + f.free_row * f.world + f.rank, f.epoch);
    }

    if (comm_cta && threadIdx.x == 0) {
        // ------------------------------------------------------------------ pusher (one thread drives bulk copies)
        __shared__ PushMeta push_meta;
        PushPipe pipe;
        pipe.init(smem_u32(smem), smem_u32(&hdr->full[0]), &push_meta);
        const int n_pushers = f.ag_ctas, me = (int)blockIdx.x;
        bool ok = true;
        unsigned int free_seen = 1u << f.rank;   // destinations whose "free for this epoch" flag has been observed
        auto dst_free = [&](int dst) -> bool {
            if (free_seen & (1u << dst)) return true;
            if (!wait_counter(f.flags[f.rank] + f.free_row * f.world + dst, f.epoch, f.limit_ns)) {
                atomicCAS(f.status, 0, (FUSED == 3 ? 0x800 : 0x300) | f.rank);
                atomicCAS(&g_gemm_status, 0, ((FUSED == 3 ? 9 : 5) << 16) | (blockIdx.x & 0xffff));
                return false;
            }
            free_seen |= 1u << dst;
            return true;
        };
        if (FUSED == 3) {
            // weight pusher: this rank's flat element range, cut at 128-row chunk boundaries, to every rank (own first)
            const int64_t CK = (int64_t)BM * p.K;                       // elements per 128-row chunk
            const int64_t lo_all = f.bg_first, hi_all = f.bg_first + f.bg_count;
            for (int di = f.skip_local ? 1 : 0; di < f.world && ok && f.bg_count > 0; ++di) {
                // own copy first, then rank-1, rank-2, ...: a rank multiplies its own rows first and continues with the
                // rows of rank+1, rank+2, ..., so it should receive from those sources in that order
                const int dst = (f.rank - di + f.world) % f.world;
                int64_t g = 0;   // running index of runs
                for (int64_t c = lo_all / CK; c * CK < hi_all && ok; ++c) {
                    const int64_t lo = lo_all > c * CK ? lo_all : c * CK;
                    const int64_t hi = hi_all < (c + 1) * CK ? hi_all : (c + 1) * CK;
                    const int64_t np = (hi - lo + BG_PIECE - 1) / BG_PIECE;           // pieces of this rank in the chunk
                    const int64_t per_run = (np + f.bg_split - 1) / f.bg_split;       // pieces per run
                    for (int64_t r0 = 0; r0 < np && ok; r0 += per_run, ++g) {
                        if (g % n_pushers != me) continue;
                        if (!dst_free(dst)) { ok = false; break; }
                        const int64_t r1 = r0 + per_run < np ? r0 + per_run : np;
                        for (int64_t pi = r0; pi < r1 && ok; ++pi) {
                            const int64_t e0 = lo + pi * BG_PIECE;
                            const uint32_t bytes = (uint32_t)((hi - e0 < BG_PIECE ? hi - e0 : BG_PIECE) * 2);
                            // only the last piece of a run carries the counter: no fence between the pieces of a run
                            ok = pipe.submit(f.bg_src + (e0 - lo_all) * 2, (char*)f.bg_dst[dst] + e0 * 2,
                                             pi + 1 == r1 ? f.bg_cnt[dst] + c : nullptr, bytes);
                        }
                    }
                }
            }
        } else {
            // all-gather pusher: this rank's rows (contiguous) to every rank's gathered matrix, destination-major
            // starting with this rank itself, then rank-1, rank-2, ... (the order in which the consumers get to them)
            const int64_t block_bytes = (int64_t)BM * p.K * 2;
            const int64_t rpb = f.ag_runs_per_block, per_run = f.ag_pieces_per_block / rpb;
            const int64_t per_dst = (int64_t)row_blocks_per_rank * rpb;
            const int skip = f.skip_local ? 1 : 0;
            const int64_t total_runs = (int64_t)(f.world - skip) * per_dst;
            for (int64_t g = me; g < total_runs && ok; g += n_pushers) {
                const int dst = (f.rank - skip - (int)(g / per_dst) + 2 * f.world) % f.world;
                const int64_t rem = g % per_dst;
                const int64_t blk = rem / rpb, run = rem % rpb;
                if (!dst_free(dst)) { ok = false; break; }
                unsigned int* cnt = f.ag_count[dst] + (f.rank * row_blocks_per_rank + blk);
                char* dbase = (char*)f.ag_dst[dst] + (int64_t)f.rank * f.ag_rows * p.K * 2;
                for (int64_t pi = run * per_run; pi < (run + 1) * per_run && ok; ++pi) {
                    const int64_t off = blk * block_bytes + pi * (int64_t)f.ag_piece_bytes;
                    // only the last piece of a run carries the counter: no fence between the pieces of a run
                    ok = pipe.submit((const char*)f.ag_src + off, dbase + off, pi + 1 == (run + 1) * per_run ? cnt : nullptr,
                                     (uint32_t)f.ag_piece_bytes);
                }
            }
        }
        if (!pipe.drain()) ok = false;
        if (!ok) {
            hdr->failed = 1;
            atomicCAS(&g_gemm_status, 0, (11 << 16) | (blockIdx.x & 0xffff));
        }
        atomicMax(&g_fused_stats[1], (unsigned long long)(global_ns() - t_kernel0));
    } else if (comm_cta) {
        // the other threads of a pusher CTA have nothing to do
    } else if (warp == 0) {
        // ------------------------------------------------------------------ TMA producer (one per CTA)
        {
            bool ok = true;
            uint64_t waited = 0;        // time spent waiting for data of other ranks (fused modes)
            uint32_t ps = 0, pph = 0;   // ring position and phase, carried across tiles
            const uint32_t smem0 = smem_u32(smem), full0 = smem_u32(&hdr->full[0]), empty0 = smem_u32(&hdr->empty[0]);
            const uint32_t full_leader0 = CTA2 ? map_to_cta(full0, 0) : full0;
            Work work(p, first_tile, tile_step, num_tiles, k_blocks, FUSED == 0 && p.sk_tiles > 0);
            for (Item it; ok && next_item(work, it);) {
                const int tile = it.tile;
                const int batch = tile / tiles_per_batch;
                const int rem = tile - batch * tiles_per_batch;
                int m_blk, n_blk;
                tile_coords(p, rem, m_blk, n_blk);
                if (FUSED == 1 && f.rs_early) m_blk = (m_blk + (f.rank + 1) * f.rs_bpr) % p.m_blocks;   // own rows last
                if (FUSED == 3) {
                    // this rank's own rows first; wait for every 128-row chunk the B tile touches
                    n_blk = (n_blk + f.bg_first_block) % p.n_blocks;
                    const int64_t r0 = (int64_t)n_blk * p.bn;
                    const int64_t r1 = (r0 + p.bn < p.N ? r0 + p.bn : p.N) - 1;
                    const uint64_t tw0 = global_ns();
                    if (lane == 0) {
                        for (int64_t c = r0 / BM; c <= r1 / BM && ok; ++c) {
                            const unsigned int target = f.epoch * f.bg_expected[c];
                            if (!wait_counter(f.bg_cnt[f.rank] + c, target, f.limit_ns)) {
                                ok = false; atomicCAS(f.status, 0, 0x900 | f.rank); atomicCAS(&g_gemm_status, 0, (10 << 16) | (blockIdx.x & 0xffff)); hdr->failed = 1;
                            }
                        }
                    }
                    ok = __all_sync(0xffffffffu, ok) != 0;   // the other lanes follow lane 0, whose loads acquired the data
                    if (!ok) break;
                    waited += global_ns() - tw0;
                    asm volatile("fence.proxy.async.global;" ::: "memory");
                }
                if (FUSED == 2) {
                    // local row blocks first, then the peers' blocks in the order in which they are pushed
                    m_blk = (m_blk + f.rank * blocks_per_rank) % p.m_blocks;
                    const unsigned int target = f.epoch * (unsigned int)f.ag_runs_per_block;
                    const int row_block = m_blk * NCTA + (int)rank;
                    const bool mine = f.skip_local && row_block / row_blocks_per_rank == f.rank;   // copied before the launch
                    const uint64_t tw0 = global_ns();
                    if (lane == 0 && !mine && !wait_counter(f.ag_count[f.rank] + row_block, target, f.limit_ns)) {
                        ok = false; atomicCAS(f.status, 0, 0x400 | f.rank); atomicCAS(&g_gemm_status, 0, (6 << 16) | (blockIdx.x & 0xffff)); hdr->failed = 1;
                    }
                    ok = __all_sync(0xffffffffu, ok) != 0;   // the other lanes follow lane 0, whose loads acquired the data
                    if (!ok) break;
                    waited += global_ns() - tw0;
                    asm volatile("fence.proxy.async.global;" ::: "memory");  // the block was written by a peer's copies, TMA reads it
                }
                const int bo = batch / (int)p.batch_inner, bi = batch - bo * (int)p.batch_inner;
                const int bib = bi / (int)p.b_inner_div;
                const int m0 = m_blk * (BM * NCTA) + (int)rank * BM;            // this CTA's rows of A
                const int n0 = n_blk * p.bn + (int)(rank * bn_local);           // this CTA's rows of the B tile
                for (int kb = it.kb0; kb < it.kb1; ++kb) {
                    if (!mbar_wait_warp(empty0 + 8 * ps, pph ^ 1)) { ok = false; if (lane == 0) { gave_up<FUSED != 0>(1, p.host_status); hdr->failed = 1; } break; }
                    const uint32_t sa = smem0 + ps * stage_bytes, sb = sa + a_bytes;
                    const int kx = kb * BK;
                    if (elect_one()) {
                        if (!CTA2) {
                            const uint32_t bar = full0 + 8 * ps;
                            mbar_expect_tx_u32(bar, stage_bytes);
                            if (!p.a_mn) {
                                tma_load_4d_u32(&tma_a, bar, sa, kx, m0, bi, bo);
                            } else if (p.a_mn5) {
                                tma_load_5d_u32(&tma_a, bar, sa, 0, kx, m0 / 64, bi, bo);
                            } else {
#pragma unroll
                                for (int c = 0; c < BM / 64; ++c) tma_load_4d_u32(&tma_a, bar, sa + c * (64 * BK * 2), m0 + c * 64, kx, bi, bo);
                            }
                            if (!p.b_mn) {
                                tma_load_4d_u32(&tma_b, bar, sb, kx, n0, bib, bo);
                            } else if (p.b_mn5) {
                                tma_load_5d_u32(&tma_b, bar, sb, 0, kx, n0 / 64, bib, bo);
                            } else {
                                for (int c = 0; c < (int)bn_local / 64; ++c) tma_load_4d_u32(&tma_b, bar, sb + c * (64 * BK * 2), n0 + c * 64, kx, bib, bo);
                            }
                        } else {
                            // both CTAs report to the leader's barrier; the leader announces the bytes of the pair
                            const uint32_t bar = full_leader0 + 8 * ps;
                            if (rank == 0) mbar_expect_tx_u32(full0 + 8 * ps, 2 * stage_bytes);
                            if (!p.a_mn) {
                                tma_load_4d_2cta_u32(&tma_a, bar, sa, kx, m0, bi, bo);
                            } else if (p.a_mn5) {
                                tma_load_5d_2cta_u32(&tma_a, bar, sa, 0, kx, m0 / 64, bi, bo);
                            } else {
#pragma unroll
                                for (int c = 0; c < BM / 64; ++c) tma_load_4d_2cta_u32(&tma_a, bar, sa + c * (64 * BK * 2), m0 + c * 64, kx, bi, bo);
                            }
                            if (!p.b_mn) {
                                tma_load_4d_2cta_u32(&tma_b, bar, sb, kx, n0, bib, bo);
                            } else if (p.b_mn5) {
                                tma_load_5d_2cta_u32(&tma_b, bar, sb, 0, kx, n0 / 64, bib, bo);
                            } else {
                                for (int c = 0; c < (int)bn_local / 64; ++c) tma_load_4d_2cta_u32(&tma_b, bar, sb + c * (64 * BK * 2), n0 + c * 64, kx, bib, bo);
                            }
                        }
                    }
                    __syncwarp();
                    if (++ps == (uint32_t)p.stages) { ps = 0; pph ^= 1; }
                }
            }
            if ((FUSED == 2 || FUSED == 3) && lane == 0) {
                atomicAdd(&g_fused_stats[0], (unsigned long long)waited);
                atomicMax(&g_fused_stats[3], (unsigned long long)waited);
            }
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------------ MMA issuer (leader CTA only in pair mode)
        // The warp stays converged and one elected lane issues: with a single-lane branch around the loop a 64-deep step
        // cost about 640 clocks of issue time whatever the tile width (the MMAs of a 128-wide tile take 256).
        if (rank == 0) {
            uint32_t tcount = 0;
            bool ok = true;
            uint32_t cs = 0, cph = 0;
            const uint32_t smem0 = smem_u32(smem), full0 = smem_u32(&hdr->full[0]), empty0 = smem_u32(&hdr->empty[0]);
            const uint32_t tfull0 = smem_u32(&hdr->tmem_full[0]), tempty0 = smem_u32(&hdr->tmem_empty[0]);
            // descriptor halves that never change; per MMA only the start address moves: K-major steps 32 bytes inside
            // the 128-byte swizzle row, MN-major steps 16 K rows (2 KiB)
            const uint32_t d_hi = desc_hi(1024);
            const uint32_t a_lbo = p.a_mn ? 64 * BK * 2 : 0, b_lbo = p.b_mn ? 64 * BK * 2 : 0;
            const uint32_t a_kstep = (p.a_mn ? UMMA_K * 128 : UMMA_K * 2) >> 4, b_kstep = (p.b_mn ? UMMA_K * 128 : UMMA_K * 2) >> 4;
            Work work(p, first_tile, tile_step, num_tiles, k_blocks, FUSED == 0 && p.sk_tiles > 0);
            for (Item it; ok && next_item(work, it); ++tcount) {
                const uint32_t acc = tcount & 1;
                const uint32_t acc_ph = (tcount >> 1) & 1;
                if (!mbar_wait_warp(tempty0 + 8 * acc, acc_ph ^ 1)) { ok = false; if (lane == 0) { gave_up<FUSED != 0>(2, p.host_status); hdr->failed = 1; } break; }
                tc_fence_after();
                const uint32_t tmem_c = tmem_base + acc * p.bn;
                for (int kb = it.kb0; kb < it.kb1; ++kb) {
                    if (!mbar_wait_warp(full0 + 8 * cs, cph)) { ok = false; if (lane == 0) { gave_up<FUSED != 0>(3, p.host_status); hdr->failed = 1; } break; }
                    tc_fence_after();
                    const uint32_t sa = smem0 + cs * stage_bytes;
                    const uint32_t a_lo = desc_lo(sa, a_lbo), b_lo = desc_lo(sa + a_bytes, b_lbo);
                    if (elect_one()) {
#pragma unroll
                        for (int k = 0; k < BK / UMMA_K; ++k) {
                            const uint64_t ad = pack_desc(a_lo + k * a_kstep, d_hi), bd = pack_desc(b_lo + k * b_kstep, d_hi);
                            const uint32_t add = (kb > it.kb0 || k != 0) ? 1u : 0u;
                            if (CTA2) umma_f16_2cta(tmem_c, ad, bd, p.idesc, add);
                            else umma_f16(tmem_c, ad, bd, p.idesc, add);
                        }
                        // frees the smem stage (in both CTAs) once these MMAs have read it
                        if (CTA2) umma_commit_2cta_u32(empty0 + 8 * cs); else umma_commit_u32(empty0 + 8 * cs);
                        if (kb + 1 == it.kb1) { if (CTA2) umma_commit_2cta_u32(tfull0 + 8 * acc); else umma_commit_u32(tfull0 + 8 * acc); }
                    }
                    __syncwarp();
                    if (++cs == (uint32_t)p.stages) { cs = 0; cph ^= 1; }
                }
            }
        }
    } else {
        // ------------------------------------------------------------------ epilogue (warps 2..9), own 128 rows
        const int quarter = warp & 3;  // TMEM lanes [32*quarter, 32*quarter + 32) are visible to this warp
        uint32_t tcount = 0;
        uint32_t rs_free_mask = 0;     // destinations whose inbox is known to be free (mode 1)
        bool ok = true;
        bool remote_open = FUSED == 1 && f.rs_early;   // this warp has not yet reported its other-rank tiles as delivered
        auto report_remote_done = [&]() {
            // the warp's stores into other ranks' inboxes are all issued: make them visible and count the warp; the last
            // warp of the rank publishes "delivered" to every rank while the tiles with own rows are still being computed
            asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");   // this thread's row copies have completed
            asm volatile("fence.proxy.async.global;" ::: "memory");
            __threadfence_system();
            __syncwarp();
            if (lane == 0) {
                __threadfence_system();
                const unsigned int done = atomicAdd(f.rs_counter, 1u) + 1u;
                if (done == f.epoch * gridDim.x * 4u) {
                    __threadfence_system();
                    for (int j = 0; j < f.world; ++j) st_release_sys_u32(f.flags[j] + f.done_row * f.world + f.rank, f.epoch);
                }
            }
            remote_open = false;
        };
        Work work(p, first_tile, tile_step, num_tiles, k_blocks, FUSED == 0 && p.sk_tiles > 0);
        for (Item it; ok && next_item(work, it); ++tcount) {
            const int tile = it.tile;
            const int batch = tile / tiles_per_batch;
            const int rem = tile - batch * tiles_per_batch;
            int m_blk, n_blk;
            tile_coords(p, rem, m_blk, n_blk);
            if (FUSED == 1 && f.rs_early) {
                if (remote_open && rem >= f.rs_remote_tiles) report_remote_done();
                m_blk = (m_blk + (f.rank + 1) * f.rs_bpr) % p.m_blocks;   // own rows last
            }
            if (FUSED == 2) m_blk = (m_blk + f.rank * blocks_per_rank) % p.m_blocks;
            if (FUSED == 3) n_blk = (n_blk + f.bg_first_block) % p.n_blocks;
            const int bo = batch / (int)p.batch_inner, bi = batch - bo * (int)p.batch_inner;
            const uint32_t acc = tcount & 1;
            const uint32_t acc_ph = (tcount >> 1) & 1;
            if (!mbar_wait_warp(smem_u32(&hdr->tmem_full[acc]), acc_ph)) { ok = false; if (lane == 0) gave_up<FUSED != 0>(4, p.host_status); break; }
            tc_fence_after();
            const int64_t row0 = (int64_t)m_blk * (BM * NCTA) + rank * BM + quarter * 32;
            const uint32_t taddr = tmem_base + ((uint32_t)(quarter * 32) << 16) + acc * p.bn;
            const int64_t tile_end = (int64_t)(n_blk + 1) * p.bn;
            const int64_t col_end = tile_end < p.N ? tile_end : p.N;
            auto release = [&]() {      // this warp has read the accumulator
                tc_fence_before();
                __syncwarp();
                if (lane == 0) {
                    if (CTA2) mbar_arrive_cluster(map_to_cta(smem_u32(&hdr->tmem_empty[acc]), 0));
                    else mbar_arrive(&hdr->tmem_empty[acc]);
                }
            };
            if (FUSED == 1) {
                const int64_t row = row0 + lane;
                const bool row_ok = row < p.M;
                char* cbase = (char*)p.c;
                int64_t coff = 0;
                if (row_ok) {
                    // route the row to the inbox of its owner; wait once per destination until that rank freed the inbox
                    const int owner = (int)(row / f.rs_rows);
                    if (owner != f.rank && !((rs_free_mask >> owner) & 1u)) {
                        if (!wait_counter(f.flags[f.rank] + f.free_row * f.world + owner, f.epoch, f.limit_ns)) {
                            atomicCAS(f.status, 0, 0x500 | f.rank); atomicCAS(&g_gemm_status, 0, (7 << 16) | (blockIdx.x & 0xffff));
                        }
                        rs_free_mask |= 1u << owner;
                    }
                    cbase = (char*)f.rs_inbox[owner];
                    coff = (row - (int64_t)owner * f.rs_rows) * p.N;
                }
                // bulk-store epilogue: pack OUT_CHUNK columns of the row in shared memory, one bulk copy per row chunk to the
                // row's owner
                const uint32_t srow = smem_u32(smem) + p.out_stage_off + (uint32_t)((quarter * 32 + lane) * OUT_PITCH);
                for (int c0 = 0; c0 < p.bn; c0 += OUT_CHUNK) {
                    const int64_t col0 = (int64_t)n_blk * p.bn + c0;
                    if (col0 >= col_end) break;
                    const int ncols = (int)(col_end - col0 < OUT_CHUNK ? col_end - col0 : OUT_CHUNK);
                    asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");   // the previous copy has read the row buffer
                    for (int sub = 0; sub < OUT_CHUNK; sub += 32) {
                        if (c0 + sub >= p.bn || col0 + sub >= col_end) break;
                        uint32_t r[32];
                        tmem_ld32(taddr + c0 + sub, r);
                        tmem_ld_wait();
                        uint32_t pk[16];
#pragma unroll
                        for (int i = 0; i < 16; ++i) {
                            const float a = __uint_as_float(r[2 * i]) * p.alpha, b = __uint_as_float(r[2 * i + 1]) * p.alpha;
                            if (p.c_dtype == BMT_DT_F16) { __half2 h = __floats2half2_rn(a, b); pk[i] = *reinterpret_cast<uint32_t*>(&h); }
                            else { __nv_bfloat162 h = __floats2bfloat162_rn(a, b); pk[i] = *reinterpret_cast<uint32_t*>(&h); }
                        }
#pragma unroll
                        for (int q = 0; q < 4; ++q)
                            asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(srow + sub * 2 + q * 16), "r"(pk[4 * q]),
                                         "r"(pk[4 * q + 1]), "r"(pk[4 * q + 2]), "r"(pk[4 * q + 3]) : "memory");
                    }
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                    if (row_ok)
                        asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;"
                                     ::"l"(cbase + (coff + col0) * 2), "r"(srow), "r"(ncols * 2) : "memory");
                    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
                }
                release();
            } else {
                const uint32_t sbuf = smem_u32(smem) + p.out_stage_off + (uint32_t)(warp - 2) * EPI_BYTES_PER_WARP;
                const int first = (warp - 2) >> 2;   // two warps see the same 32 rows: they take the 32-column pieces in turn
                const int64_t coff = bi * p.c_bs0 + bo * p.c_bs1, n0 = (int64_t)n_blk * p.bn;
                Partials sk;
                sk.count = 0;
                if (it.kind != 0) {
                    const int cta = first_tile * NCTA + (int)rank;
                    uint32_t* flag = p.sk_flags + cta * SK_WARPS + (warp - 2);
                    const int n_chunks = (int)((col_end - n0 + 31) / 32);
                    float4* slot = p.sk_part + (int64_t)cta * p.sk_slot + (uint32_t)quarter * (p.sk_slot / 4) + lane;
                    if (it.kind == 1) {
                        store_partials(slot, flag, p.sk_tag, n_chunks, taddr, lane, first, release);
                        continue;
                    }
                    sk.slot = (int64_t)NCTA * p.sk_slot;
                    sk.at = slot - sk.slot;
                    sk.count = first_tile - Work::first_of(p, first_tile, tile, k_blocks);
                    if (!wait_partials(flag - NCTA * SK_WARPS, NCTA * SK_WARPS, sk.count, p.sk_tag, lane)) {
                        ok = false;
                        if (lane == 0) { gave_up<FUSED != 0>(12, p.host_status); hdr->failed = 1; }
                        sk.count = -1;
                    } else      // the last item of this CTA: its loads have landed and its MMAs have read them
                        sk.start(smem_u32(smem) + (uint32_t)(warp - 2) * (SK_AHEAD * 4096) + lane * 16, first, 2, n_chunks);
                }
                if (p.c_dtype == BMT_DT_F16) epilogue_tile(p, (__half*)p.c + coff, row0, n0, col_end, taddr, sbuf, lane, first, sk, release);
                else if (p.c_dtype == BMT_DT_BF16) epilogue_tile(p, (__nv_bfloat16*)p.c + coff, row0, n0, col_end, taddr, sbuf, lane, first, sk, release);
                else epilogue_rows_any(p, (float*)p.c + coff, row0, n0, col_end, taddr, sbuf, lane, first, sk, release);
            }
        }
        if (remote_open) report_remote_done();
        if (FUSED == 1) {
            // row copies read this CTA's shared memory and write the inboxes: complete them before the teardown barrier
            asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
            asm volatile("fence.proxy.async.global;" ::: "memory");
            __threadfence_system();
        }
    }

    // ---------------------------------------------------------------------- teardown
    __syncthreads();
    if (FUSED != 0 && threadIdx.x == 0) atomicMax(&g_fused_stats[2], (unsigned long long)(global_ns() - t_kernel0));
    if (hdr->failed) {
        // a wait ran out: give copies that are still in flight time to land before the CTA's shared memory goes away
        const uint64_t t0 = global_ns();
        while (global_ns() - t0 < 2000000ull) __nanosleep(1000);
        __syncthreads();
    }
    if (CTA2) cluster_sync();   // the peer may still be signalling barriers in this CTA's shared memory
    tc_fence_after();
    if (warp == 1) { if (CTA2) tmem_dealloc_2cta(tmem_base, tmem_cols); else tmem_dealloc(tmem_base, tmem_cols); }

    if (FUSED == 1) {
        // ---- reduce phase of GEMM -> reduce-scatter
        __shared__ int rs_ok;
        if (threadIdx.x == 0) {
            bool ok = true;
            if (!f.rs_early) {
                __threadfence_system();  // this CTA's inbox stores (ordered before by the barrier above) become visible system-wide
                const unsigned int done = atomicAdd(f.rs_counter, 1u) + 1u;
                if (done == f.epoch * gridDim.x) {
                    // last CTA of this rank: everything is delivered
                    __threadfence_system();
                    for (int j = 0; j < f.world; ++j) st_release_sys_u32(f.flags[j] + f.done_row * f.world + f.rank, f.epoch);
                }
            } else if (!f.rs_split) {
                // "delivered" went out when the other ranks' tiles were done; the tiles with own rows only have to be complete
                // on this GPU: count the CTA and wait (bounded) for the rest of the grid, all of which is resident
                __threadfence();
                atomicAdd(f.rs_counter + 1, 1u);
                ok = wait_counter(f.rs_counter + 1, f.epoch * gridDim.x, f.limit_ns);
            }
            if (!f.rs_split) {
                const uint64_t tw0 = global_ns();
                for (int j = 0; j < f.world && ok; ++j) ok = wait_counter(f.flags[f.rank] + f.done_row * f.world + j, f.epoch, f.limit_ns);
                atomicMax(&g_fused_stats[5], (unsigned long long)(global_ns() - tw0));
                atomicAdd(&g_fused_stats[7], (unsigned long long)(global_ns() - tw0));
                if (!ok) { atomicCAS(f.status, 0, 0x600 | f.rank); atomicCAS(&g_gemm_status, 0, (8 << 16) | (blockIdx.x & 0xffff)); }
            }
            rs_ok = (ok && !f.rs_split) ? 1 : 0;
        }
        __syncthreads();
        if (rs_ok) {
            const int64_t nvec = f.rs_rows * p.N / 8;
            const int64_t slot_elems = f.rs_rows * p.N;
            if (p.c_dtype == BMT_DT_F16) rs_reduce_all<__half>(f.rs_inbox_local, slot_elems, f.world, f.rs_bias, p.N, f.rs_out, nvec);
            else rs_reduce_all<__nv_bfloat16>(f.rs_inbox_local, slot_elems, f.world, f.rs_bias, p.N, f.rs_out, nvec);
            if (threadIdx.x == 0) atomicMax(&g_fused_stats[6], (unsigned long long)(global_ns() - t_kernel0));
        }
    }
}

// Second half of a split GEMM -> reduce-scatter: sums the inbox slots (+ bias) of this rank's rows once every rank's
// "delivered" flag has been seen by the wait kernel launched before it.  The last CTA tells every rank that this
// rank's inbox may be overwritten by the next use of the ring slot.
template <typename T>
__global__ void __launch_bounds__(NUM_THREADS) rs_reduce_kernel(const void* inbox, int64_t slot_elems, int world, const void* bias, int64_t N,
                                                                 void* out, int64_t nvec, FusedComm f, unsigned int next_epoch) {
    rs_reduce_all<T>(inbox, slot_elems, world, bias, N, out, nvec);
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        const unsigned int done = atomicAdd(f.rs_counter + 1, 1u) + 1u;
        if (done == f.epoch * gridDim.x) {
            for (int j = 0; j < f.world; ++j) st_release_sys_u32(f.flags[j] + f.free_row * f.world + f.rank, next_epoch);
        }
    }
}

// ------------------------------------------------------------------------------------------------ host side
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn get_encode() {
    static EncodeTiledFn fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess && q == cudaDriverEntryPointSuccess)
            fn = (EncodeTiledFn)p;
    });
    return fn;
}

// Makes the primary context current on this thread (autograd worker threads may not have one yet).  cudaFree does that, but
// it invalidates a stream capture, so it is called only where there is none.
void bind_context() {
    typedef CUresult (*GetCurrentFn)(CUcontext*);
    static GetCurrentFn fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuCtxGetCurrent", &p, cudaEnableDefault, &q) == cudaSuccess && q == cudaDriverEntryPointSuccess)
            fn = (GetCurrentFn)p;
    });
    CUcontext ctx = nullptr;
    if (!fn || fn(&ctx) != CUDA_SUCCESS || !ctx) cudaFree(0);
}

struct MapKey {
    const void* ptr;
    int64_t d[4], s[3];
    int box0, box1, dtype;
    int chunks;   // 0: 4-D map; > 0: 5-D map of an MN-major operand with this many 64-element chunks per box
    bool operator==(const MapKey& o) const { return memcmp(this, &o, sizeof(MapKey)) == 0; }
};
struct MapKeyHash {
    size_t operator()(const MapKey& k) const {
        const uint64_t* w = (const uint64_t*)&k;
        size_t h = 1469598103934665603ull;
        for (size_t i = 0; i < sizeof(MapKey) / 8; ++i) h = (h ^ w[i]) * 1099511628211ull;
        return h;
    }
};
std::unordered_map<MapKey, CUtensorMap, MapKeyHash> g_maps;
std::mutex g_maps_mu;

// 4-D map: dims {inner, rows, batch_inner, batch_outer}; element strides for dims 1..3.
int make_map(CUtensorMap* out, const void* ptr, int dtype, int64_t inner, int64_t rows, int64_t ld, int64_t nb0, int64_t bs0,
             int64_t nb1, int64_t bs1, int box_inner, int box_rows) {
    MapKey key;
    memset(&key, 0, sizeof(key));
    key.ptr = ptr; key.d[0] = inner; key.d[1] = rows; key.d[2] = nb0; key.d[3] = nb1;
    key.s[0] = ld; key.s[1] = bs0; key.s[2] = bs1; key.box0 = box_inner; key.box1 = box_rows; key.dtype = dtype;
    {
        std::lock_guard<std::mutex> lk(g_maps_mu);
        auto it = g_maps.find(key);
        if (it != g_maps.end()) { *out = it->second; return 0; }
    }
    EncodeTiledFn enc = get_encode();
    if (!enc) return -10;
    if (((uintptr_t)ptr & 15) || (ld & 7) || (nb0 > 1 && (bs0 & 7)) || (nb1 > 1 && (bs1 & 7))) return -11;
    cuuint64_t dims[4] = {(cuuint64_t)inner, (cuuint64_t)rows, (cuuint64_t)nb0, (cuuint64_t)nb1};
    // strides of unit-extent dims are irrelevant but must still be legal (multiple of 16 bytes, non-zero)
    cuuint64_t st[3] = {(cuuint64_t)ld * 2, (cuuint64_t)(nb0 > 1 ? bs0 : ld * rows) * 2, (cuuint64_t)(nb1 > 1 ? bs1 : ld * rows) * 2};
    if (st[1] == 0) st[1] = 16;
    if (st[2] == 0) st[2] = 16;
    cuuint32_t box[4] = {(cuuint32_t)box_inner, (cuuint32_t)box_rows, 1, 1};
    cuuint32_t es[4] = {1, 1, 1, 1};
    bind_context();
    CUresult r = enc(out, dtype == BMT_DT_F16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, (void*)ptr,
                     dims, st, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                     CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        fprintf(stderr, "bmtrain_b200: cuTensorMapEncodeTiled failed (%d): ptr=%p dims={%lld,%lld,%lld,%lld} strides={%lld,%lld,%lld} box={%d,%d}\n",
                (int)r, ptr, (long long)dims[0], (long long)dims[1], (long long)dims[2], (long long)dims[3], (long long)st[0],
                (long long)st[1], (long long)st[2], box_inner, box_rows);
        return -12;
    }
    std::lock_guard<std::mutex> lk(g_maps_mu);
    if (g_maps.size() > 8192) g_maps.clear();
    g_maps[key] = *out;
    return 0;
}

}  // namespace

// Cached 4-D tensor map {inner, rows, batch_inner, batch_outer} for the other tensor-core kernels of this library.
int bmt_tma_map_4d(CUtensorMap* out, const void* ptr, int dtype, int64_t inner, int64_t rows, int64_t ld, int64_t nb0, int64_t bs0,
                   int64_t nb1, int64_t bs1, int box_inner, int box_rows) {
    return make_map(out, ptr, dtype, inner, rows, ld, nb0, bs0, nb1, bs1, box_inner, box_rows);
}

int bmt_tma_map_f32_3d(CUtensorMap* out, const void* ptr, int64_t inner, int64_t rows, int64_t nb, int box_inner, int box_rows) {
    EncodeTiledFn enc = get_encode();
    if (!enc) return -10;
    if (((uintptr_t)ptr & 15) || (inner & 3)) return -11;
    cuuint64_t dims[3] = {(cuuint64_t)inner, (cuuint64_t)rows, (cuuint64_t)nb};
    cuuint64_t st[2] = {(cuuint64_t)inner * 4, (cuuint64_t)(inner * rows) * 4};
    cuuint32_t box[3] = {(cuuint32_t)box_inner, (cuuint32_t)box_rows, 1};
    cuuint32_t es[3] = {1, 1, 1};
    bind_context();
    const CUresult r = enc(out, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, (void*)ptr, dims, st, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
                           CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? 0 : -12;
}

namespace {

// 5-D map of an MN-major operand (element (k, mn) at ptr + k * ld + mn, mn contiguous): dims {64, k rows, mn / 64 chunks,
// batch_inner, batch_outer}; the chunk dimension has a stride of 64 elements, so one box {64, box_rows, chunks} lands in
// shared memory as `chunks` consecutive [box_rows][64] swizzled blocks -- the layout one copy per chunk produces, with one
// copy.  Only for mn extents that are multiples of 64 (the inner dimension is the fixed 64 of a chunk, so a ragged last
// chunk could not be bounds-checked by the copy engine).
int make_map_mn5(CUtensorMap* out, const void* ptr, int dtype, int64_t mn, int64_t rows, int64_t ld, int64_t nb0, int64_t bs0,
                 int64_t nb1, int64_t bs1, int box_rows, int chunks) {
    if (mn % 64 != 0) return -13;
    MapKey key;
    memset(&key, 0, sizeof(key));
    key.ptr = ptr; key.d[0] = mn; key.d[1] = rows; key.d[2] = nb0; key.d[3] = nb1;
    key.s[0] = ld; key.s[1] = bs0; key.s[2] = bs1; key.box0 = 64; key.box1 = box_rows; key.dtype = dtype; key.chunks = chunks;
    {
        std::lock_guard<std::mutex> lk(g_maps_mu);
        auto it = g_maps.find(key);
        if (it != g_maps.end()) { *out = it->second; return 0; }
    }
    EncodeTiledFn enc = get_encode();
    if (!enc) return -10;
    if (((uintptr_t)ptr & 15) || (ld & 7) || (nb0 > 1 && (bs0 & 7)) || (nb1 > 1 && (bs1 & 7))) return -11;
    cuuint64_t dims[5] = {64, (cuuint64_t)rows, (cuuint64_t)(mn / 64), (cuuint64_t)nb0, (cuuint64_t)nb1};
    cuuint64_t st[4] = {(cuuint64_t)ld * 2, 128, (cuuint64_t)(nb0 > 1 ? bs0 : ld * rows) * 2, (cuuint64_t)(nb1 > 1 ? bs1 : ld * rows) * 2};
    if (st[2] == 0) st[2] = 16;
    if (st[3] == 0) st[3] = 16;
    cuuint32_t box[5] = {64, (cuuint32_t)box_rows, (cuuint32_t)chunks, 1, 1};
    cuuint32_t es[5] = {1, 1, 1, 1, 1};
    bind_context();
    CUresult r = enc(out, dtype == BMT_DT_F16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 5, (void*)ptr,
                     dims, st, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                     CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return -12;   // the caller falls back to one 4-D copy per chunk
    std::lock_guard<std::mutex> lk(g_maps_mu);
    if (g_maps.size() > 8192) g_maps.clear();
    g_maps[key] = *out;
    return 0;
}

// SMs that fused (compute + collective) kernels leave free.  Their CTAs wait for other ranks while they hold their SM; when
// kernels of another parallel dimension (NCCL gathers of a ZeRO group) must be able to start next to them at any time, a
// few SMs stay out of the fused grids so that such a kernel always finds room (bmt_gemm_reserve_sms).
int g_reserved_sms = 0;

// Tile selection.  Per k-block (64 deep) an SM spends about 2.05 * BN clocks on the MMAs of its 128 accumulator rows
// and has to pull (128 + BN / ncta) * 128 bytes from L2 at about 64 bytes per clock; the slower of the two sets
// the pace.  A CTA pair (cta_group::2, 256 x BN tile) halves the B bytes per SM, which is what lifts large
// problems off the L2->SM limit.  The cost also counts waves on the available SMs and a fixed per-tile overhead.
//
// Split tiles (`split`) spread the tiles of the partial wave, with the wave before it if there is one, evenly over all CTAs, or over
// as many as leave a range SK_MIN k-blocks.  Handing the sums over costs about SK_COST clocks, mostly waiting and fp32 through L2: 3 us
// behind a long reduction and up to 10 where all SMs write and read their slots at once.  So the estimate has to win by 12 %
// where there is less than a wave (1024 x 2560 x 8192 in the dgrad layout: 50 -> 43 us; 56 x 720 x 9144: 41 -> 19; 777 x 2560 x 7680,
// estimated 11 % better, took 41 instead of 40) and by 2 % behind whole waves (4096 x 5120 x 27648: 807 -> 738 us;
// 2048 x 57344 x 8192: 1256 -> 1208; 2560 x 8192 x 1024, not chosen, would take 44 instead of 38).  A single row of tiles reads its large operand
// once: where that lies along N, does not fit L2, and nearly all SMs have a whole wide tile of it, the memory is the bound and the tiles stay
// whole (88 x 17944 x 24864 in the dgrad layout: 153 us, at 5.9 TB/s, against 176; 24 x 17752 x 16256: 91 and 118).  Not so in the other layout (80 x 16928
// x 23016: 164 us divided, 212 whole) or with more rows (128 x 17456 x 16536: 123 and 146).
struct TileChoice { int bn, cta2, sk_tiles, sk_workers; };
constexpr int SK_MIN = 4, SK_MOST = 8;      // k-blocks of a range at least, CTAs per tile at most
constexpr double SK_COST = 16000.0;
constexpr double L2_BYTES = 126e6;

// `sms`: that do math
TileChoice pick_tile(int64_t M, int64_t N, int64_t K, int64_t batches, bool b_mn, int force_bn, int force_cta2, bool split, int sms) {
    TileChoice best{0, 0, 0, 0}, best_split{0, 0, 0, 0};
    double best_cost = 1e30, best_split_cost = 1e30, busy = 0.0;      // part of the SMs that `best` keeps busy, if it takes one wave
    const int64_t kblocks = (K + BK - 1) / BK;
    for (int cta2 = 0; cta2 <= 1; ++cta2) {
        if (force_cta2 >= 0 && cta2 != force_cta2) continue;
        if (cta2 && M <= BM) continue;
        const int ncta = cta2 ? 2 : 1;
        const int step = (b_mn ? 64 : 16) * ncta;
        for (int bn = (b_mn ? 64 : 32) * ncta; bn <= 256; bn += step) {
            if (force_bn > 0 && bn != force_bn) continue;
            const int64_t tiles = ((M + BM * ncta - 1) / (BM * ncta)) * ((N + bn - 1) / bn) * batches;
            const int64_t slots = sms / ncta;
            const int64_t waves = (tiles + slots - 1) / slots;
            const double mma = 2.05 * bn, load = 2.0 * (128 + bn / ncta);
            const double per_block = mma > load ? mma : load, fixed = 600.0 + 6.0 * bn;   // + fill/drain and epilogue
            const double cost = (double)waves * (kblocks * per_block + fixed);
            if (cost < best_cost * 0.999) { best_cost = cost; best = TileChoice{bn, cta2, 0, 0}; busy = waves == 1 ? (double)tiles / slots : 0.0; }
            if (!split || tiles % slots == 0) continue;
            const bool behind = tiles > slots;              // behind whole waves
            const int64_t sk_tiles = tiles % slots + (behind ? slots : 0), total = sk_tiles * kblocks;
            int64_t workers = slots;
            if (workers > sk_tiles * SK_MOST) workers = sk_tiles * SK_MOST;
            if (workers > total / SK_MIN) workers = total / SK_MIN;
            if (workers <= sk_tiles && !behind) continue;
            const int64_t whole_waves = (tiles - sk_tiles) / slots;
            const double parts = (double)workers / sk_tiles;        // a CTA adds what the others left of its tile: 8 * bn clocks a slot
            const double estimate = (whole_waves * kblocks + (double)total / workers) * per_block + (whole_waves + 2) * fixed + SK_COST +
                                    (parts > 1 ? (parts - 1) * 8 * bn : 0);
            const double c = estimate / (behind ? 0.98 : 0.88);
            if (c < best_split_cost) { best_split_cost = c; best_split = TileChoice{bn, cta2, (int)sk_tiles, (int)workers}; }
        }
    }
    const double bytes = 2.0 * batches * ((double)M * K + (double)N * K + (double)M * N);
    if (b_mn && M <= 96 && best.bn >= 128 && busy >= 0.85 && bytes > L2_BYTES) return best;
    return best_split_cost < best_cost ? best_split : best;
}

// The choice for a problem costs 2 to 4 us of divisions; a thread keeps its last ones.
TileChoice planned_tile(int64_t M, int64_t N, int64_t K, int64_t batches, bool b_mn, int force_bn, int force_cta2, bool split, int sms) {
    struct Plan { int64_t m, n, k, batches; int how, sms; TileChoice tc; };
    static thread_local Plan plans[256];
    const int how = 1 + (b_mn ? 1 : 0) + (split ? 2 : 0) + 4 * (force_cta2 + 1) + 16 * force_bn;
    const uint64_t hash = ((uint64_t)M * 0x9e3779b97f4a7c15ull) ^ ((uint64_t)N * 0xc2b2ae3d27d4eb4full) ^ ((uint64_t)K * 0x165667b19e3779f9ull) ^
                          ((uint64_t)batches * 0x27d4eb2f165667c5ull) ^ ((uint64_t)how * 0x85ebca77c2b2ae63ull);
    Plan& p = plans[(hash >> 40) & 255];
    if (p.how != how || p.m != M || p.n != N || p.k != K || p.batches != batches || p.sms != sms)
        p = Plan{M, N, K, batches, how, sms, pick_tile(M, N, K, batches, b_mn, force_bn, force_cta2, split, sms)};
    return p.tc;
}

// Tensor of a scratch: flags of all CTAs, then their slots.
int64_t sk_bytes(int ctas, int bn) { return (int64_t)ctas * (SK_WARPS * 4 + 128 * ((bn + 31) / 32 * 32) * 4); }
std::atomic<uint32_t> g_sk_tag{0};

void set_split(GemmParams& p, const TileChoice& tc, int k_blocks) {
    p.sk_tiles = tc.sk_tiles; p.sk_workers = tc.sk_workers;
    p.sk_snap = (int64_t)tc.sk_tiles * k_blocks / tc.sk_workers >= 16 ? 3 : 1;     // ranges stay longer than two snaps
}

// CTAs (pairs) of a launch with split tiles: whole tiles come only in full waves.
int64_t whole_or_split(int64_t tiles, int64_t slots, const TileChoice& tc) { return tiles > tc.sk_tiles ? slots : tc.sk_workers; }

// Where kernels report waits that ran out (see gave_up).
int* g_host_status = nullptr;

// Once, whichever thread comes first.
int prepare_kernels() {
    static std::atomic<bool> done{false};
    if (done.load(std::memory_order_acquire)) return 0;
    static std::mutex mu;
    std::lock_guard<std::mutex> lock(mu);
    if (done.load(std::memory_order_relaxed)) return 0;
    const int most = (int)(SMEM_MAX - SMEM_FIXED + 1024 + 512);
    for (const auto kernel : {gemm_tcgen05_kernel<false, 0>, gemm_tcgen05_kernel<true, 0>, gemm_tcgen05_kernel<false, 1>, gemm_tcgen05_kernel<false, 2>,
                              gemm_tcgen05_kernel<false, 3>, gemm_tcgen05_kernel<true, 1>, gemm_tcgen05_kernel<true, 2>, gemm_tcgen05_kernel<true, 3>})
        BMT_CUDA_OK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, most));
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;      // allocates, which the first launch may have to do under a capture
    BMT_CUDA_OK(cudaThreadExchangeStreamCaptureMode(&mode));
    const cudaError_t e = cudaHostAlloc((void**)&g_host_status, sizeof(int), cudaHostAllocPortable | cudaHostAllocMapped);
    cudaThreadExchangeStreamCaptureMode(&mode);
    BMT_CUDA_OK(e);
    *g_host_status = 0;
    done.store(true, std::memory_order_release);
    return 0;
}

int launch_gemm(const BmtGemmDesc& g, cudaStream_t stream, const FusedComm* fused = nullptr) {
    const int64_t m = g.m, n = g.n, k = g.k;
    const void* a = g.a; const void* b = g.b; void* c = g.c; const void* bias = g.bias;
    const int64_t lda = g.lda, ldb = g.ldb, ldc = g.ldc;
    const int a_major = g.a_major, b_major = g.b_major, c_dtype = g.c_dtype, act = g.act, accumulate = g.accumulate, ab_dtype = g.ab_dtype;
    const int64_t a_bs0 = g.a_bs0, a_bs1 = g.a_bs1, b_bs0 = g.b_bs0, b_bs1 = g.b_bs1, c_bs0 = g.c_bs0, c_bs1 = g.c_bs1;
    const int64_t batch_inner = g.batch_inner > 0 ? g.batch_inner : 1, batch_outer = g.batch_outer > 0 ? g.batch_outer : 1;
    const int64_t b_inner_div = g.b_inner_div;
    const float alpha = g.alpha;
    if (m <= 0 || n <= 0 || batch_inner <= 0 || batch_outer <= 0) return 0;
    if (k <= 0) return -20;
    const int sms = bmt::sm_count();
    if (const int rc = prepare_kernels()) return rc;
    if (!fused && *(volatile int*)g_host_status != 0) return -60;     // until bmt_gemm_status has been read
    static int force_bn = -1, force_cta2 = -2;
    if (force_bn < 0) { const char* e = getenv("BMT_GEMM_BN"); force_bn = e ? atoi(e) : 0; }
    if (force_cta2 == -2) { const char* e = getenv("BMT_GEMM_CTA2"); force_cta2 = e ? atoi(e) : -1; }

    GemmParams p;
    memset(&p, 0, sizeof(p));
    p.M = m; p.N = n; p.K = k;
    p.a_mn = a_major; p.b_mn = b_major;
    const int comm_ctas = (fused && (fused->mode == 2 || fused->mode == 3)) ? fused->ag_ctas : 0;
    const int held_back = fused ? comm_ctas + g_reserved_sms : 0;
    // a fused kernel can run as CTA pairs when its pusher CTAs pair up too and (mode 2) a rank's rows fill whole 256-row tiles
    const bool pair_ok = !fused || (comm_ctas % 2 == 0 && (fused->mode != 2 || fused->ag_rows % (2 * BM) == 0));
    // Split tiles need scratch whose flags nobody else uses.  A captured launch may be replayed next to any other, on any stream: there
    // the tiles stay whole.
    bool split = !fused && g.scratch && k < (1 << 26) && g.scratch_bytes >= sk_bytes(sms, 256);
    if (split) {
        cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
        if (cudaStreamIsCapturing(stream, &capture) != cudaSuccess || capture != cudaStreamCaptureStatusNone) { cudaGetLastError(); split = false; }
    }
    TileChoice tc = planned_tile(m, n, k, batch_inner * batch_outer, b_major != 0, force_bn, pair_ok ? force_cta2 : 0, split, sms - held_back);
    if (tc.bn == 0) tc = pick_tile(m, n, k, batch_inner * batch_outer, b_major != 0, 0, -1, split, sms);  // forced shape not applicable here
    if (tc.bn == 0) return -22;
    p.bn = tc.bn;
    const int ncta = tc.cta2 ? 2 : 1;
    const uint32_t stage_bytes = BM * BK * 2 + (p.bn / ncta) * BK * 2;
    const uint32_t out_stage_bytes = (fused && fused->mode == 1) ? BM * OUT_PITCH : epilogue_warps(0) * EPI_BYTES_PER_WARP;
    int stages = (int)((SMEM_MAX - SMEM_FIXED - out_stage_bytes) / stage_bytes);
    p.stages = stages > MAX_STAGES ? MAX_STAGES : stages;
    p.m_blocks = (int)((m + BM * ncta - 1) / (BM * ncta));
    p.n_blocks = (int)((n + p.bn - 1) / p.bn);
    p.batch_inner = batch_inner; p.batch_outer = batch_outer; p.b_inner_div = b_inner_div > 0 ? b_inner_div : 1;
    p.c = c; p.ldc = ldc; p.c_bs0 = c_bs0; p.c_bs1 = c_bs1; p.c_dtype = c_dtype;
    p.host_status = g_host_status;
    p.bias = bias; p.bias_dtype = ab_dtype; p.act = act; p.accumulate = accumulate; p.alpha = alpha;
    static int group_env = -1;
    if (group_env < 0) { const char* e = getenv("BMT_GEMM_GROUP_M"); group_env = e ? atoi(e) : 0; }
    p.group_m = group_env > 0 ? group_env : 16;
    if (tc.sk_tiles) {
        set_split(p, tc, (int)((k + BK - 1) / BK));
        do p.sk_tag = g_sk_tag.fetch_add(1, std::memory_order_relaxed) + 1; while (p.sk_tag == 0);
        p.sk_flags = (uint32_t*)g.scratch;
        p.sk_part = (float4*)((char*)g.scratch + (int64_t)sms * SK_WARPS * 4);
        p.sk_slot = (uint32_t)(128 * ((p.bn + 31) / 32 * 32) / 4);
    }
    if (p.group_m > p.m_blocks) p.group_m = p.m_blocks;
    if (fused && fused->mode == 3) p.group_m = p.m_blocks;  // all row tiles of one weight chunk in a row: chunks are needed in order
    const bool rs_early = fused && fused->mode == 1 && fused->rs_rows % (BM * ncta) == 0;
    if (rs_early) {
        const int per_rank = (int)(fused->rs_rows / (BM * ncta));
        while (per_rank % p.group_m) --p.group_m;   // groups must not mix rows of this rank with rows of others
    }
    if (fused && fused->mode == 2) {
        // groups must not straddle the rows of two ranks (the tile order is rotated rank by rank)
        const int per_rank = (int)(fused->ag_rows / (BM * ncta));
        while (per_rank % p.group_m) --p.group_m;
    }
    p.residual = g.residual; p.ldr = g.ldr; p.round_first = g.residual ? g.round_first : 0; p.aux = g.aux; p.ld_aux = g.ld_aux; p.aux_mode = g.aux ? g.aux_mode : 0;
    if ((p.residual || p.aux_mode) && batch_inner * batch_outer != 1) return -21;  // fused extras are for plain (unbatched) GEMMs
    {
        // the compiled forms of the epilogue move 16-byte vectors of the operand type: every pitch and pointer has to allow it
        auto vec16 = [](const void* ptr, int64_t ld) { return (ld & 7) == 0 && ((uintptr_t)ptr & 15) == 0; };
        const int extras = (accumulate ? 1 : 0) + (p.residual ? 1 : 0) + (p.aux_mode ? 1 : 0);
        const bool ok = c_dtype == ab_dtype && n % 8 == 0 && vec16(c, ldc) && ((c_bs0 | c_bs1) & 7) == 0 && act != 2 && extras <= 1 &&
                        vec16(bias, 0) && vec16(p.residual, p.residual ? p.ldr : 0) && vec16(p.aux, p.aux_mode ? p.ld_aux : 0);
        p.epi = !ok ? -1 : (accumulate || p.residual) ? 1 : p.aux_mode == 1 ? 2 : p.aux_mode == 2 ? 3 : 0;
    }
    const uint32_t fmt = ab_dtype == BMT_DT_F16 ? 0u : 1u;
    p.idesc = (1u << 4) | (fmt << 7) | (fmt << 10) | ((uint32_t)(a_major ? 1 : 0) << 15) | ((uint32_t)(b_major ? 1 : 0) << 16) |
              ((uint32_t)(p.bn >> 3) << 17) | ((uint32_t)((BM * ncta) >> 4) << 24);

    CUtensorMap ma, mb;
    int rc;
    const int64_t nb_b = (batch_inner + p.b_inner_div - 1) / p.b_inner_div;
    static int mn5_env = -1;
    if (mn5_env < 0) { const char* e = getenv("BMT_GEMM_MN5"); mn5_env = e ? atoi(e) : 1; }
    if (!a_major) rc = make_map(&ma, a, ab_dtype, k, m, lda, batch_inner, a_bs0, batch_outer, a_bs1, BK, BM);
    else {
        rc = mn5_env ? make_map_mn5(&ma, a, ab_dtype, m, k, lda, batch_inner, a_bs0, batch_outer, a_bs1, BK, BM / 64) : -1;
        p.a_mn5 = rc == 0 ? 1 : 0;
        if (rc) rc = make_map(&ma, a, ab_dtype, m, k, lda, batch_inner, a_bs0, batch_outer, a_bs1, 64, BK);
    }
    if (rc) return rc;
    if (!b_major) rc = make_map(&mb, b, ab_dtype, k, n, ldb, nb_b, b_bs0, batch_outer, b_bs1, BK, p.bn / ncta);
    else {
        rc = mn5_env ? make_map_mn5(&mb, b, ab_dtype, n, k, ldb, nb_b, b_bs0, batch_outer, b_bs1, BK, (p.bn / ncta) / 64) : -1;
        p.b_mn5 = rc == 0 ? 1 : 0;
        if (rc) rc = make_map(&mb, b, ab_dtype, n, k, ldb, nb_b, b_bs0, batch_outer, b_bs1, 64, BK);
    }
    if (rc) return rc;

    const int64_t tiles = (int64_t)p.m_blocks * p.n_blocks * batch_inner * batch_outer;
    if (tiles > 0x3fffffff) return -23;   // the kernel counts tiles in 32 bits (2^30 tiles are 3e13 elements of C)
    p.out_stage_off = (uint32_t)p.stages * stage_bytes;
    p.hdr_off = p.out_stage_off + out_stage_bytes;
    if (comm_ctas > 0 && p.hdr_off < PUSH_STAGES * PUSH_PIECE_BYTES) p.hdr_off = PUSH_STAGES * PUSH_PIECE_BYTES;
    const size_t smem = (size_t)p.hdr_off + sizeof(SharedHeader) + 1024;
    FusedComm none;
    memset(&none, 0, sizeof(none));
    if (fused) {
        const int compute = (sms - held_back) / ncta;   // CTAs (or CTA pairs) that do math
        const unsigned grid = (unsigned)(ncta * (tiles < compute ? tiles : compute)) + comm_ctas;
        FusedComm fc = *fused;
        if (fc.mode == 3) fc.bg_first_block = (int)(((fc.bg_first / k) / p.bn) % p.n_blocks);
        if (fc.mode == 1) {
            fc.rs_early = rs_early ? 1 : 0;
            fc.rs_bpr = rs_early ? (int)(fc.rs_rows / (BM * ncta)) : 0;
            fc.rs_remote_tiles = rs_early ? (int64_t)(p.m_blocks - fc.rs_bpr) * p.n_blocks : 0;
        }
        if (!tc.cta2) {
            if (fc.mode == 1) gemm_tcgen05_kernel<false, 1><<<grid, NUM_THREADS, smem, stream>>>(ma, mb, p, fc);
            else if (fc.mode == 2) gemm_tcgen05_kernel<false, 2><<<grid, num_threads(2), smem, stream>>>(ma, mb, p, fc);
            else gemm_tcgen05_kernel<false, 3><<<grid, num_threads(3), smem, stream>>>(ma, mb, p, fc);
            bmt_count_launch(1);
            return (int)cudaGetLastError();
        }
        cudaLaunchConfig_t cfg;
        memset(&cfg, 0, sizeof(cfg));
        cfg.gridDim = dim3(grid);
        cfg.blockDim = dim3(num_threads(fc.mode));
        cfg.dynamicSmemBytes = smem;
        cfg.stream = stream;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = 2; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr; cfg.numAttrs = 1;
        cudaError_t e;
        if (fc.mode == 1) e = cudaLaunchKernelEx(&cfg, gemm_tcgen05_kernel<true, 1>, ma, mb, p, fc);
        else if (fc.mode == 2) e = cudaLaunchKernelEx(&cfg, gemm_tcgen05_kernel<true, 2>, ma, mb, p, fc);
        else e = cudaLaunchKernelEx(&cfg, gemm_tcgen05_kernel<true, 3>, ma, mb, p, fc);
        bmt_count_launch(1);
        return e != cudaSuccess ? (int)e : (int)cudaGetLastError();
    }
    if (!tc.cta2) {
        const unsigned grid = (unsigned)(tc.sk_tiles ? whole_or_split(tiles, sms, tc) : tiles < sms ? tiles : sms);
        const cudaError_t e = bmt::launch(gemm_tcgen05_kernel<false, 0>, grid, num_threads(0), smem, stream, 1, ma, mb, p, none);
        bmt_count_launch(1);
        return e != cudaSuccess ? (int)e : (int)cudaGetLastError();
    }
    const int64_t pairs = sms / 2;
    const unsigned grid = (unsigned)(2 * (tc.sk_tiles ? whole_or_split(tiles, pairs, tc) : tiles < pairs ? tiles : pairs));
    const cudaError_t e = bmt::launch(gemm_tcgen05_kernel<true, 0>, grid, num_threads(0), smem, stream, 2, ma, mb, p, none);
    bmt_count_launch(1);
    return e != cudaSuccess ? (int)e : (int)cudaGetLastError();
}

}  // namespace

extern "C" int bmt_gemm_reserve_sms(int n) {
    g_reserved_sms = n <= 0 ? 0 : (n > 64 ? 64 : (n & ~1));
    return 0;
}

// How a GEMM that has scratch is divided: plan = {tile width, CTAs per tile, tiles, split tiles, CTAs (pairs) that share them, CTAs
// (pairs) of the grid}; the items of `worker` (tile, first and last k-block, kind, first of the workers that leave sums) go to `items`.
// Returns their number.  Host arithmetic only.
extern "C" int bmt_gemm_plan(int64_t m, int64_t n, int64_t k, int b_major, int worker, int64_t* plan, int* items, int most) {
    const int sms = bmt::sm_count();
    const TileChoice tc = pick_tile(m, n, k, 1, b_major != 0, 0, -1, true, sms);
    const int ncta = tc.cta2 ? 2 : 1, k_blocks = (int)((k + BK - 1) / BK);
    const int64_t tiles = ((m + BM * ncta - 1) / (BM * ncta)) * ((n + tc.bn - 1) / tc.bn), slots = sms / ncta;
    const int64_t grid = tc.sk_tiles ? whole_or_split(tiles, slots, tc) : tiles < slots ? tiles : slots;
    const int64_t out[6] = {tc.bn, ncta, tiles, tc.sk_tiles, tc.sk_workers, grid};
    memcpy(plan, out, sizeof(out));
    GemmParams p;
    memset(&p, 0, sizeof(p));
    if (tc.sk_tiles) set_split(p, tc, k_blocks);
    Work work(p, worker, (int)grid, (int)tiles, k_blocks, tc.sk_tiles > 0);
    int count = 0;
    for (Item it; work.next(it); ++count) {
        if (count >= most) return -2;
        const int row[5] = {it.tile, it.kb0, it.kb1, it.kind, it.kind == 2 ? Work::first_of(p, worker, it.tile, k_blocks) : worker};
        memcpy(items + 5 * count, row, sizeof(row));
    }
    return count;
}

extern "C" int64_t bmt_gemm_scratch_bytes(void) {
    return sk_bytes(bmt::sm_count(), 256);
}

extern "C" int bmt_gemm_ex(const BmtGemmDesc* desc, void* stream) { return launch_gemm(*desc, (cudaStream_t)stream); }

extern "C" int bmt_gemm(int64_t m, int64_t n, int64_t k, const void* a, int64_t lda, int a_major, const void* b, int64_t ldb,
                        int b_major, void* c, int64_t ldc, int c_dtype, const void* bias, int act, int accumulate, int ab_dtype,
                        void* scratch, int64_t scratch_bytes, void* stream) {
    BmtGemmDesc g;
    memset(&g, 0, sizeof(g));
    g.m = m; g.n = n; g.k = k; g.a = a; g.lda = lda; g.a_major = a_major; g.b = b; g.ldb = ldb; g.b_major = b_major;
    g.c = c; g.ldc = ldc; g.c_dtype = c_dtype; g.bias = bias; g.act = act; g.accumulate = accumulate; g.ab_dtype = ab_dtype;
    g.batch_inner = g.batch_outer = g.b_inner_div = 1; g.alpha = 1.0f; g.scratch = scratch; g.scratch_bytes = scratch_bytes;
    return launch_gemm(g, (cudaStream_t)stream);
}

extern "C" int bmt_gemm_batched(int64_t m, int64_t n, int64_t k, const void* a, int64_t lda, int a_major, int64_t a_bs0,
                                int64_t a_bs1, const void* b, int64_t ldb, int b_major, int64_t b_bs0, int64_t b_bs1, void* c,
                                int64_t ldc, int c_dtype, int64_t c_bs0, int64_t c_bs1, int64_t batch_inner, int64_t batch_outer,
                                int64_t b_inner_div, float alpha, int ab_dtype, void* stream) {
    BmtGemmDesc g;
    memset(&g, 0, sizeof(g));
    g.m = m; g.n = n; g.k = k; g.a = a; g.lda = lda; g.a_major = a_major; g.a_bs0 = a_bs0; g.a_bs1 = a_bs1;
    g.b = b; g.ldb = ldb; g.b_major = b_major; g.b_bs0 = b_bs0; g.b_bs1 = b_bs1;
    g.c = c; g.ldc = ldc; g.c_dtype = c_dtype; g.c_bs0 = c_bs0; g.c_bs1 = c_bs1;
    g.batch_inner = batch_inner; g.batch_outer = batch_outer; g.b_inner_div = b_inner_div; g.alpha = alpha; g.ab_dtype = ab_dtype;
    return launch_gemm(g, (cudaStream_t)stream);
}

// GEMM -> reduce-scatter over the rows of C (see FusedComm mode 1).  `inbox_slots[j]`: where this rank's slot starts in rank
// j's inbox; `grid_hint` receives the number of CTAs launched (the caller's counter advances by it per call).
// Reduce phase of a split GEMM -> reduce-scatter (bmt_gemm_reduce_scatter_main): to be launched after a wait kernel has
// seen every rank's "delivered" flag for `epoch`.  `counter_u32`: the same two counters the main kernel was given.
extern "C" int bmt_gemm_rs_reduce(const void* inbox_local, int64_t rows_per_rank, int64_t n, int world, int rank, void* const* flags,
                                  int free_row, unsigned int epoch, void* counter_u32, void* out, const void* bias, int dtype,
                                  void* stream) {
    if (world < 2 || world > 8 || n % 8 != 0) return -40;
    FusedComm f;
    memset(&f, 0, sizeof(f));
    f.world = world; f.rank = rank; f.free_row = free_row; f.epoch = epoch; f.rs_counter = (unsigned int*)counter_u32;
    for (int j = 0; j < world; ++j) f.flags[j] = (unsigned int*)flags[j];
    const int64_t nvec = rows_per_rank * n / 8, slot_elems = rows_per_rank * n;
    int64_t blocks = (nvec + NUM_THREADS * 4 - 1) / (NUM_THREADS * 4);
    if (blocks > 148) blocks = 148;
    if (blocks < 1) blocks = 1;
    cudaStream_t st = (cudaStream_t)stream;
    if (dtype == BMT_DT_F16) rs_reduce_kernel<__half><<<(unsigned)blocks, NUM_THREADS, 0, st>>>(inbox_local, slot_elems, world, bias, n, out, nvec, f, epoch + 1);
    else rs_reduce_kernel<__nv_bfloat16><<<(unsigned)blocks, NUM_THREADS, 0, st>>>(inbox_local, slot_elems, world, bias, n, out, nvec, f, epoch + 1);
    bmt_count_launch(1);
    return (int)cudaGetLastError();
}

static int gemm_reduce_scatter_impl(const BmtGemmDesc* desc, int world, int rank, void* const* flags, int free_row, int done_row,
                                    unsigned int epoch, void* const* inbox_slots, const void* inbox_local, int64_t rows_per_rank,
                                    void* counter_u32, void* out, const void* bias, void* status_i32, double timeout_s,
                                    void* stream, int split);

// First half of a split GEMM -> reduce-scatter: the GEMM whose epilogue delivers every row to its owner's inbox and which
// publishes "delivered" when done.  No CTA waits for another rank's result or for its own grid.  Follow it with a wait
// on (done_row, epoch) and bmt_gemm_rs_reduce.
extern "C" int bmt_gemm_reduce_scatter_main(const BmtGemmDesc* desc, int world, int rank, void* const* flags, int free_row, int done_row,
                                            unsigned int epoch, void* const* inbox_slots, const void* inbox_local,
                                            int64_t rows_per_rank, void* counter_u32, void* status_i32, double timeout_s, void* stream) {
    return gemm_reduce_scatter_impl(desc, world, rank, flags, free_row, done_row, epoch, inbox_slots, inbox_local, rows_per_rank,
                                    counter_u32, nullptr, nullptr, status_i32, timeout_s, stream, 1);
}

extern "C" int bmt_gemm_reduce_scatter(const BmtGemmDesc* desc, int world, int rank, void* const* flags, int free_row, int done_row,
                                       unsigned int epoch, void* const* inbox_slots, const void* inbox_local, int64_t rows_per_rank,
                                       void* counter_u32, void* out, const void* bias, void* status_i32, double timeout_s,
                                       void* stream) {
    return gemm_reduce_scatter_impl(desc, world, rank, flags, free_row, done_row, epoch, inbox_slots, inbox_local, rows_per_rank,
                                    counter_u32, out, bias, status_i32, timeout_s, stream, 0);
}

static int gemm_reduce_scatter_impl(const BmtGemmDesc* desc, int world, int rank, void* const* flags, int free_row, int done_row,
                                    unsigned int epoch, void* const* inbox_slots, const void* inbox_local, int64_t rows_per_rank,
                                    void* counter_u32, void* out, const void* bias, void* status_i32, double timeout_s,
                                    void* stream, int split) {
    if (world < 2 || world > 8 || desc->m != rows_per_rank * world) return -40;
    if (desc->n % 8 != 0) return -41;
    FusedComm f;
    memset(&f, 0, sizeof(f));
    f.rs_split = split;
    f.mode = 1; f.world = world; f.rank = rank; f.free_row = free_row; f.done_row = done_row; f.epoch = epoch;
    f.status = (int*)status_i32; f.limit_ns = (uint64_t)(timeout_s * 1e9);
    for (int j = 0; j < world; ++j) { f.flags[j] = (unsigned int*)flags[j]; f.rs_inbox[j] = inbox_slots[j]; }
    f.rs_inbox_local = inbox_local; f.rs_rows = rows_per_rank; f.rs_counter = (unsigned int*)counter_u32; f.rs_out = out;
    f.rs_bias = bias;
    BmtGemmDesc g = *desc;
    g.bias = nullptr; g.residual = nullptr; g.aux = nullptr; g.accumulate = 0; g.act = 0;
    g.batch_inner = g.batch_outer = g.b_inner_div = 1;
    g.c = (void*)inbox_local; g.ldc = desc->n; g.c_dtype = desc->ab_dtype;
    return launch_gemm(g, (cudaStream_t)stream, &f);
}

// Number of CTAs the fused GEMM -> reduce-scatter launches for this problem (its completion counter advances by that much).
extern "C" int bmt_gemm_rs_grid(int64_t m, int64_t n, int64_t k, int b_major) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return -1;
    const int sms = bmt::sm_count();
    const TileChoice tc = pick_tile(m, n, k, 1, b_major != 0, 0, 0, false, sms);
    const int64_t tiles = ((m + BM - 1) / BM) * ((n + tc.bn - 1) / tc.bn);
    return (int)(tiles < sms ? tiles : sms);
}

// all-gather -> GEMM over the rows of A (see FusedComm mode 2).  The gathered matrix (world * rows x K, pitch K) lives in
// `gathered[rank]`; desc->a must point at it and desc->m = world * rows.  rows must be a multiple of 128.
extern "C" int bmt_all_gather_gemm(const BmtGemmDesc* desc, int world, int rank, void* const* flags, int free_row,
                                   unsigned int epoch, const void* src, int64_t ld_src, int64_t rows, void* const* gathered,
                                   void* const* counters, int comm_ctas, int skip_local, void* status_i32, double timeout_s,
                                   void* stream) {
    if (world < 2 || world > 8 || desc->m != rows * world || rows % BM != 0 || desc->a_major != 0) return -42;
    if (desc->k % 8 != 0 || desc->lda != desc->k || ld_src != desc->k || ((uintptr_t)src & 15)) return -43;
    FusedComm f;
    memset(&f, 0, sizeof(f));
    f.mode = 2; f.world = world; f.rank = rank; f.free_row = free_row; f.epoch = epoch;
    f.status = (int*)status_i32; f.limit_ns = (uint64_t)(timeout_s * 1e9);
    for (int j = 0; j < world; ++j) { f.flags[j] = (unsigned int*)flags[j]; f.ag_dst[j] = gathered[j]; f.ag_count[j] = (unsigned int*)counters[j]; }
    f.ag_ctas = comm_ctas; f.ag_src = src; f.ag_ld_src = ld_src; f.ag_rows = rows; f.skip_local = skip_local;
    // a 128-row block has 256 * K bytes = 2048 * (K / 8): pieces of 2048 * d bytes with d the largest divisor of K / 8 up to 16
    int d = 16;
    while ((desc->k / 8) % d) --d;
    f.ag_piece_bytes = 2048 * d; f.ag_pieces_per_block = (int)(desc->k / 8) / d;
    // runs: enough of them to keep every pusher CTA busy, otherwise one per block
    int rpb = 1;
    while ((int64_t)(world - (skip_local ? 1 : 0)) * (rows / BM) * rpb < 2 * (int64_t)comm_ctas && f.ag_pieces_per_block % (rpb * 2) == 0) rpb *= 2;
    f.ag_runs_per_block = rpb;
    BmtGemmDesc g = *desc;
    g.batch_inner = g.batch_outer = g.b_inner_div = 1;
    return launch_gemm(g, (cudaStream_t)stream, &f);
}

// How many CTAs of a fused kernel should push instead of multiply: the kernel ends when both the math (on the remaining
// SMs) and the pushes are done, so pick the even count that balances the two.  Rates are rough measured figures: a pusher
// CTA moves about 14 GB/s, all pushers together at most about 550 GB/s to remote destinations, and the math runs at
// about 1.1 PFLOP/s on a full GPU.  push_bytes counts every destination (own copy included), remote_bytes the peers only.
extern "C" int bmt_fused_comm_ctas(double flops, double push_bytes, double remote_bytes) {
    static int sms = 0;
    if (sms == 0) {
        int dev = 0;
        if (cudaGetDevice(&dev) != cudaSuccess) return 16;
        if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms < 64) { sms = 0; return 16; }
    }
    int best = 8;
    double best_t = 1e30;
    for (int c = 8; c <= sms - 32; c += 4) {
        const double t_math = flops / (1.1e15 * (double)(sms - c) / (double)sms);
        double t_push = push_bytes / (c * 14e9);
        const double t_link = remote_bytes / 550e9;
        if (t_link > t_push) t_push = t_link;
        const double t = t_math > t_push ? t_math : t_push;
        if (t < best_t * 0.98) { best_t = t; best = c; }
    }
    return best;
}

static int zero_gather_split(int64_t n, int world, int comm_ctas);

// ZeRO weight gather -> GEMM (FusedComm mode 3).  desc->b points at the weight inside this rank's gathered buffer (N x K,
// rows contiguous, pitch K); this rank contributes the flat element range [first, first + count) of it, read from `src`.
// `expected` is a device array with the number of pieces every 128-row chunk receives from all ranks together
// (see bmt_zero_gather_expected).
extern "C" int bmt_zero_gather_gemm(const BmtGemmDesc* desc, int world, int rank, void* const* flags, int free_row,
                                    unsigned int epoch, const void* src, int64_t first, int64_t count, void* const* weight_on_rank,
                                    void* const* counters, const void* expected_u32, int comm_ctas, int skip_local,
                                    void* status_i32, double timeout_s, void* stream) {
    if (world < 2 || world > 8 || desc->b_major != 0 || desc->ldb != desc->k) return -44;
    if ((first & 7) || (count & 7) || ((uintptr_t)src & 15)) return -45;
    FusedComm f;
    memset(&f, 0, sizeof(f));
    f.mode = 3; f.world = world; f.rank = rank; f.free_row = free_row; f.epoch = epoch;
    f.status = (int*)status_i32; f.limit_ns = (uint64_t)(timeout_s * 1e9);
    for (int j = 0; j < world; ++j) { f.flags[j] = (unsigned int*)flags[j]; f.bg_dst[j] = weight_on_rank[j]; f.bg_cnt[j] = (unsigned int*)counters[j]; }
    f.ag_ctas = comm_ctas; f.bg_src = (const char*)src; f.bg_first = first; f.bg_count = count; f.skip_local = skip_local;
    f.bg_expected = (const unsigned int*)expected_u32;
    f.bg_split = zero_gather_split(desc->n, world, comm_ctas);
    BmtGemmDesc g = *desc;
    g.batch_inner = g.batch_outer = g.b_inner_div = 1;
    return launch_gemm(g, (cudaStream_t)stream, &f);
}

// Runs into which a rank's part of one chunk is cut: more when the weight has few chunks, so every pusher CTA has work.
static int zero_gather_split(int64_t n, int world, int comm_ctas) {
    const int64_t chunks = (n + BM - 1) / BM;
    int split = 1;
    while (chunks * world * split < 2 * (int64_t)comm_ctas && split < 8) split *= 2;
    return split;
}

// Host helper: counter bumps each 128-row chunk of an (n x k) weight receives when rank j owns the flat element range
// [first[j], first[j] + count[j]) and the kernel runs with `comm_ctas` pusher CTAs.  out has ceil(n / 128) entries.
extern "C" int bmt_zero_gather_expected(int64_t n, int64_t k, int world, const int64_t* first, const int64_t* count, int comm_ctas,
                                        unsigned int* out) {
    const int split = zero_gather_split(n, world, comm_ctas);
    const int64_t CK = (int64_t)BM * k;
    const int64_t chunks = (n + BM - 1) / BM;
    for (int64_t c = 0; c < chunks; ++c) out[c] = 0;
    for (int j = 0; j < world; ++j) {
        const int64_t lo_all = first[j], hi_all = first[j] + count[j];
        if (count[j] <= 0) continue;
        for (int64_t c = lo_all / CK; c * CK < hi_all && c < chunks; ++c) {
            const int64_t lo = lo_all > c * CK ? lo_all : c * CK;
            const int64_t hi = hi_all < (c + 1) * CK ? hi_all : (c + 1) * CK;
            const int64_t np = (hi - lo + BG_PIECE - 1) / BG_PIECE, per_run = (np + split - 1) / split;
            out[c] += (unsigned int)((np + per_run - 1) / per_run);
        }
    }
    return 0;
}

// Timing counters of the fused kernels launched on the current device since the last call (see g_fused_stats); the
// counters are cleared.  out: 8 values.  Synchronises with the device.
extern "C" int bmt_fused_stats(unsigned long long* out) {
    unsigned long long v[8], zero[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    if (cudaMemcpyFromSymbol(v, g_fused_stats, sizeof(v)) != cudaSuccess) return -1;
    if (cudaMemcpyToSymbol(g_fused_stats, zero, sizeof(zero)) != cudaSuccess) return -1;
    for (int i = 0; i < 8; ++i) out[i] = v[i];
    return 0;
}

// Status word of the GEMM kernels: 0, or (role << 16 | cta) of the first CTA whose bounded wait ran out.  Reading clears it.
extern "C" int bmt_gemm_status(void) {
    int v = 0, zero = 0;
    if (cudaMemcpyFromSymbol(&v, g_gemm_status, sizeof(int)) != cudaSuccess) return -1;
    if (v) cudaMemcpyToSymbol(g_gemm_status, &zero, sizeof(int));
    if (v && g_host_status) *g_host_status = 0;
    return v;
}

// The wait of a CTA for the sums of another, for a flag that the caller may or may not have set to 1: what a hand-over that fails does.
__global__ void gemm_wait_kernel(uint32_t* flag, int* host_status) {
    if (!wait_partials(flag, 0, 1, 1, (int)threadIdx.x) && threadIdx.x == 0) gave_up<false>(12, host_status);
}
extern "C" int bmt_gemm_wait(void* flag, void* stream) {
    if (const int rc = prepare_kernels()) return rc;
    gemm_wait_kernel<<<1, 32, 0, (cudaStream_t)stream>>>((uint32_t*)flag, g_host_status);
    return (int)cudaGetLastError();
}
