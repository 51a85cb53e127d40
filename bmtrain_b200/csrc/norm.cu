// LayerNorm / RMSNorm forward and backward for sm_100a.
//
// Forward: a team of warps per row, which holds it in registers and takes exact two-pass statistics over it.  Saves (mean, rstd) per row.
// Backward: persistent grids (at most nblk CTAs) that get whole rows as bulk copies through a ring in shared memory, produce dx
// and keep partial dgamma / dbeta in registers, written once to a (blocks x d) fp32 scratch that a second kernel folds.
// Both also exist with one CTA per row, staged in shared memory (BMT_NORM_STAGED=1, and the combinations the others do not take).
// (The reference calls F.layer_norm: example/layers/layernorm.py:29.)
#include <math.h>
#include <stdlib.h>
#include <type_traits>

#include "api.h"
#include "common.cuh"
#include "tcgen05.cuh"

namespace {

constexpr int NT = 256;
constexpr int MAXIT = 8;  // d <= NT * 8 * MAXIT = 16384

template <typename T>
__global__ void __launch_bounds__(NT) norm_fwd_kernel(int64_t rows, int d, const T* __restrict__ x, const T* __restrict__ w,
                                                      const T* __restrict__ b, float eps, int rms, T* __restrict__ y,
                                                      float* __restrict__ stats) {
    extern __shared__ float row[];
    __shared__ float scratch[33];
    const int64_t r = blockIdx.x;
    const T* __restrict__ xr = x + r * d;
    float s = 0.f;
    for (int c = threadIdx.x * 8; c < d; c += NT * 8) {
        bmt::Vec16<T> v = bmt::ld16(xr + c);
#pragma unroll
        for (int k = 0; k < 8; ++k) { float f = bmt::Cvt<T>::to_f(v.v[k]); row[c + k] = f; s += f; }
    }
    float mean = 0.f;
    if (!rms) mean = bmt::block_allreduce<false>(s, scratch) / d;
    float q = 0.f;
    for (int c = threadIdx.x * 8; c < d; c += NT * 8) {
#pragma unroll
        for (int k = 0; k < 8; ++k) { float f = row[c + k] - mean; q += f * f; }
    }
    const float var = bmt::block_allreduce<false>(q, scratch) / d;
    const float rstd = rsqrtf(var + eps);
    if (threadIdx.x == 0) { stats[r] = mean; stats[rows + r] = rstd; }
    T* __restrict__ yr = y + r * d;
    for (int c = threadIdx.x * 8; c < d; c += NT * 8) {
        bmt::Vec16<T> wv = bmt::ld16(w + c), o;
        bmt::Vec16<T> bv;
        if (b) bv = bmt::ld16(b + c);
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            float f = (row[c + k] - mean) * rstd * bmt::Cvt<T>::to_f(wv.v[k]);
            if (b) f += bmt::Cvt<T>::to_f(bv.v[k]);
            o.v[k] = bmt::Cvt<T>::from_f(f);
        }
        bmt::st16(yr + c, o);
    }
}

template <typename T>
__global__ void __launch_bounds__(NT) norm_bwd_kernel(int64_t rows, int d, const T* __restrict__ x, const T* __restrict__ dy,
                                                      const T* __restrict__ w, const float* __restrict__ stats, int rms,
                                                      T* __restrict__ dx, float* __restrict__ partial, const T* __restrict__ dres) {
    __shared__ float scratch[33];
    float dg[MAXIT][8], db[MAXIT][8];
#pragma unroll
    for (int it = 0; it < MAXIT; ++it)
#pragma unroll
        for (int k = 0; k < 8; ++k) dg[it][k] = db[it][k] = 0.f;

    for (int64_t r = blockIdx.x; r < rows; r += gridDim.x) {
        const float mean = stats[r], rstd = stats[rows + r];
        const T* __restrict__ xr = x + r * d;
        const T* __restrict__ gr = dy + r * d;
        float s1 = 0.f, s2 = 0.f;
#pragma unroll
        for (int it = 0; it < MAXIT; ++it) {
            const int c = threadIdx.x * 8 + it * NT * 8;
            if (c < d) {
                bmt::Vec16<T> xv = bmt::ld16(xr + c), gv = bmt::ld16(gr + c), wv = bmt::ld16(w + c);
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    const float xh = (bmt::Cvt<T>::to_f(xv.v[k]) - mean) * rstd;
                    const float g = bmt::Cvt<T>::to_f(gv.v[k]);
                    const float wg = g * bmt::Cvt<T>::to_f(wv.v[k]);
                    s1 += wg; s2 += wg * xh;
                    dg[it][k] += g * xh; db[it][k] += g;
                }
            }
        }
        if (rms) s1 = 0.f; else s1 = bmt::block_allreduce<false>(s1, scratch) / d;
        s2 = bmt::block_allreduce<false>(s2, scratch) / d;
        T* __restrict__ dr = dx + r * d;
#pragma unroll
        for (int it = 0; it < MAXIT; ++it) {
            const int c = threadIdx.x * 8 + it * NT * 8;
            if (c < d) {
                bmt::Vec16<T> xv = bmt::ld16(xr + c), gv = bmt::ld16(gr + c), wv = bmt::ld16(w + c), o, rv;
                if (dres) rv = bmt::ld16(dres + r * d + c);
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    const float xh = (bmt::Cvt<T>::to_f(xv.v[k]) - mean) * rstd;
                    const float wg = bmt::Cvt<T>::to_f(gv.v[k]) * bmt::Cvt<T>::to_f(wv.v[k]);
                    float val = rstd * (wg - s1 - xh * s2);
                    if (dres) val += bmt::Cvt<T>::to_f(rv.v[k]);
                    o.v[k] = bmt::Cvt<T>::from_f(val);
                }
                bmt::st16(dr + c, o);
            }
        }
    }
    float* pg = partial + (int64_t)blockIdx.x * d;
    float* pb = partial + ((int64_t)gridDim.x + blockIdx.x) * d;
#pragma unroll
    for (int it = 0; it < MAXIT; ++it) {
        const int c = threadIdx.x * 8 + it * NT * 8;
        if (c < d) {
#pragma unroll
            for (int k = 0; k < 8; ++k) { pg[c + k] = dg[it][k]; pb[c + k] = db[it][k]; }
        }
    }
}

// Fold the per-CTA partial sums: block = 32 columns x 32 row lanes, rows strided over the lanes, smem tree at the end.
template <typename T>
__global__ void __launch_bounds__(1024) norm_fold_kernel(int d, int nblk, const float* __restrict__ partial, T* __restrict__ dw, T* __restrict__ db) {
    bmt::after_previous();
    __shared__ float sa[32][33], sb[32][33];
    const int tx = threadIdx.x, ty = threadIdx.y;
    const int c = blockIdx.x * 32 + tx;
    float a = 0.f, bsum = 0.f;
    if (c < d) {
        for (int i = ty; i < nblk; i += 32) {
            a += partial[(int64_t)i * d + c];
            if (db) bsum += partial[((int64_t)nblk + i) * d + c];
        }
    }
    sa[ty][tx] = a; sb[ty][tx] = bsum;
    __syncthreads();
    if (ty == 0 && c < d) {
        float ra = 0.f, rb = 0.f;
#pragma unroll 8
        for (int l = 0; l < 32; ++l) { ra += sa[l][tx]; rb += sb[l][tx]; }
        dw[c] = bmt::Cvt<T>::from_f(ra);
        if (db) db[c] = bmt::Cvt<T>::from_f(rb);
    }
}

// Forward: a team of WPR warps has a row in its registers, a block one row or, if a warp is a team, four.  All loads are issued before
// the first use; statistics are exact two-pass sums over the registers.  Bytes bound it once little is issued for an element: values are
// worked on in pairs, blocks come and go instead of a resident grid striding over the rows with the next row's loads ahead of its
// arithmetic (which left an SM 16 warps, and issued 19 instructions for an element).  16384 x 5120 bf16, RMSNorm: 66 us with the
// resident grid, now 51 (6.6 TB/s); LayerNorm 85, now 54; 1024 x 2560 6.4, now 3.8.
constexpr int FWD_WARPS(int wpr) { return wpr == 1 ? 4 : wpr; }
template <typename T, int VPL, int WPR, bool RMS, bool EARLY>
__global__ void __launch_bounds__(FWD_WARPS(WPR) * 32) norm_fwd_row_kernel(int64_t rows, int d, const T* __restrict__ x, const T* __restrict__ w,
                                                                           const T* __restrict__ b, float eps, T* __restrict__ y,
                                                                           float* __restrict__ stats) {
    if (EARLY) bmt::after_previous();
    constexpr int RPC = FWD_WARPS(WPR) / WPR;          // 1, or 4 teams without a barrier
    __shared__ float ex[2][FWD_WARPS(WPR)];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int sub = warp % WPR, slot = warp / WPR;
    const int64_t r = (int64_t)blockIdx.x * RPC + slot;
    const bool live = r < rows;                        // the same for a team
    const int c0 = live ? (sub * 32 + lane) * 8 : d;   // the lane's vectors: columns c0 + i * WPR * 256 below d
    const auto team_sum = [&](float v, int which) {
        v = bmt::warp_sum(v);
        if (WPR == 1) return v;
        if (lane == 0) ex[which][warp] = v;
        __syncthreads();
        v = 0.f;
#pragma unroll
        for (int i = 0; i < WPR; ++i) v += ex[which][slot * WPR + i];
        return v;
    };
    const T* __restrict__ xr = x + r * d;
    bmt::Vec16<T> raw[VPL];
#pragma unroll
    for (int i = 0; i < VPL; ++i)
        if (c0 + i * WPR * 256 < d) raw[i] = bmt::ld16(xr + c0 + i * WPR * 256);
    // the sums add one value after another, in a fixed order: a mean that differs in its last bit moves roundings of the result, and with
    // them the signs of activations near zero
    uint64_t f[VPL][4];
    float sum = 0.f, mean = 0.f;
#pragma unroll
    for (int i = 0; i < VPL; ++i)
        if (c0 + i * WPR * 256 < d) {
            const uint32_t* u = reinterpret_cast<const uint32_t*>(raw[i].v);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                f[i][k] = bmt::to_f2<T>(u[k]);
                float lo, hi;
                bmt::unpack_f2(f[i][k], lo, hi);
                if (RMS) sum = fmaf(hi, hi, fmaf(lo, lo, sum));
                else { sum += lo; sum += hi; }
            }
        }
    if (!RMS) {
        mean = team_sum(sum, 0) / d;
        const uint64_t minus = bmt::pack_f2(-mean, -mean);
        sum = 0.f;
#pragma unroll
        for (int i = 0; i < VPL; ++i)
            if (c0 + i * WPR * 256 < d) {
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    f[i][k] = bmt::add_f2(f[i][k], minus);
                    float lo, hi;
                    bmt::unpack_f2(f[i][k], lo, hi);
                    sum = fmaf(hi, hi, fmaf(lo, lo, sum));
                }
            }
    }
    const float rstd = rsqrtf(team_sum(sum, 1) / d + eps);
    if (live && sub == 0 && lane == 0) { stats[r] = mean; stats[rows + r] = rstd; }
    const uint64_t by = bmt::pack_f2(rstd, rstd);
#pragma unroll
    for (int i = 0; i < VPL; ++i)
        if (const int c = c0 + i * WPR * 256; c < d) {
            const bmt::Vec16<T> wv = bmt::ld16(w + c);       // a few KB that every row reads: in L1
            bmt::Vec16<T> bv, o;
            if (b) bv = bmt::ld16(b + c);
            const uint32_t *uw = reinterpret_cast<const uint32_t*>(wv.v), *ub = reinterpret_cast<const uint32_t*>(bv.v);
            uint32_t* uo = reinterpret_cast<uint32_t*>(o.v);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const uint64_t t = bmt::mul_f2(f[i][k], by), m = bmt::to_f2<T>(uw[k]);
                uo[k] = bmt::from_f2<T>(b ? bmt::fma_f2(t, m, bmt::to_f2<T>(ub[k])) : bmt::mul_f2(t, m));
            }
            bmt::st16(y + r * d + c, o);
        }
}

// Many rows of one vector a lane are launched normally: a block of four lives for less than a microsecond, and waiting for the kernel before it takes
// as long (300000 x 256 RMSNorm 55 us so, 79 when launched early; 100000 x 64 18 and 27, 30000 x 128 alike; 100000 x 512, two vectors, 35 and 32).
template <typename T, int VPL, int WPR>
void launch_fwd_row(int64_t rows, int d, const void* x, const void* w, const void* b, float eps, int rms, void* y, void* stats, cudaStream_t s) {
    constexpr int RPC = FWD_WARPS(WPR) / WPR;
    const unsigned blocks = (unsigned)((rows + RPC - 1) / RPC);
    if (VPL > 1 || blocks <= 8192) {
        const auto kernel = rms ? norm_fwd_row_kernel<T, VPL, WPR, true, true> : norm_fwd_row_kernel<T, VPL, WPR, false, true>;
        bmt::launch(kernel, blocks, FWD_WARPS(WPR) * 32, 0, s, 1, rows, d, (const T*)x, (const T*)w, (const T*)b, eps, (T*)y, (float*)stats);
    } else if constexpr (VPL == 1) {
        const auto kernel = rms ? norm_fwd_row_kernel<T, VPL, WPR, true, false> : norm_fwd_row_kernel<T, VPL, WPR, false, false>;
        kernel<<<blocks, FWD_WARPS(WPR) * 32, 0, s>>>(rows, d, (const T*)x, (const T*)w, (const T*)b, eps, (T*)y, (float*)stats);
    }
}

// vpl: vectors a lane has to hold; wide teams have at least 5
template <typename T, int WPR, typename... Args>
void fwd_row(int vpl, Args... args) {
    if constexpr (WPR == 1) {
        if (vpl <= 1) return launch_fwd_row<T, 1, WPR>(args...);
        if (vpl == 2) return launch_fwd_row<T, 2, WPR>(args...);
        if (vpl == 3) return launch_fwd_row<T, 3, WPR>(args...);
        if (vpl == 4) return launch_fwd_row<T, 4, WPR>(args...);
    }
    if (vpl <= 5) launch_fwd_row<T, 5, WPR>(args...);
    else if (vpl == 6) launch_fwd_row<T, 6, WPR>(args...);
    else if (vpl == 7) launch_fwd_row<T, 7, WPR>(args...);
    else launch_fwd_row<T, 8, WPR>(args...);
}

template <typename T>
int fwd(int64_t rows, int64_t d, const void* x, const void* w, const void* b, float eps, int rms, void* y, void* stats, cudaStream_t s) {
    static const bool staged = [] { const char* e = getenv("BMT_NORM_STAGED"); return e && atoi(e) == 1; }();
    if (!staged && d <= 16384) {
        // the smallest team with at most 8 vectors a lane
        const int wpr = d <= 2048 ? 1 : d <= 4096 ? 2 : d <= 8192 ? 4 : 8, vpl = (int)((d + 256 * wpr - 1) / (256 * wpr));
        const auto run = [&](auto team) { fwd_row<T, decltype(team)::value>(vpl, rows, (int)d, x, w, b, eps, rms, y, stats, s); };
        if (wpr == 1) run(std::integral_constant<int, 1>());
        else if (wpr == 2) run(std::integral_constant<int, 2>());
        else if (wpr == 4) run(std::integral_constant<int, 4>());
        else run(std::integral_constant<int, 8>());
        bmt_count_launch(1);
        return (int)cudaGetLastError();
    }
    norm_fwd_kernel<T><<<(unsigned)rows, NT, d * sizeof(float), s>>>(rows, (int)d, (const T*)x, (const T*)w, (const T*)b, eps, rms, (T*)y, (float*)stats);
    bmt_count_launch(1);
    return (int)cudaGetLastError();
}

// Backward: a team of WPR warps per row, every lane owns fixed columns (VPL vectors of 8).  The per-column sums of dy * xhat
// and dy accumulate in registers over all rows a lane sees; they are combined once per CTA through shared memory into the
// scratch that norm_fold_kernel reduces.
// HBM bytes bound it (x, dy and the residual's gradient in, dx out), so what counts is bytes in flight.  Loading a row into
// registers and then working on it ran at 0.41 of the copy rate (16384 x 5120 RMS 193 us), one row ahead in registers at 0.48
// (160 us): a load takes longer than a row's arithmetic.  So whole rows come as bulk copies into a ring of up to BWD_STAGES
// stages in shared memory, refilled by one thread right behind the barrier that every row has anyway; the rows' statistics
// are fetched for BWD_BATCH rows at a time: 124 us (LayerNorm 194 -> 171).  Then the instructions bound it, 33 for an element: columns
// are worked on in pairs, the stage to refill is carried along instead of found by a 64-bit division in the thread that all others
// wait for, and LayerNorm too has three vectors a lane (it reads the row from shared memory twice): 89 us, LayerNorm 98.
// RMSNorm (RMS) has no bias and drops the second accumulator.
constexpr int BWD_STAGES = 8, BWD_BATCH = 32;
__device__ int g_norm_status = 0;   // 0, or (1 << 16) | blockIdx.x of the first CTA whose wait for a bulk copy ran out

template <int WPR> struct BwdTeam {
    static constexpr int THREADS = WPR == 16 ? 512 : 256, CTAS = WPR == 16 ? 1 : 2, RPC = THREADS / 32 / WPR;
};

__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(dst), "l"(src), "r"(bytes), "r"(bar) : "memory");
}

template <typename T, int VPL, int WPR, bool RMS>
__global__ void __launch_bounds__(BwdTeam<WPR>::THREADS, BwdTeam<WPR>::CTAS)
norm_bwd_stream_kernel(int64_t rows, int d, int stages, const T* __restrict__ x, const T* __restrict__ dy, const T* __restrict__ w,
                       const float* __restrict__ stats, T* __restrict__ dx, float* __restrict__ partial, const T* __restrict__ dres) {
    bmt::after_previous();
    constexpr int RPC = BwdTeam<WPR>::RPC, WARPS = BwdTeam<WPR>::THREADS / 32;
    constexpr bool AGAIN = VPL > (RMS ? 3 : 2);        // a row is read from shared memory again: no registers for it
    extern __shared__ __align__(128) uint8_t ring[];   // stages x {x, dy[, dres]} x RPC rows; 2 * d floats at the end of the kernel
    __shared__ __align__(8) uint64_t full[BWD_STAGES];
    __shared__ int late[2];                            // by parity of the row: a thread's wait for its copy ran out
    __shared__ float ex[2][2][WARPS], mu[BWD_BATCH * RPC], rs[BWD_BATCH * RPC];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int sub = warp % WPR, slot = warp / WPR;
    const uint32_t part_bytes = (uint32_t)(RPC * d * 2), stage_bytes = part_bytes * (dres ? 3 : 2);
    const int64_t groups = (rows + RPC - 1) / RPC;
    const int64_t n_it = (int64_t)blockIdx.x < groups ? (groups - 1 - blockIdx.x) / gridDim.x + 1 : 0;
    auto refill = [&](int64_t it, int st) {            // one thread: the rows of iteration `it` into stage it % stages
        const int64_t r0 = (blockIdx.x + it * gridDim.x) * RPC;
        const uint32_t bytes = (uint32_t)((rows - r0 < RPC ? rows - r0 : RPC) * d * 2);
        const uint32_t bar = bmt_tc::smem_u32(&full[st]), dst = bmt_tc::smem_u32(ring) + st * stage_bytes;
        bmt_tc::mbar_expect_tx_u32(bar, bytes * (dres ? 3u : 2u));
        bulk_load(dst, x + r0 * d, bytes, bar);
        bulk_load(dst + part_bytes, dy + r0 * d, bytes, bar);
        if (dres) bulk_load(dst + 2 * part_bytes, dres + r0 * d, bytes, bar);
    };
    if (threadIdx.x == 0) {
        for (int i = 0; i < stages; ++i) bmt_tc::mbar_init(&full[i], 1);
        bmt_tc::fence_barrier_init();
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        for (int it = 0; it < stages && it < n_it; ++it) refill(it, it);
        late[0] = late[1] = 0;
    }
    uint64_t dg[VPL][4], db[RMS ? 1 : VPL][4];         // pairs of columns
    bmt::Vec16<T> wv[VPL];
#pragma unroll
    for (int v = 0; v < VPL; ++v) {
        const int c = ((v * WPR + sub) * 32 + lane) * 8;
#pragma unroll
        for (int k = 0; k < 4; ++k) { dg[v][k] = 0; if (!RMS) db[v][k] = 0; }
        if (c < d) wv[v] = bmt::ld16(w + c);
    }
    __syncthreads();
    int st = 0;
    uint32_t phase = 0;
    bool failed = false;                               // the same in all threads
    for (int64_t it = 0; it < n_it; ++it) {
        const int64_t r = (blockIdx.x + it * gridDim.x) * RPC + slot;
        const bool live = r < rows;
        if (it % BWD_BATCH == 0) {
            __syncthreads();                           // the previous batch has been read
            for (int i = threadIdx.x; i < BWD_BATCH * RPC; i += BwdTeam<WPR>::THREADS) {
                const int64_t rr = (blockIdx.x + (it + i / RPC) * gridDim.x) * RPC + i % RPC;
                mu[i] = rr < rows && !RMS ? stats[rr] : 0.f;
                rs[i] = rr < rows ? stats[rows + rr] : 0.f;
            }
            __syncthreads();
        }
        const float mean = mu[(it % BWD_BATCH) * RPC + slot], rstd = rs[(it % BWD_BATCH) * RPC + slot];
        if (!bmt_tc::mbar_wait(&full[st], phase)) late[it & 1] = 1;   // bounded
        const T* xs = reinterpret_cast<const T*>(ring + st * stage_bytes) + slot * d;
        const T* gs = reinterpret_cast<const T*>(ring + st * stage_bytes + part_bytes) + slot * d;
        bmt::Vec16<T> xv[VPL], gv[VPL];
        const uint64_t by = bmt::pack_f2(rstd, rstd), minus = bmt::pack_f2(-mean, -mean);
        const auto xhat = [&](uint32_t u) {
            const uint64_t f = bmt::to_f2<T>(u);
            return bmt::mul_f2(RMS ? f : bmt::add_f2(f, minus), by);
        };
        const auto words = [](const bmt::Vec16<T>& v) { return reinterpret_cast<const uint32_t*>(v.v); };
        uint64_t t1 = 0, t2 = 0;
#pragma unroll
        for (int v = 0; v < VPL; ++v) {
            const int c = ((v * WPR + sub) * 32 + lane) * 8;
            if (live && c < d) {
                xv[v] = bmt::ld16(xs + c);
                gv[v] = bmt::ld16(gs + c);
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const uint64_t xh = xhat(words(xv[v])[k]), g = bmt::to_f2<T>(words(gv[v])[k]);
                    const uint64_t wg = bmt::mul_f2(g, bmt::to_f2<T>(words(wv[v])[k]));
                    if (!RMS) t1 = bmt::add_f2(t1, wg);
                    t2 = bmt::fma_f2(wg, xh, t2);
                    dg[v][k] = bmt::fma_f2(g, xh, dg[v][k]);
                    if (!RMS) db[v][k] = bmt::add_f2(db[v][k], g);
                }
            }
        }
        float s1 = bmt::sum_f2(t1), s2 = bmt::sum_f2(t2);
        if (!RMS) s1 = bmt::warp_sum(s1);
        s2 = bmt::warp_sum(s2);
        const int par = (int)(it & 1);
        if (WPR > 1 && lane == 0) { ex[par][0][warp] = s1; ex[par][1][warp] = s2; }
        __syncthreads();
        failed = late[par] != 0;                       // not written again before all have passed the next row's barrier
        if (failed) break;
        // every warp is through with the previous row: its stage takes the row `stages - 1` ahead of this one
        if (threadIdx.x == 0 && it > 0 && it - 1 + stages < n_it) refill(it - 1 + stages, st == 0 ? stages - 1 : st - 1);
        if (WPR > 1) {
            s1 = s2 = 0.f;
#pragma unroll
            for (int i = 0; i < WPR; ++i) { if (!RMS) s1 += ex[par][0][slot * WPR + i]; s2 += ex[par][1][slot * WPR + i]; }
        }
        s1 = s1 / d;
        s2 = s2 / d;
        const uint64_t less1 = bmt::pack_f2(-s1, -s1), less2 = bmt::pack_f2(-s2, -s2);
        const T* ds = reinterpret_cast<const T*>(ring + st * stage_bytes + 2 * part_bytes) + slot * d;
#pragma unroll
        for (int v = 0; v < VPL; ++v) {
            const int c = ((v * WPR + sub) * 32 + lane) * 8;
            if (live && c < d) {
                bmt::Vec16<T> o, rv;
                if (dres) rv = bmt::ld16(ds + c);
                const bmt::Vec16<T> xc = AGAIN ? bmt::ld16(xs + c) : xv[v], gc = AGAIN ? bmt::ld16(gs + c) : gv[v];
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const uint64_t xh = xhat(words(xc)[k]), g = bmt::to_f2<T>(words(gc)[k]), m = bmt::to_f2<T>(words(wv[v])[k]);
                    const uint64_t t = bmt::fma_f2(xh, less2, RMS ? bmt::mul_f2(g, m) : bmt::fma_f2(g, m, less1));
                    reinterpret_cast<uint32_t*>(o.v)[k] = bmt::from_f2<T>(dres ? bmt::fma_f2(t, by, bmt::to_f2<T>(words(rv)[k])) : bmt::mul_f2(t, by));
                }
                bmt::st16(dx + r * d + c, o);
            }
        }
        if (++st == stages) { st = 0; phase ^= 1; }
    }
    if (failed) {
        // a copy did not arrive: report it, give those in flight time to land before the ring is used again, and let the column sums
        // say that they are none
        if (threadIdx.x == 0) atomicCAS(&g_norm_status, 0, (1 << 16) | (int)(blockIdx.x & 0xffff));
        const uint64_t t0 = bmt_tc::global_ns();
        while (bmt_tc::global_ns() - t0 < 2000000ull) __nanosleep(1000);
        __syncthreads();
#pragma unroll
        for (int v = 0; v < VPL; ++v)
#pragma unroll
            for (int k = 0; k < 4; ++k) { dg[v][k] = bmt::pack_f2(NAN, NAN); if (!RMS) db[v][k] = bmt::pack_f2(NAN, NAN); }
    }
    // combine the RPC row slots of this CTA (slot 0 ends up with the CTA's column sums); every copy into the ring has landed
    float* fold = reinterpret_cast<float*>(ring);
    float* pg = partial + (int64_t)blockIdx.x * d;
    float* pb = partial + ((int64_t)gridDim.x + blockIdx.x) * d;
    for (int s_ = 1; s_ < RPC; ++s_) {
        __syncthreads();
        if (slot == s_) {
#pragma unroll
            for (int v = 0; v < VPL; ++v) {
                const int c = ((v * WPR + sub) * 32 + lane) * 8;
                if (c < d) {
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        reinterpret_cast<uint64_t*>(fold + c)[k] = dg[v][k];
                        if (!RMS) reinterpret_cast<uint64_t*>(fold + d + c)[k] = db[v][k];
                    }
                }
            }
        }
        __syncthreads();
        if (slot == 0) {
#pragma unroll
            for (int v = 0; v < VPL; ++v) {
                const int c = ((v * WPR + sub) * 32 + lane) * 8;
                if (c < d) {
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        dg[v][k] = bmt::add_f2(dg[v][k], reinterpret_cast<const uint64_t*>(fold + c)[k]);
                        if (!RMS) db[v][k] = bmt::add_f2(db[v][k], reinterpret_cast<const uint64_t*>(fold + d + c)[k]);
                    }
                }
            }
        }
    }
    if (slot == 0) {
#pragma unroll
        for (int v = 0; v < VPL; ++v) {
            const int c = ((v * WPR + sub) * 32 + lane) * 8;
            if (c < d) {
#pragma unroll
                for (int k = 0; k < 4; k += 2) {
                    *reinterpret_cast<ulonglong2*>(pg + c + 2 * k) = make_ulonglong2(dg[v][k], dg[v][k + 1]);
                    if (!RMS) *reinterpret_cast<ulonglong2*>(pb + c + 2 * k) = make_ulonglong2(db[v][k], db[v][k + 1]);
                }
            }
        }
    }
}

// Returns the number of CTAs (rows of partial sums per accumulator) that were launched, or a negative code.
template <typename T, int VPL, int WPR>
int launch_bwd_stream(int64_t rows, int d, const void* x, const void* dy, const void* w, const void* stats, int rms, int nblk, void* dx,
                      void* partial, const void* dres, cudaStream_t s) {
    using Team = BwdTeam<WPR>;
    // the ring: as many stages as fit the CTA's share of the shared memory; at least two (16384 columns with a residual: 192 KiB)
    const size_t budget = (size_t)(Team::CTAS == 1 ? 208 : 100) * 1024, stage = (size_t)Team::RPC * d * 2 * (dres ? 3 : 2);
    int stages = (int)(budget / stage);
    if (stages > BWD_STAGES) stages = BWD_STAGES;
    size_t smem = stages * stage;
    if (Team::RPC > 1 && smem < (size_t)2 * d * sizeof(float)) smem = (size_t)2 * d * sizeof(float);
    int64_t grid = (rows + Team::RPC - 1) / Team::RPC;
    if (grid > (int64_t)bmt::sm_count() * Team::CTAS) grid = (int64_t)bmt::sm_count() * Team::CTAS;
    if (grid > nblk) grid = nblk;
    const auto run = [&](auto kernel) {
        if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)budget) != cudaSuccess) return -30;
        kernel<<<(unsigned)grid, Team::THREADS, smem, s>>>(rows, d, stages, (const T*)x, (const T*)dy, (const T*)w, (const float*)stats, (T*)dx,
                                                           (float*)partial, (const T*)dres);
        return (int)grid;
    };
    return rms ? run(norm_bwd_stream_kernel<T, VPL, WPR, true>) : run(norm_bwd_stream_kernel<T, VPL, WPR, false>);
}

template <typename T, int WPR, typename... Args>
int bwd_stream_vpl(int vpl, Args... args) {
    if (vpl <= 1) return launch_bwd_stream<T, 1, WPR>(args...);
    if (vpl == 2) return launch_bwd_stream<T, 2, WPR>(args...);
    if constexpr (WPR == 16) if (vpl > 3) return launch_bwd_stream<T, 4, WPR>(args...);
    return launch_bwd_stream<T, 3, WPR>(args...);
}

template <typename T>
int bwd(int64_t rows, int64_t d, const void* x, const void* dy, const void* w, const void* stats, int rms, int nblk, void* dx,
        void* partial, void* dw, void* db, cudaStream_t s, const void* dres = nullptr, int* left = nullptr) {
    // `left`: the sums are left in `partial`, as so many rows of them
    const auto fold = [&](int blocks) {
        if (left) { *left = blocks; return; }
        const unsigned g = (unsigned)((d + 31) / 32);
        bmt::launch(norm_fold_kernel<T>, g, dim3(32, 32), 0, s, 1, (int)d, blocks, (const float*)partial, (T*)dw, (T*)db);
    };
    static const bool use_reg = [] { const char* e = getenv("BMT_NORM_STAGED"); return !(e && atoi(e) == 1); }();
    if (use_reg && d <= 16384 && !(rms && db)) {
        // the narrowest team with at most 3 vectors a lane (16384 x 5120: RMSNorm 118 us with 2 at most, 89 with 3; LayerNorm 132 and 98;
        // 4 or 5 gain nothing more); above 12288 columns the widest team
        const int64_t nv = (d + 255) / 256, most = 3;   // nv: vectors a lane of one warp would have
        const int wpr = nv <= most ? 1 : nv <= 2 * most ? 2 : nv <= 4 * most ? 4 : nv <= 8 * most ? 8 : 16;
        const int vpl = (int)((nv + wpr - 1) / wpr);
        const int blocks = wpr == 1 ? bwd_stream_vpl<T, 1>(vpl, rows, (int)d, x, dy, w, stats, rms, nblk, dx, partial, dres, s)
                         : wpr == 2 ? bwd_stream_vpl<T, 2>(vpl, rows, (int)d, x, dy, w, stats, rms, nblk, dx, partial, dres, s)
                         : wpr == 4 ? bwd_stream_vpl<T, 4>(vpl, rows, (int)d, x, dy, w, stats, rms, nblk, dx, partial, dres, s)
                         : wpr == 8 ? bwd_stream_vpl<T, 8>(vpl, rows, (int)d, x, dy, w, stats, rms, nblk, dx, partial, dres, s)
                                    : bwd_stream_vpl<T, 16>(vpl, rows, (int)d, x, dy, w, stats, rms, nblk, dx, partial, dres, s);
        if (blocks < 0) return blocks;
        fold(blocks);
        bmt_count_launch(left ? 1 : 2);
        return (int)cudaGetLastError();
    }
    norm_bwd_kernel<T><<<nblk, NT, 0, s>>>(rows, (int)d, (const T*)x, (const T*)dy, (const T*)w, (const float*)stats, rms, (T*)dx, (float*)partial, (const T*)dres);
    fold(nblk);
    bmt_count_launch(left ? 1 : 2);
    return (int)cudaGetLastError();
}

}  // namespace

extern "C" int bmt_norm_fwd(int64_t rows, int64_t d, const void* x, const void* w, const void* b, float eps, int rms, int dtype,
                            void* y, void* stats, void* stream) {
    if (rows <= 0) return 0;
    if (d % 8 != 0 || d > 16384 || dtype == BMT_DT_F32) return -3;
    cudaStream_t s = (cudaStream_t)stream;
    return dtype == BMT_DT_F16 ? fwd<__half>(rows, d, x, w, b, eps, rms, y, stats, s)
                               : fwd<__nv_bfloat16>(rows, d, x, w, b, eps, rms, y, stats, s);
}

extern "C" int bmt_norm_bwd(int64_t rows, int64_t d, const void* x, const void* dy, const void* w, const void* stats, int rms,
                            int dtype, int nblk, void* dx, void* partial, void* dw, void* db, void* stream) {
    if (rows <= 0) return 0;
    if (d % 8 != 0 || d > NT * 8 * MAXIT || dtype == BMT_DT_F32) return -3;
    cudaStream_t s = (cudaStream_t)stream;
    return dtype == BMT_DT_F16 ? bwd<__half>(rows, d, x, dy, w, stats, rms, nblk, dx, partial, dw, db, s)
                               : bwd<__nv_bfloat16>(rows, d, x, dy, w, stats, rms, nblk, dx, partial, dw, db, s);
}

// Backward that also adds a residual-branch gradient: dx = dres + norm_backward(dy).
extern "C" int bmt_norm_bwd_res(int64_t rows, int64_t d, const void* x, const void* dy, const void* w, const void* stats, int rms,
                                int dtype, int nblk, void* dx, void* partial, void* dw, void* db, const void* dres, void* stream) {
    if (rows <= 0) return 0;
    if (d % 8 != 0 || d > NT * 8 * MAXIT || dtype == BMT_DT_F32) return -3;
    cudaStream_t s = (cudaStream_t)stream;
    return dtype == BMT_DT_F16 ? bwd<__half>(rows, d, x, dy, w, stats, rms, nblk, dx, partial, dw, db, s, dres)
                               : bwd<__nv_bfloat16>(rows, d, x, dy, w, stats, rms, nblk, dx, partial, dw, db, s, dres);
}

extern "C" int bmt_norm_bwd_partial(int64_t rows, int64_t d, const void* x, const void* dy, const void* w, const void* stats, int rms, int dtype,
                                    int nblk, void* dx, void* partial, const void* dres, int* blocks, void* stream) {
    *blocks = 0;
    if (rows <= 0) return 0;
    if (d % 8 != 0 || d > NT * 8 * MAXIT || dtype == BMT_DT_F32) return -3;
    cudaStream_t s = (cudaStream_t)stream;
    return dtype == BMT_DT_F16 ? bwd<__half>(rows, d, x, dy, w, stats, rms, nblk, dx, partial, nullptr, nullptr, s, dres, blocks)
                               : bwd<__nv_bfloat16>(rows, d, x, dy, w, stats, rms, nblk, dx, partial, nullptr, nullptr, s, dres, blocks);
}

// status of the norm backward: 0, or (1 << 16 | CTA) of the first CTA that gave up waiting for its rows; reading clears it
extern "C" int bmt_norm_status(void) {
    int v = 0, zero = 0;
    if (cudaMemcpyFromSymbol(&v, g_norm_status, sizeof(int)) != cudaSuccess) return -1;
    if (v != 0) cudaMemcpyToSymbol(g_norm_status, &zero, sizeof(int));
    return v;
}

// ---------------------------------------------------------------------------------------------------------------
// Allocation-free variant (see norm_noalloc.h).  Same kernels as bmt_norm_bwd; the partial-sum scratch lives in a
// file-scope device array whose address is resolved once per device.
#include <mutex>
#include <stdio.h>

#include "norm_noalloc.h"

static __device__ __align__(256) float g_norm_noalloc_scratch[2 * BMT_NORM_NOALLOC_MAX_CTAS * BMT_NORM_NOALLOC_MAX_D];

namespace {
constexpr int kMaxDevices = 64;
float* g_noalloc_ptr[kMaxDevices] = {nullptr};
std::mutex g_noalloc_mu;

// Device address of the scratch array on the current device.  In host code the array's name is only a handle for
// the runtime, not a device address, so it is never passed to a kernel directly.
int noalloc_scratch(float** out) {
    int dev = 0;
    BMT_CUDA_OK(cudaGetDevice(&dev));
    if (dev < 0 || dev >= kMaxDevices) return BMT_NORM_NOALLOC_BAD_ARG;
    std::lock_guard<std::mutex> lk(g_noalloc_mu);
    if (g_noalloc_ptr[dev] == nullptr) {
        float* p = nullptr;
        BMT_CUDA_OK(cudaGetSymbolAddress((void**)&p, g_norm_noalloc_scratch));
        g_noalloc_ptr[dev] = p;
    }
    *out = g_noalloc_ptr[dev];
    return 0;
}
}  // namespace

extern "C" int bmt_norm_bwd_noalloc(int64_t rows, int64_t d, const void* x, const void* dy, const void* w, const void* stats,
                                    int rms, int dtype, void* dx, void* dw, void* db, void* stream) {
    if (rows <= 0) return 0;
    if (d > BMT_NORM_NOALLOC_MAX_D) {
        fprintf(stderr, "bmt_norm_bwd_noalloc: d = %lld exceeds the built-in scratch (max d %d); use bmt_norm_bwd with your own scratch\n",
                (long long)d, BMT_NORM_NOALLOC_MAX_D);
        return BMT_NORM_NOALLOC_TOO_LARGE;
    }
    if (d <= 0 || d % 8 != 0 || (dtype != BMT_DT_F16 && dtype != BMT_DT_BF16) || (rms && db != nullptr)) {
        fprintf(stderr, "bmt_norm_bwd_noalloc: unsupported arguments (d = %lld must be a positive multiple of 8, dtype fp16/bf16, no bias gradient for RMSNorm)\n",
                (long long)d);
        return BMT_NORM_NOALLOC_BAD_ARG;
    }
    float* scratch = nullptr;
    const int rc = noalloc_scratch(&scratch);
    if (rc != 0) return rc;
    const int nblk = rows < BMT_NORM_NOALLOC_MAX_CTAS ? (int)rows : BMT_NORM_NOALLOC_MAX_CTAS;
    cudaStream_t s = (cudaStream_t)stream;
    return dtype == BMT_DT_F16 ? bwd<__half>(rows, d, x, dy, w, stats, rms, nblk, dx, scratch, dw, db, s)
                               : bwd<__nv_bfloat16>(rows, d, x, dy, w, stats, rms, nblk, dx, scratch, dw, db, s);
}
