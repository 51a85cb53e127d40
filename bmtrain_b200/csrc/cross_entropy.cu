// Cross-entropy for sm_100a: single-pass (online softmax) row statistics and a recomputing backward.
//
// bmt_ce_row_stats: per row i of logits (m x n) -> max_i, sum_j exp(x_ij - max_i), x[i, target_i - vocab_start]
//                   (0 when the target is outside [vocab_start, vocab_start + n)).  One read of the logits.
// bmt_ce_backward : out_ij = (exp(x_ij - lse_i) - [j == target_i - vocab_start]) * grad_i, 0 for ignored rows.
// The reference (csrc/cuda/cross_entropy.cu:9-199) makes three strided passes per row and stores the whole softmax.
#include "api.h"
#include "common.cuh"

#include <type_traits>

namespace {

// 2^x on the special-function unit (one instruction; the C library's exp2f adds range handling around it)
__device__ __forceinline__ float ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// Logits are multiplied by log2(e) before the exponent is taken.  The lowest finite numbers of fp32 and bf16, which classes
// are hidden with, overflow in that product: as a reference it is kept finite, so that they count for nothing beside others.
constexpr float LOWEST = -3.402823466e38f;

// Elements of a row before its first 16-byte boundary.
template <typename T> __device__ __forceinline__ int64_t row_head(const T* row, int64_t n) {
    const int64_t h = ((16 - ((uintptr_t)row & 15)) & 15) / sizeof(T);
    return h < n ? h : n;
}

template <typename T>
__global__ void __launch_bounds__(256) ce_row_stats_kernel(int64_t m, int64_t n, const T* __restrict__ x,
                                                           const int64_t* __restrict__ target, int64_t vocab_start,
                                                           float* __restrict__ out) {
    __shared__ float scratch[33];
    const int64_t row = blockIdx.x;
    const T* __restrict__ xr = x + row * n;
    constexpr int V = bmt::Vec16<T>::N;
    // mx: largest logit so far; se: sum of 2^(x * log2e - ref) with ref = mx * log2e as it is rounded.  Taking the rounded product
    // as the reference keeps the exponent exact to one rounding of the FMA; its distance from mx * log2e is made up for once, at
    // the end.
    float mx = -INFINITY, ref = 0.f, se = 0.f;
    // Rows of an odd number of classes start anywhere: the few elements before the first 16-byte boundary and behind the last
    // whole vector go one by one, the rest as vectors (4096 x 50257 bf16 element by element: 242 us forward, 356 us backward;
    // 104 and 141 us so).
    // U vectors per thread and trip: all loads are issued before the first use, the running maximum moves at most
    // once per trip, and every element costs one FMA and one ex2
    constexpr int U = 4;
    constexpr float L2E = 1.4426950408889634f;
    const int64_t head = row_head<T>(xr, n), nv = (n - head) / V, tail = head + nv * V;
    const T* __restrict__ xv = xr + head;
    const auto move_to = [&](float v) {
        if (!(v > mx)) return;
        const float r = fmaxf(v * L2E, LOWEST);
        if (mx != -INFINITY) se *= ex2(ref - r);
        mx = v;
        ref = r;
    };
    for (int64_t i = threadIdx.x; i < head + n - tail; i += blockDim.x) {
        const float f = bmt::Cvt<T>::to_f(xr[i < head ? i : tail + i - head]);
        move_to(f);
        se += ex2(fmaf(f, L2E, -ref));       // ref is 0 as long as all classes are hidden (-inf): they add nothing
    }
    for (int64_t i0 = threadIdx.x; i0 < nv; i0 += (int64_t)blockDim.x * U) {
        bmt::Vec16<T> v[U];
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (i0 + (int64_t)u * blockDim.x < nv) v[u] = bmt::ld16(xv + (i0 + (int64_t)u * blockDim.x) * V);
        float lm = -INFINITY;
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (i0 + (int64_t)u * blockDim.x < nv) {
#pragma unroll
                for (int k = 0; k < V; ++k) lm = fmaxf(lm, bmt::Cvt<T>::to_f(v[u].v[k]));
            }
        move_to(lm);
        const float off = -ref;
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (i0 + (int64_t)u * blockDim.x < nv) {
#pragma unroll
                for (int k = 0; k < V; ++k) se += ex2(fmaf(bmt::Cvt<T>::to_f(v[u].v[k]), L2E, off));
            }
    }
    const float gmx = bmt::block_allreduce<true>(mx, scratch);
    const float contrib = se == 0.f ? 0.f : se * ex2(-fmaf(gmx, L2E, -ref));   // zero: no class that counts (a NaN is not lost)
    const float gse = bmt::block_allreduce<false>(contrib, scratch);
    if (threadIdx.x == 0) {
        const int64_t t = target[row] - vocab_start;
        out[row] = gmx;
        out[m + row] = gse;
        out[2 * m + row] = (t >= 0 && t < n) ? bmt::Cvt<T>::to_f(xr[t]) : 0.f;
    }
}

// Largest of the 8 values of a packet, found on packed pairs (no conversion to fp32 per element, so the compiler has no
// reason to keep 8 converted values per packet alive between the maximum pass and the exponent pass).
__device__ __forceinline__ float packet_max(const bmt::Vec16<__half>& v) {
    const __half2* h = reinterpret_cast<const __half2*>(v.v);
    const __half2 m = __hmax2(__hmax2(h[0], h[1]), __hmax2(h[2], h[3]));
    return __half2float(__hmax(__low2half(m), __high2half(m)));
}
__device__ __forceinline__ float packet_max(const bmt::Vec16<__nv_bfloat16>& v) {
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(v.v);
    const __nv_bfloat162 m = __hmax2(__hmax2(h[0], h[1]), __hmax2(h[2], h[3]));
    return __bfloat162float(__hmax(__low2bfloat16(m), __high2bfloat16(m)));
}

// (max, sum of exp relative to max) pairs combine associatively
__device__ __forceinline__ void lse_combine(float& m, float& s, float m2, float s2) {
    constexpr float L2E = 1.4426950408889634f;
    const float nm = fmaxf(m, m2);
    const float a = s == 0.f ? 0.f : s * ex2((m - nm) * L2E);       // zero: no class that counts yet
    const float b = s2 == 0.f ? 0.f : s2 * ex2((m2 - nm) * L2E);
    m = nm;
    s = a + b;
}

// Streaming form for rows of 16-byte vectors: a persistent grid walks over (row, trip) chunks of 256 * U vectors; the
// loads of the next chunk are issued before the arithmetic on the current one, so every thread has U loads in flight all
// the time.  One barrier per row: warps leave their (max, sum) pair in one of two alternating slot sets and thread 0
// combines them.
template <typename T, int U>
__global__ void __launch_bounds__(256) ce_row_stats_stream_kernel(int64_t m, int64_t n, int trips, const T* __restrict__ x,
                                                                  const int64_t* __restrict__ target, int64_t vocab_start,
                                                                  float* __restrict__ out) {
    bmt::after_previous();
    constexpr int V = bmt::Vec16<T>::N;
    constexpr float L2E = 1.4426950408889634f;
    __shared__ float sm_m[2][8], sm_s[2][8];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t nv = n / V;
    const int64_t my_rows = (int64_t)blockIdx.x < m ? (m - 1 - blockIdx.x) / gridDim.x + 1 : 0;
    const int64_t chunks = my_rows * trips;
    bmt::Vec16<T> a[U], b[U];
    const auto load = [&](bmt::Vec16<T>(&v)[U], int64_t c) {
        const int64_t row = blockIdx.x + (c / trips) * gridDim.x;
        const int64_t base = (c % trips) * (int64_t)U * 256 + threadIdx.x;
        const T* __restrict__ xr = x + row * n;
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (base + u * 256 < nv) v[u] = bmt::ld16(xr + (base + u * 256) * V);
    };
    float mx = -INFINITY, se = 0.f;
    int par = 0;
    const auto process = [&](bmt::Vec16<T>(&v)[U], int64_t c) {
        const int64_t row = blockIdx.x + (c / trips) * gridDim.x;
        const int trip = (int)(c % trips);
        const int64_t base = (int64_t)trip * U * 256 + threadIdx.x;
        float lm = -INFINITY;
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (base + u * 256 < nv) lm = fmaxf(lm, packet_max(v[u]));
        if (lm > mx) { se *= ex2((mx - lm) * L2E); mx = lm; }   // mx = -inf: se is 0 and stays 0 (0 * 2^-inf)
        const float off = mx == -INFINITY ? 0.f : -fmaxf(mx * L2E, LOWEST);
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (base + u * 256 < nv) {
#pragma unroll
                for (int k = 0; k < V; ++k) se += ex2(fmaf(bmt::Cvt<T>::to_f(v[u].v[k]), L2E, off));
            }
        if (trip == trips - 1) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                const float m2 = __shfl_xor_sync(0xffffffffu, mx, o), s2 = __shfl_xor_sync(0xffffffffu, se, o);
                lse_combine(mx, se, m2, s2);
            }
            if (lane == 0) { sm_m[par][warp] = mx; sm_s[par][warp] = se; }
            __syncthreads();
            if (threadIdx.x == 0) {
                float gm = sm_m[par][0], gs = sm_s[par][0];
#pragma unroll
                for (int i = 1; i < 8; ++i) lse_combine(gm, gs, sm_m[par][i], sm_s[par][i]);
                const int64_t t = target[row] - vocab_start;
                out[row] = gm;
                out[m + row] = gs;
                out[2 * m + row] = (t >= 0 && t < n) ? bmt::Cvt<T>::to_f(x[row * n + t]) : 0.f;
            }
            par ^= 1;
            mx = -INFINITY;
            se = 0.f;
        }
    };
    if (chunks > 0) load(a, 0);
    for (int64_t c = 0; c < chunks; c += 2) {
        if (c + 1 < chunks) load(b, c + 1);
        process(a, c);
        if (c + 1 < chunks) {
            if (c + 2 < chunks) load(a, c + 2);
            process(b, c + 1);
        }
    }
}

// The reduced loss from the row statistics (3 x m: maximum, sum, target logit): lse of every row, the loss (sum over the rows
// whose target counts, divided by their number when `mean`) and that divisor.  One block up to CE_FINISH_ROWS rows, in the
// place of the dozen elementwise launches that cost the host more than the device.  It takes a fifth of a microsecond per 1024
// rows; above, every block leaves the sum of its rows and their number in the place of its first row's maximum and target
// logit, and a second launch adds them up.  The order is fixed either way.
constexpr int CE_FINISH_THREADS = 1024;
constexpr int64_t CE_FINISH_ROWS = 8192;
__device__ __forceinline__ void ce_result(float sum, float count, int mean, float* loss, float* divisor) {
    *loss = mean ? sum / count : sum;
    *divisor = mean ? count : 1.f;
}
__global__ void __launch_bounds__(CE_FINISH_THREADS) ce_finish_kernel(int64_t m, int64_t chunk, float* __restrict__ rows,
                                                                      const int64_t* __restrict__ target, int64_t ignore_index, int mean,
                                                                      float* __restrict__ lse, float* __restrict__ loss,
                                                                      float* __restrict__ divisor) {
    bmt::after_previous();
    __shared__ float scratch[33];
    const int64_t first = blockIdx.x * chunk, end = first + chunk < m ? first + chunk : m;
    float sum = 0.f, count = 0.f;
#pragma unroll 4
    for (int64_t i = first + threadIdx.x; i < end; i += CE_FINISH_THREADS) {
        const float l = rows[i] + logf(rows[m + i] + 1e-10f);
        lse[i] = l;
        if (target[i] != ignore_index) { sum += l - rows[2 * m + i]; count += 1.f; }
    }
    sum = bmt::block_allreduce<false>(sum, scratch);       // (barriers inside: all maxima of the block have been read)
    count = bmt::block_allreduce<false>(count, scratch);
    if (threadIdx.x != 0) return;
    if (gridDim.x == 1) ce_result(sum, count, mean, loss, divisor);
    else { rows[first] = sum; rows[2 * m + first] = count; }
}
__global__ void __launch_bounds__(256) ce_total_kernel(int64_t m, int blocks, int64_t chunk, const float* __restrict__ rows,
                                                       int mean, float* __restrict__ loss, float* __restrict__ divisor) {
    __shared__ float scratch[33];
    float sum = 0.f, count = 0.f;
    for (int b = threadIdx.x; b < blocks; b += 256) { sum += rows[b * chunk]; count += rows[2 * m + b * chunk]; }
    sum = bmt::block_allreduce<false>(sum, scratch);
    count = bmt::block_allreduce<false>(count, scratch);
    if (threadIdx.x == 0) ce_result(sum, count, mean, loss, divisor);
}

// `divisor` null: grad holds one value per row; else one value for all rows, to be divided by *divisor.
template <typename T>
__global__ void __launch_bounds__(256) ce_backward_kernel(int64_t m, int64_t n, const T* __restrict__ x,
                                                          const int64_t* __restrict__ target, const float* __restrict__ lse,
                                                          const float* __restrict__ grad, const float* __restrict__ divisor,
                                                          int64_t vocab_start, int64_t ignore_index, T* __restrict__ out) {
    bmt::after_previous();
    const int64_t row = blockIdx.x;
    const T* __restrict__ xr = x + row * n;
    T* __restrict__ orow = out + row * n;
    const int64_t tg = target[row];
    const bool ignored = tg == ignore_index;
    const int64_t t = tg - vocab_start;
    constexpr int V = bmt::Vec16<T>::N;
    if (ignored) {       // zeros whatever the logits are: 0 * NaN is none
        const int64_t head = row_head<T>(orow, n), nv = (n - head) / V, tail = head + nv * V;
        bmt::Vec16<T> zero;
#pragma unroll
        for (int k = 0; k < V; ++k) zero.v[k] = bmt::Cvt<T>::from_f(0.f);
        for (int64_t i = threadIdx.x; i < head + n - tail; i += blockDim.x) orow[i < head ? i : tail + i - head] = zero.v[0];
        for (int64_t i = threadIdx.x; i < nv; i += blockDim.x) bmt::st16(orow + head + i * V, zero);
        return;
    }
    const float l = lse[row];
    const float g = divisor ? grad[0] / divisor[0] : grad[row];
    constexpr float L2E = 1.4426950408889634f;
    // p = 2^(x * log2e + off) * 2^rest: `off` is -l * log2e as it is rounded, which near p = 1 is not exact enough, `rest` what
    // the rounding dropped (exact); the second factor goes into the multiplication by g
    const bool huge = fabsf(l) > 1e38f;
    const float off = huge && l > -INFINITY ? fminf(-l * L2E, -LOWEST) : -l * L2E, rest = huge ? 0.f : fmaf(-l, L2E, -off);
    const float pg = g * ex2(rest);
    // as in the forward kernel; vectors need the logits and the gradient to be off the 16-byte boundary by the same amount
    const bool same = (((uintptr_t)xr ^ (uintptr_t)orow) & 15) == 0;
    const int64_t head = same ? row_head<T>(xr, n) : n, nv = (n - head) / V, tail = head + nv * V;
    for (int64_t i = threadIdx.x; i < head + n - tail; i += blockDim.x) {
        const int64_t c = i < head ? i : tail + i - head;
        const float p = ex2(fmaf(bmt::Cvt<T>::to_f(xr[c]), L2E, off));
        orow[c] = bmt::Cvt<T>::from_f(fmaf(p, pg, c == t ? -g : 0.f));
    }
    constexpr int U = 4;
    for (int64_t i0 = threadIdx.x; i0 < nv; i0 += (int64_t)blockDim.x * U) {
        bmt::Vec16<T> v[U];
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (i0 + (int64_t)u * blockDim.x < nv) v[u] = bmt::ld16(xr + head + (i0 + (int64_t)u * blockDim.x) * V);
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int64_t i = i0 + (int64_t)u * blockDim.x;
            if (i >= nv) continue;
            bmt::Vec16<T> o;
#pragma unroll
            for (int k = 0; k < V; ++k) {
                const float p = ex2(fmaf(bmt::Cvt<T>::to_f(v[u].v[k]), L2E, off));
                o.v[k] = bmt::Cvt<T>::from_f(fmaf(p, pg, head + i * V + k == t ? -g : 0.f));
            }
            bmt::st16(orow + head + i * V, o);
        }
    }
}

}  // namespace

extern "C" int bmt_ce_row_stats(int64_t m, int64_t n, const void* logits, int dtype, const void* target, int64_t vocab_start,
                                void* out, void* stream) {
    if (m <= 0) return 0;
    cudaStream_t s = (cudaStream_t)stream;
    static const bool streaming = [] { const char* e = getenv("BMT_CE_STREAM"); return !(e && atoi(e) == 0); }();
    if (streaming && dtype != BMT_DT_F32 && n % 8 == 0 && n >= 2048 && ((uintptr_t)logits & 15) == 0) {
        const int64_t per_thread = (n / 8 + 255) / 256;
        // vectors per trip: the size that leaves the fewest slots of the last trip empty, the larger one when it does not matter
        // (50304 classes: 25 vectors a thread, 4 trips of 8 101 us, 5 trips of 5 96 us)
        int u = 8, trips = (int)((per_thread + 7) / 8);
        for (int c : {6, 5, 4}) {
            const int n_trips = (int)((per_thread + c - 1) / c);
            if (n_trips * c < trips * u) { u = c; trips = n_trips; }
        }
#define BMT_CE_STREAM(T, UU)                                                                                                   \
        do {                                                                                                                   \
            static int per_sm = 0;   /* resident CTAs per SM of this instantiation: the grid is exactly one wave */           \
            if (!per_sm && (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, ce_row_stats_stream_kernel<T, UU>, 256, 0) != cudaSuccess || per_sm < 1)) \
                per_sm = 2;                                                                                                    \
            const int64_t cap = (int64_t)148 * per_sm;                                                                         \
            bmt::launch(ce_row_stats_stream_kernel<T, UU>, (unsigned)(m < cap ? m : cap), 256, 0, s, 1,                                    \
                m, n, trips, (const T*)logits, (const int64_t*)target, vocab_start, (float*)out);                              \
        } while (0)
#define BMT_CE_STREAM_U(T) \
        do { if (u == 4) BMT_CE_STREAM(T, 4); else if (u == 5) BMT_CE_STREAM(T, 5); else if (u == 6) BMT_CE_STREAM(T, 6); else BMT_CE_STREAM(T, 8); } while (0)
        if (dtype == BMT_DT_F16) BMT_CE_STREAM_U(__half); else BMT_CE_STREAM_U(__nv_bfloat16);
#undef BMT_CE_STREAM_U
#undef BMT_CE_STREAM
        bmt_count_launch(1);
        return (int)cudaGetLastError();
    }
    if (dtype == BMT_DT_F16) ce_row_stats_kernel<__half><<<(unsigned)m, 256, 0, s>>>(m, n, (const __half*)logits, (const int64_t*)target, vocab_start, (float*)out);
    else if (dtype == BMT_DT_BF16) ce_row_stats_kernel<__nv_bfloat16><<<(unsigned)m, 256, 0, s>>>(m, n, (const __nv_bfloat16*)logits, (const int64_t*)target, vocab_start, (float*)out);
    else ce_row_stats_kernel<float><<<(unsigned)m, 256, 0, s>>>(m, n, (const float*)logits, (const int64_t*)target, vocab_start, (float*)out);
    bmt_count_launch(1);
    return (int)cudaGetLastError();
}

static int ce_backward(int64_t m, int64_t n, const void* logits, int dtype, const void* target, const void* lse, const void* grad,
                       const void* divisor, int64_t vocab_start, int64_t ignore_index, void* out, void* stream) {
    if (m <= 0) return 0;
    cudaStream_t s = (cudaStream_t)stream;
    const auto run = [&](auto* zero) {
        using T = std::remove_pointer_t<decltype(zero)>;
        bmt::launch(ce_backward_kernel<T>, (unsigned)m, 256, 0, s, 1, m, n, (const T*)logits, (const int64_t*)target, (const float*)lse, (const float*)grad,
                                                          (const float*)divisor, vocab_start, ignore_index, (T*)out);
    };
    if (dtype == BMT_DT_F16) run((__half*)nullptr);
    else if (dtype == BMT_DT_BF16) run((__nv_bfloat16*)nullptr);
    else run((float*)nullptr);
    bmt_count_launch(1);
    return (int)cudaGetLastError();
}

extern "C" int bmt_ce_backward(int64_t m, int64_t n, const void* logits, int dtype, const void* target, const void* lse,
                               const void* grad, int64_t vocab_start, int64_t ignore_index, void* out, void* stream) {
    return ce_backward(m, n, logits, dtype, target, lse, grad, nullptr, vocab_start, ignore_index, out, stream);
}

// Forward and backward of the reduced loss (mean or sum over the rows whose target is not ignore_index).  scratch: 3 * m floats;
// lse: m floats; loss, divisor: one float each (the divisor is what the gradient is divided by).
extern "C" int bmt_ce_reduced_forward(int64_t m, int64_t n, const void* logits, int dtype, const void* target, int64_t ignore_index,
                                      int mean, void* scratch, void* lse, void* loss, void* divisor, void* stream) {
    const int rc = bmt_ce_row_stats(m, n, logits, dtype, target, 0, scratch, stream);
    if (rc != 0) return rc;
    const int64_t share = (m + bmt::sm_count() - 1) / bmt::sm_count();     // a block per SM, of at least 1024 rows
    const int64_t chunk = m <= CE_FINISH_ROWS ? CE_FINISH_ROWS : share > 1024 ? share : 1024;
    const int64_t blocks = m <= CE_FINISH_ROWS ? 1 : (m + chunk - 1) / chunk;
    bmt::launch(ce_finish_kernel, (unsigned)blocks, CE_FINISH_THREADS, 0, (cudaStream_t)stream, 1, m, chunk, (float*)scratch, (const int64_t*)target, ignore_index, mean,
                                                                                       (float*)lse, (float*)loss, (float*)divisor);
    if (blocks > 1) ce_total_kernel<<<1, 256, 0, (cudaStream_t)stream>>>(m, (int)blocks, chunk, (const float*)scratch, mean, (float*)loss, (float*)divisor);
    bmt_count_launch(blocks > 1 ? 2 : 1);
    return (int)cudaGetLastError();
}

extern "C" int bmt_ce_reduced_backward(int64_t m, int64_t n, const void* logits, int dtype, const void* target, const void* lse,
                                       const void* grad, const void* divisor, int64_t ignore_index, void* out, void* stream) {
    return ce_backward(m, n, logits, dtype, target, lse, grad, divisor, 0, ignore_index, out, stream);
}
