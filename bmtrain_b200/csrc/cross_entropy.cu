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

__device__ __forceinline__ float packet_max(const bmt::Vec16<float>& v) { return fmaxf(fmaxf(v.v[0], v.v[1]), fmaxf(v.v[2], v.v[3])); }

// Statistics of a row, one block each: its maximum, the sum of exp relative to it, the logit of its target.  Every thread has U
// vectors in flight while it works on the U before them; the few elements before the first 16-byte boundary of a row (rows of an odd
// number of classes start anywhere) and behind its last whole vector go one by one.  The bytes bound it, because little is issued for
// an element beyond a conversion, an FMA, an ex2 and an addition; a persistent grid whose chunks were found by 64-bit divisions issued
// twice as much, and held rows back for its last wave.  4096 x 50304 bf16: 91 us, now 66
// (6.2 TB/s); 4096 x 50257, element by element at the edges in a kernel of its own: 88, now 67; 16384 x 10240: 93, now 68.
// The rows go from the last to the first, so that the backward, which begins with the first, finds some in L2.
template <typename T, int U>
__global__ void __launch_bounds__(256) ce_row_stats_kernel(int64_t m, int64_t n, const T* __restrict__ x, const int64_t* __restrict__ target,
                                                           int64_t vocab_start, float* __restrict__ out) {
    bmt::after_previous();
    constexpr int V = bmt::Vec16<T>::N;
    constexpr float L2E = 1.4426950408889634f;
    __shared__ float sm_m[8], sm_s[8];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t row = m - 1 - (int64_t)blockIdx.x;
    const T* __restrict__ xr = x + row * n;
    const int64_t head = row_head<T>(xr, n), nv = (n - head) / V, tail = head + nv * V;
    const int64_t t = threadIdx.x == 0 ? target[row] - vocab_start : -1;
    const T* __restrict__ p = xr + head + (int64_t)threadIdx.x * V;
    int64_t left = nv - threadIdx.x;              // this thread has a vector at p + u * 256 * V where u * 256 < left
    // (a vector that is not there is not set to something either: that would wait for the load in its place)
    struct Trip { bmt::Vec16<T> v[U]; int in; } a, b;
    const auto load = [&](Trip& to) {
        to.in = left > U * 256 ? U * 256 : (int)left;
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (u * 256 < to.in) to.v[u] = bmt::ld16(p + u * 256 * V);
        p += U * 256 * V;
        left -= U * 256;
    };
    // mx: largest logit so far; se: sum of 2^(x * log2e + off), off = -mx * log2e as it is rounded.  Taking the rounded product as the
    // reference keeps the exponent exact to one rounding of the FMA; its distance from mx * log2e is made up for once, at the end.
    float mx = -INFINITY, off = 0.f, se = 0.f;    // (off is 0 as long as all classes are hidden: -inf adds nothing)
    const auto move_to = [&](float v) {
        if (!(v > mx)) return;
        const float o = -fmaxf(v * L2E, LOWEST);
        if (mx != -INFINITY) se *= ex2(o - off);
        mx = v;
        off = o;
    };
    const auto add = [&](const Trip& from) {
        float lm = -INFINITY;
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (u * 256 < from.in) lm = fmaxf(lm, packet_max(from.v[u]));
        move_to(lm);
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (u * 256 < from.in) {
#pragma unroll
                for (int k = 0; k < V; ++k) se += ex2(fmaf(bmt::Cvt<T>::to_f(from.v[u].v[k]), L2E, off));
            }
    };
    load(a);
    T hit = bmt::Cvt<T>::from_f(0.f);
    if (t >= 0 && t < n) hit = xr[t];
    if ((int64_t)threadIdx.x < head + n - tail) {
        const float f = bmt::Cvt<T>::to_f(xr[threadIdx.x < head ? threadIdx.x : tail + threadIdx.x - head]);
        move_to(f);
        se += ex2(fmaf(f, L2E, off));
    }
    for (;;) {
        const bool more = left > 0;
        if (more) load(b);
        add(a);
        if (!more) break;
        const bool again = left > 0;
        if (again) load(a);
        add(b);
        if (!again) break;
    }
    // one factor takes a thread's sum to the row's maximum, so that its error enters once
    const float warp_most = bmt::warp_max(mx);
    if (lane == 0) sm_m[warp] = warp_most;
    __syncthreads();
    float most = sm_m[0];
#pragma unroll
    for (int i = 1; i < 8; ++i) most = fmaxf(most, sm_m[i]);
    se = bmt::warp_sum(se == 0.f ? 0.f : se * ex2(-fmaf(most, L2E, off)));      // zero: no class that counts (a NaN is not lost)
    if (lane == 0) sm_s[warp] = se;
    __syncthreads();
    if (threadIdx.x == 0) {
        se = sm_s[0];
#pragma unroll
        for (int i = 1; i < 8; ++i) se += sm_s[i];
        out[row] = most;
        out[m + row] = se;
        out[2 * m + row] = bmt::Cvt<T>::to_f(hit);
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
    const auto run = [&](auto* zero) {
        using T = std::remove_pointer_t<decltype(zero)>;
        const int64_t per_thread = (n / bmt::Vec16<T>::N + 255) / 256;
        // 5 vectors in flight, 4 where that leaves fewer places of the last trip empty (8: 85 us instead of 68 at 4096 x 50304); short
        // rows take no more than they have (4096 x 1000: 11.0 us with 1, 12.9 with 5)
        const auto places = [&](int u) { return (per_thread + u - 1) / u * u; };
        const auto kernel = per_thread <= 1 ? ce_row_stats_kernel<T, 1> : per_thread <= 2 ? ce_row_stats_kernel<T, 2>
                          : places(4) < places(5) ? ce_row_stats_kernel<T, 4> : ce_row_stats_kernel<T, 5>;
        bmt::launch(kernel, (unsigned)m, 256, 0, s, 1, m, n, (const T*)logits, (const int64_t*)target, vocab_start, (float*)out);
    };
    if (dtype == BMT_DT_F16) run((__half*)nullptr);
    else if (dtype == BMT_DT_BF16) run((__nv_bfloat16*)nullptr);
    else run((float*)nullptr);
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
