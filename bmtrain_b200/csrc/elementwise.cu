// SwiGLU forward/backward and column sums (bias gradient).
#include "api.h"
#include "common.cuh"

namespace {

// The kernels below move 16-byte vectors, EW_U positions a thread, one piece of EW_BLOCK positions a block: resident blocks that loop wait
// for their loads and stores in turn and copied at 0.9 of the rate.  A position is divided into row and column once per block in
// 64 bits and per position in 32: with a 64-bit division for every vector the arithmetic set the pace.
constexpr int EW_THREADS = 256, EW_U = 2, EW_BLOCK = EW_THREADS * EW_U;

struct RowPlace { int64_t row; uint32_t rest; };      // of a block's first position among rows of `per_row`
__device__ __forceinline__ RowPlace block_place(uint32_t per_row) {
    const int64_t first = (int64_t)blockIdx.x * EW_BLOCK, row = first / per_row;
    return RowPlace{row, (uint32_t)(first - row * per_row)};
}

// 4096 x 13824 bf16: 84 -> 72 us forward, 105 -> 95 us backward, fp16 72 -> 67 and 109 -> 88.  An approximate reciprocal for the division would take
// 61 and 87, at the cost of a rounding.
template <typename T>
__global__ void __launch_bounds__(EW_THREADS) swiglu_fwd_kernel(int64_t total, int64_t f, const T* __restrict__ x, T* __restrict__ out) {
    bmt::after_previous();
    const uint32_t per_row = (uint32_t)(f / 8);
    const RowPlace at = block_place(per_row);
    bmt::Vec16<T> g[EW_U], u[EW_U];
    int64_t o[EW_U];
#pragma unroll
    for (int i = 0; i < EW_U; ++i) {
        const uint32_t n = at.rest + threadIdx.x + i * EW_THREADS, r = n / per_row, c = (n - r * per_row) * 8;
        o[i] = (int64_t)blockIdx.x * EW_BLOCK + threadIdx.x + i * EW_THREADS < total ? (at.row + r) * f + c : -1;
        if (o[i] >= 0) {
            const T* p = x + (at.row + r) * 2 * f + c;
            g[i] = bmt::ld16(p);
            u[i] = bmt::ld16(p + f);
        }
    }
#pragma unroll
    for (int i = 0; i < EW_U; ++i) {
        if (o[i] < 0) continue;
        bmt::Vec16<T> y;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const float gv = bmt::Cvt<T>::to_f(g[i].v[k]);
            y.v[k] = bmt::Cvt<T>::from_f(gv / (1.f + __expf(-gv)) * bmt::Cvt<T>::to_f(u[i].v[k]));
        }
        bmt::st16(out + o[i], y);
    }
}

template <typename T>
__global__ void __launch_bounds__(EW_THREADS) swiglu_bwd_kernel(int64_t total, int64_t f, const T* __restrict__ x, const T* __restrict__ go, T* __restrict__ dx) {
    bmt::after_previous();
    const uint32_t per_row = (uint32_t)(f / 8);
    const RowPlace at = block_place(per_row);
    bmt::Vec16<T> g[EW_U], u[EW_U], d[EW_U];
    int64_t o[EW_U];
#pragma unroll
    for (int i = 0; i < EW_U; ++i) {
        const uint32_t n = at.rest + threadIdx.x + i * EW_THREADS, r = n / per_row, c = (n - r * per_row) * 8;
        o[i] = (int64_t)blockIdx.x * EW_BLOCK + threadIdx.x + i * EW_THREADS < total ? (at.row + r) * 2 * f + c : -1;
        if (o[i] >= 0) {
            g[i] = bmt::ld16(x + o[i]);
            u[i] = bmt::ld16(x + o[i] + f);
            d[i] = bmt::ld16(go + (at.row + r) * f + c);
        }
    }
#pragma unroll
    for (int i = 0; i < EW_U; ++i) {
        if (o[i] < 0) continue;
        bmt::Vec16<T> dg, du;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const float gv = bmt::Cvt<T>::to_f(g[i].v[k]), uv = bmt::Cvt<T>::to_f(u[i].v[k]), dv = bmt::Cvt<T>::to_f(d[i].v[k]);
            const float sg = 1.f / (1.f + __expf(-gv)), silu = gv * sg;
            dg.v[k] = bmt::Cvt<T>::from_f(dv * uv * (sg + silu * (1.f - sg)));
            du.v[k] = bmt::Cvt<T>::from_f(dv * silu);
        }
        bmt::st16(dx + o[i], dg);
        bmt::st16(dx + o[i] + f, du);
    }
}

// Column sums of an (m, n) matrix (bias gradients).  Block = 8 column packets (64 columns) x 32 row lanes; grid =
// (column blocks, row splits): with `splits` > 1 every CTA writes its 64 fp32 partial sums to `scratch[split][n]`, and
// the CTA that finishes last in its column block (a ticket counter behind the partials, reset for the next call) adds
// the partials up in split order -- the result does not depend on the order in which CTAs run.  `acc`: out += sums.
template <typename T>
__global__ void __launch_bounds__(256) colsum_kernel(int64_t m, int64_t n, const T* __restrict__ x, T* __restrict__ out, int acc,
                                                     float* __restrict__ scratch, unsigned int* __restrict__ tickets) {
    bmt::after_previous();
    __shared__ float red[32][65];
    __shared__ unsigned int last_s;
    const int cv = threadIdx.x & 7, lane = threadIdx.x >> 3;
    const int splits = gridDim.y, split = blockIdx.y;
    const int64_t c = (int64_t)blockIdx.x * 64 + cv * 8;
    float a0[8] = {0, 0, 0, 0, 0, 0, 0, 0}, a1[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    if (c < n) {
        const int64_t step = (int64_t)32 * splits;
        int64_t r = (int64_t)split * 32 + lane;
        for (; r + step < m; r += 2 * step) {          // two independent loads in flight per thread
            const bmt::Vec16<T> v0 = bmt::ld16(x + r * n + c), v1 = bmt::ld16(x + (r + step) * n + c);
#pragma unroll
            for (int k = 0; k < 8; ++k) { a0[k] += bmt::Cvt<T>::to_f(v0.v[k]); a1[k] += bmt::Cvt<T>::to_f(v1.v[k]); }
        }
        if (r < m) {
            const bmt::Vec16<T> v0 = bmt::ld16(x + r * n + c);
#pragma unroll
            for (int k = 0; k < 8; ++k) a0[k] += bmt::Cvt<T>::to_f(v0.v[k]);
        }
    }
#pragma unroll
    for (int k = 0; k < 8; ++k) red[lane][cv * 8 + k] = a0[k] + a1[k];
    __syncthreads();
    const int64_t col = (int64_t)blockIdx.x * 64 + threadIdx.x;
    float s = 0.f;
    if (threadIdx.x < 64) {
#pragma unroll 8
        for (int l = 0; l < 32; ++l) s += red[l][threadIdx.x];
    }
    if (splits == 1) {
        if (threadIdx.x < 64 && col < n) out[col] = bmt::Cvt<T>::from_f(acc ? s + bmt::Cvt<T>::to_f(out[col]) : s);
        return;
    }
    if (threadIdx.x < 64 && col < n) scratch[(int64_t)split * n + col] = s;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
        const unsigned int t = atomicAdd(tickets + blockIdx.x, 1u);
        last_s = (t == (unsigned int)splits - 1) ? 1u : 0u;
        if (last_s) tickets[blockIdx.x] = 0;            // every CTA of this column block has taken its ticket
    }
    __syncthreads();
    if (!last_s) return;
    __threadfence();
    if (threadIdx.x < 64 && col < n) {
        float t = 0.f;
        for (int i = 0; i < splits; ++i) t += __ldcg(scratch + (int64_t)i * n + col);
        out[col] = bmt::Cvt<T>::from_f(acc ? t + bmt::Cvt<T>::to_f(out[col]) : t);
    }
}

// Column sums of several matrices in one launch: 32 columns a block, which walks over all rows, so that nothing is handed over between
// blocks.  Latency bounds it: 8 loads of 16 bytes a thread in flight, one pass over what the backward has just left in L2.  A block's
// backward has four bias gradients and four sums of its norms.  256 tokens of 256: 16.1 us for the four alone, a launch each, 3.2 us
// for all eight here; 1024 of 2560: 34 and 19.5; 2048 of 4096: 62 and 44.
struct ColsumTable { BmtColsum item[BMT_MAX_COLSUMS]; int count; };
template <typename T>
__global__ void __launch_bounds__(256) colsum_multi_kernel(const __grid_constant__ ColsumTable tab, int acc) {
    bmt::after_previous();
    __shared__ float red[64][33], part[8][32];
    int it = 0;
    while (it + 1 < tab.count && (int)blockIdx.x >= tab.item[it + 1].first) ++it;
    const BmtColsum& item = tab.item[it];
    const int64_t m = item.m, n = item.n, c0 = (int64_t)((int)blockIdx.x - item.first) * 32;
    const int lanes = item.f32 ? 32 : 64;
    float a[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    if (!item.f32) {
        const int cv = (threadIdx.x & 3) * 8, lane = threadIdx.x >> 2;
        if (c0 + cv < n) {
            const T* x = (const T*)item.x + c0 + cv;
            for (int64_t r = lane; r < m; r += 64 * 8) {
                bmt::Vec16<T> v[8];
#pragma unroll
                for (int u = 0; u < 8; ++u)
                    if (r + u * 64 < m) v[u] = bmt::ld16(x + (r + u * 64) * n);
#pragma unroll
                for (int u = 0; u < 8; ++u)
                    if (r + u * 64 < m) {
#pragma unroll
                        for (int k = 0; k < 8; ++k) a[k] += bmt::Cvt<T>::to_f(v[u].v[k]);
                    }
            }
        }
#pragma unroll
        for (int k = 0; k < 8; ++k) red[lane][cv + k] = a[k];
    } else {
        const int cv = (threadIdx.x & 7) * 4, lane = threadIdx.x >> 3;
        if (c0 + cv < n) {
            const float* x = (const float*)item.x + c0 + cv;
            for (int64_t r = lane; r < m; r += 32 * 8) {
                float4 v[8];
#pragma unroll
                for (int u = 0; u < 8; ++u)
                    if (r + u * 32 < m) v[u] = *reinterpret_cast<const float4*>(x + (r + u * 32) * n);
#pragma unroll
                for (int u = 0; u < 8; ++u)
                    if (r + u * 32 < m) { a[0] += v[u].x; a[1] += v[u].y; a[2] += v[u].z; a[3] += v[u].w; }
            }
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) red[lane][cv + k] = a[k];
    }
    __syncthreads();
    const int col = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float s = 0.f;
    for (int l = warp; l < lanes; l += 8) s += red[l][col];
    part[warp][col] = s;
    __syncthreads();
    if (warp == 0 && c0 + col < n) {
        float t = 0.f;
#pragma unroll
        for (int w = 0; w < 8; ++w) t += part[w][col];
        T* out = (T*)item.out + c0 + col;
        *out = bmt::Cvt<T>::from_f(acc ? t + bmt::Cvt<T>::to_f(*out) : t);
    }
}

// 4096 x 27648 bf16: 128 us with erff, 107 here; the instructions bound it, no longer the bytes (0.64 of the copy rate)
template <typename T>
__global__ void __launch_bounds__(EW_THREADS) gelu_kernel(int64_t n8, const T* __restrict__ x, T* __restrict__ out) {
    bmt::after_previous();
    const int64_t first = (int64_t)blockIdx.x * EW_BLOCK + threadIdx.x;
    bmt::Vec16<T> v[EW_U];
#pragma unroll
    for (int i = 0; i < EW_U; ++i)
        if (first + i * EW_THREADS < n8) v[i] = bmt::ld16(x + (first + i * EW_THREADS) * 8);
#pragma unroll
    for (int i = 0; i < EW_U; ++i) {
        if (first + i * EW_THREADS >= n8) continue;
        const uint32_t* in = reinterpret_cast<const uint32_t*>(v[i].v);
        bmt::Vec16<T> o;
#pragma unroll
        for (int k = 0; k < 4; ++k) reinterpret_cast<uint32_t*>(o.v)[k] = bmt::from_f2<T>(bmt::gelu(bmt::to_f2<T>(in[k])));
        bmt::st16(out + (first + i * EW_THREADS) * 8, o);
    }
}

// Rotary position embedding on a packed projection.  `packed` is (b, s, hk, g + 2, d): per kv head g query heads, one key
// head, one value head ("half rotation" convention: element i pairs with i + d/2, angle = pos * theta^(-2i/d); `cs` holds
// (cos, sin) of every (position, i) as interleaved fp32 pairs, (pos0 + seq) x d/2 of them).
// SPLIT: packed -> q (b, s, hk*g, d) rotated, k (b, s, hk, d) rotated, v (b, s, hk, d) copied, all contiguous.
// !SPLIT (backward): gradients of q, k, v -> gradient of packed (contiguous), q and k parts rotated back.
// A thread moves 8 elements of the lower half of a head and their 8 partners of the upper half at a time, EW_U of them, all of one token:
// blocks of (positions of a token, tokens), so that a token's place is divided out once and a position's by multiplication.  4096 tokens,
// 120 heads x 128: 64 us with divisions for every position, now 56; the 64 bytes of the table for every 32 are the rest.  Four heads a
// thread, which read the table once for all of them, took 74.
struct FastDiv {
    uint32_t d, m;          // ceil(2^32 / d), exact for numerators below 65536; 0: d = 1, or larger numerators
    FastDiv(uint32_t d_, bool small) : d(d_), m(d_ > 1 && small ? (uint32_t)((0x100000000ull + d_ - 1) / d_) : 0u) {}
    __device__ __forceinline__ uint32_t operator()(uint32_t n) const { return m ? __umulhi(n, m) : d == 1 ? n : n / d; }
};

template <typename T, bool SPLIT>
__global__ void __launch_bounds__(EW_THREADS) rope_qkv_kernel(int64_t tokens, int64_t seq, int hk, int g, int d, FastDiv by_vecs, FastDiv by_group,
                                                              T* __restrict__ packed, int64_t p_tok, int64_t p_batch, T* __restrict__ q,
                                                              T* __restrict__ k, T* __restrict__ v, const float* __restrict__ cs, int64_t pos0) {
    bmt::after_previous();
    const int64_t token = (int64_t)blockIdx.x * blockDim.y + threadIdx.y;
    if (token >= tokens) return;
    const int half = d / 2;
    const uint32_t per_tok = by_vecs.d * (uint32_t)hk * by_group.d, p0 = blockIdx.y * blockDim.x * EW_U + threadIdx.x;
    const int64_t bb = token / seq, t = token - bb * seq;
    T* const pin = packed + bb * p_batch + t * p_tok;
    const float* const row = cs + (pos0 + t) * half * 2;
    bmt::Vec16<T> lo[EW_U], hi[EW_U];
    T* dst[EW_U];
    int turn[EW_U];              // the first of the 8 frequencies, or -1: values are copied
#pragma unroll
    for (int i = 0; i < EW_U; ++i) {
        const uint32_t p = p0 + i * blockDim.x;
        dst[i] = nullptr;
        if (p >= per_tok) continue;
        const uint32_t slot = by_vecs(p), kvh = by_group(slot), j = slot - kvh * by_group.d;
        const int c = (int)(p - slot * by_vecs.d) * 8;
        T* const in = pin + (int64_t)slot * d + c;
        T* const sep = (j < (uint32_t)g ? q + ((token * hk + kvh) * g + j) * d : (j == (uint32_t)g ? k : v) + (token * hk + kvh) * d) + c;
        const T* const src = SPLIT ? in : sep;
        dst[i] = SPLIT ? sep : in;
        turn[i] = j <= (uint32_t)g ? c : -1;
        lo[i] = bmt::ld16(src);
        hi[i] = bmt::ld16(src + half);
    }
#pragma unroll
    for (int i = 0; i < EW_U; ++i) {
        if (!dst[i]) continue;
        if (turn[i] >= 0) {
            // (cos, sin) of position x frequency from the table (seq x d/2 pairs, built once per shape; it stays in L2)
            const float4* tab = reinterpret_cast<const float4*>(row + turn[i] * 2);
            float4 q4[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) q4[e] = tab[e];
            const float* f = reinterpret_cast<const float*>(q4);
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                const float co = f[2 * e];
                const float sn = SPLIT ? f[2 * e + 1] : -f[2 * e + 1];
                const float a = bmt::Cvt<T>::to_f(lo[i].v[e]), b2 = bmt::Cvt<T>::to_f(hi[i].v[e]);
                lo[i].v[e] = bmt::Cvt<T>::from_f(a * co - b2 * sn);
                hi[i].v[e] = bmt::Cvt<T>::from_f(a * sn + b2 * co);
            }
        }
        bmt::st16(dst[i], lo[i]);
        bmt::st16(dst[i] + half, hi[i]);
    }
}

unsigned blocks_of(int64_t positions) { return (unsigned)bmt::ceil_div64(positions, EW_BLOCK); }

}  // namespace

extern "C" int bmt_swiglu_fwd(int64_t rows, int64_t f, const void* x, int dtype, void* out, void* stream) {
    if (rows <= 0 || f <= 0) return 0;
    if (f % 8 || dtype == BMT_DT_F32) return -3;
    cudaStream_t s = (cudaStream_t)stream;
    if (dtype == BMT_DT_F16) bmt::launch(swiglu_fwd_kernel<__half>, blocks_of(rows * (f / 8)), EW_THREADS, 0, s, 1, rows * (f / 8), f, (const __half*)x, (__half*)out);
    else bmt::launch(swiglu_fwd_kernel<__nv_bfloat16>, blocks_of(rows * (f / 8)), EW_THREADS, 0, s, 1, rows * (f / 8), f, (const __nv_bfloat16*)x, (__nv_bfloat16*)out);
    bmt_count_launch(1);
    return (int)cudaGetLastError();
}

extern "C" int bmt_swiglu_bwd(int64_t rows, int64_t f, const void* x, const void* g, int dtype, void* dx, void* stream) {
    if (rows <= 0 || f <= 0) return 0;
    if (f % 8 || dtype == BMT_DT_F32) return -3;
    cudaStream_t s = (cudaStream_t)stream;
    if (dtype == BMT_DT_F16) bmt::launch(swiglu_bwd_kernel<__half>, blocks_of(rows * (f / 8)), EW_THREADS, 0, s, 1, rows * (f / 8), f, (const __half*)x, (const __half*)g, (__half*)dx);
    else bmt::launch(swiglu_bwd_kernel<__nv_bfloat16>, blocks_of(rows * (f / 8)), EW_THREADS, 0, s, 1, rows * (f / 8), f, (const __nv_bfloat16*)x, (const __nv_bfloat16*)g, (__nv_bfloat16*)dx);
    bmt_count_launch(1);
    return (int)cudaGetLastError();
}

// `scratch` (optional): fp32 work space, `scratch_bytes` large; its first 4 KB hold the ticket counters and must be zero
// before the first call (the kernel leaves them zero), the rest takes the per-split partial sums.  Calls that share a
// scratch must be ordered on one stream.  Without scratch one CTA per 64 columns walks over all rows.
extern "C" int bmt_colsum_ex(int64_t m, int64_t n, const void* x, int dtype, void* out, int accumulate, void* scratch,
                             int64_t scratch_bytes, void* stream) {
    if (n <= 0) return 0;
    if (n % 8 || dtype == BMT_DT_F32) return -3;
    cudaStream_t s = (cudaStream_t)stream;
    const int64_t cb = (n + 63) / 64;
    int64_t splits = 1;
    if (scratch && cb <= 1024) {
        splits = (4 * 148 + cb - 1) / cb;                                  // about four CTAs per SM
        const int64_t by_rows = m / 128, by_mem = (scratch_bytes - 4096) / (n * 4);
        if (splits > by_rows) splits = by_rows;                            // at least four rows per lane
        if (splits > by_mem) splits = by_mem;
        if (splits > 64) splits = 64;
        if (splits < 1) splits = 1;
    }
    const dim3 g((unsigned)cb, (unsigned)splits);
    unsigned int* tickets = (unsigned int*)scratch;
    float* partial = scratch ? (float*)((char*)scratch + 4096) : nullptr;
    if (dtype == BMT_DT_F16) bmt::launch(colsum_kernel<__half>, g, 256, 0, s, 1, m, n, (const __half*)x, (__half*)out, accumulate, partial, tickets);
    else bmt::launch(colsum_kernel<__nv_bfloat16>, g, 256, 0, s, 1, m, n, (const __nv_bfloat16*)x, (__nv_bfloat16*)out, accumulate, partial, tickets);
    bmt_count_launch(1);
    return (int)cudaGetLastError();
}

// Beyond 2048 rows the kernel that splits them is as fast or faster (four sums of a 4096-token block of 4096: 86 us there, 93 here;
// 8192 tokens: 137 and 157): its blocks are short, so the last wave is.
extern "C" int bmt_colsum_multi(const BmtColsum* items, int count, int dtype, int accumulate, void* scratch, int64_t scratch_bytes, void* stream) {
    if (count < 0 || count > BMT_MAX_COLSUMS || dtype == BMT_DT_F32) return -3;
    ColsumTable tab;
    tab.count = 0;
    int64_t blocks = 0;
    for (int i = 0; i < count; ++i) {
        const BmtColsum& it = items[i];
        if (it.n <= 0) continue;
        if (it.n % 8) return -3;
        const int64_t wide = bmt::ceil_div64(it.n, 32);
        if (!it.f32 && it.m > 2048) {
            const int rc = bmt_colsum_ex(it.m, it.n, it.x, dtype, it.out, accumulate, scratch, scratch_bytes, stream);
            if (rc) return rc;
            continue;
        }
        tab.item[tab.count] = it;
        tab.item[tab.count++].first = (int)blocks;
        blocks += wide;
    }
    if (blocks == 0) return 0;
    if (blocks > 0x7fffffff) return -3;
    if (dtype == BMT_DT_F16) bmt::launch(colsum_multi_kernel<__half>, (unsigned)blocks, 256, 0, (cudaStream_t)stream, 1, tab, accumulate);
    else bmt::launch(colsum_multi_kernel<__nv_bfloat16>, (unsigned)blocks, 256, 0, (cudaStream_t)stream, 1, tab, accumulate);
    bmt_count_launch(1);
    return (int)cudaGetLastError();
}

extern "C" int bmt_colsum(int64_t m, int64_t n, const void* x, int dtype, void* out, void* stream) {
    return bmt_colsum_ex(m, n, x, dtype, out, 0, nullptr, 0, stream);
}

// out = gelu(x), n elements (multiple of 8), exact erf form
extern "C" int bmt_gelu_fwd(int64_t n, const void* x, int dtype, void* out, void* stream) {
    if (n <= 0) return 0;
    if (n % 8 || dtype == BMT_DT_F32) return -3;
    cudaStream_t s = (cudaStream_t)stream;
    if (dtype == BMT_DT_F16) bmt::launch(gelu_kernel<__half>, blocks_of(n / 8), EW_THREADS, 0, s, 1, n / 8, (const __half*)x, (__half*)out);
    else bmt::launch(gelu_kernel<__nv_bfloat16>, blocks_of(n / 8), EW_THREADS, 0, s, 1, n / 8, (const __nv_bfloat16*)x, (__nv_bfloat16*)out);
    bmt_count_launch(1);
    return (int)cudaGetLastError();
}

// Rotary embedding of a packed (b, s, hk, g + 2, d) projection (token / batch strides p_tok / p_batch, the last three
// dims contiguous).  split != 0: writes rotated q, k and the copied v (contiguous); split == 0: the backward, reads the
// three gradients and writes the packed gradient (contiguous, p_tok / p_batch describe it).  d: multiple of 16.
// cos_sin: fp32 table of (cos, sin) pairs, (pos0 + seq) x d/2, 16-byte aligned.
extern "C" int bmt_rope_qkv(int64_t batch, int64_t seq, int hk, int g, int d, void* packed, int64_t p_tok, int64_t p_batch, void* q,
                            void* k, void* v, const void* cos_sin, int64_t pos0, int split, int dtype, void* stream) {
    if (batch <= 0 || seq <= 0) return 0;
    if (d % 16 || dtype == BMT_DT_F32 || (p_tok & 7) || (p_batch & 7) || !cos_sin || ((uintptr_t)cos_sin & 15)) return -3;
    cudaStream_t s = (cudaStream_t)stream;
    const int64_t tokens = batch * seq, per_tok = (int64_t)hk * (g + 2) * (d / 16);
    const bool small = per_tok < 65536;
    unsigned x = 4;                        // threads along a token's positions (131072 tokens of three heads x 64: 67 us with 32, 30 with 8)
    while (x < EW_THREADS && (int64_t)x * EW_U < per_tok) x *= 2;
    const dim3 block(x, EW_THREADS / x), grid((unsigned)bmt::ceil_div64(tokens, block.y), (unsigned)bmt::ceil_div64(per_tok, x * EW_U));
    const auto run = [&](auto zero) {
        using T = decltype(zero);
        const auto kernel = split ? rope_qkv_kernel<T, true> : rope_qkv_kernel<T, false>;
        return bmt::launch(kernel, grid, block, 0, s, 1, tokens, seq, hk, g, d, FastDiv((uint32_t)(d / 16), small), FastDiv((uint32_t)(g + 2), small), (T*)packed, p_tok,
                           p_batch, (T*)q, (T*)k, (T*)v, (const float*)cos_sin, pos0);
    };
    if (dtype == BMT_DT_F16) run(__half());
    else run(__nv_bfloat16());
    bmt_count_launch(1);
    return (int)cudaGetLastError();
}
