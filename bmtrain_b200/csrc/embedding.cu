// Embedding gather and its gradient (ids < 0: zeros in forward, skipped in backward).
#include <type_traits>

#include "api.h"
#include "common.cuh"

namespace {

template <typename T, bool EARLY>
__global__ void __launch_bounds__(128) emb_fwd_kernel(int64_t d, const int64_t* __restrict__ ids, const T* __restrict__ w, T* __restrict__ out) {
    if (EARLY) bmt::after_previous();
    const int64_t t = blockIdx.x;
    const int64_t id = ids[t];
    T* __restrict__ o = out + t * d;
    constexpr int V = bmt::Vec16<T>::N;
    if (id < 0) {
        bmt::Vec16<T> z;
#pragma unroll
        for (int k = 0; k < V; ++k) z.v[k] = bmt::Cvt<T>::from_f(0.f);
        for (int64_t c = threadIdx.x * V; c < d; c += blockDim.x * V) bmt::st16(o + c, z);
        return;
    }
    const T* __restrict__ src = w + id * d;
    for (int64_t c = threadIdx.x * V; c < d; c += blockDim.x * V) bmt::st16(o + c, bmt::ld16(src + c));
}

// Gradient of the table: row r = sum of the gradients of the tokens with id r, added in fp32, rounded once.
// A table has far more rows than a batch has tokens, so what bounds it is writing the table (50304 x 4096 bf16: 63 us at the
// copy rate).  Zeroing an fp32 table, adding to it atomically and converting it moved five times that (490 us there).  So the
// tokens are ordered by id first -- three small kernels over tokens or rows: count and rank, a start for every row that has
// tokens, order -- and every row is then written once, by a team of threads that adds up its tokens.  Rows with more than
// EMB_HOT tokens (padding) are left to a kernel that spreads one row's tokens over warps and its columns over blocks.
constexpr int EMB_HOT = 64;

struct EmbScratch {                 // one int32 array: total, hot rows | count[rows] | start[rows] | hot[hot_cap] | rank[tokens] | order[tokens]
    int *total, *n_hot, *count, *start, *hot, *rank, *order;
};
__host__ __device__ __forceinline__ int64_t emb_hot_cap(int64_t tokens) { return tokens / EMB_HOT + 1; }
EmbScratch emb_scratch(void* base, int64_t tokens, int64_t rows) {
    EmbScratch e;
    int* p = (int*)base;
    e.total = p; e.n_hot = p + 1; e.count = p + 2; e.start = e.count + rows; e.hot = e.start + rows; e.rank = e.hot + emb_hot_cap(tokens);
    e.order = e.rank + tokens;
    return e;
}

__global__ void __launch_bounds__(256) emb_count_kernel(int64_t tokens, int64_t rows, const int64_t* __restrict__ ids, EmbScratch e) {
    bmt::after_previous();
    const int64_t t = (int64_t)blockIdx.x * 256 + threadIdx.x;
    if (t >= tokens) return;
    const int64_t id = ids[t];
    if (id >= 0 && id < rows) e.rank[t] = atomicAdd(e.count + id, 1);
}
__global__ void __launch_bounds__(256) emb_start_kernel(int64_t rows, EmbScratch e) {
    bmt::after_previous();
    const int64_t r = (int64_t)blockIdx.x * 256 + threadIdx.x;
    if (r >= rows) return;
    const int c = e.count[r];
    if (c == 0) return;
    e.start[r] = atomicAdd(e.total, c);
    if (c > EMB_HOT) e.hot[atomicAdd(e.n_hot, 1)] = (int)r;
}
__global__ void __launch_bounds__(256) emb_order_kernel(int64_t tokens, int64_t rows, const int64_t* __restrict__ ids, EmbScratch e) {
    bmt::after_previous();
    const int64_t t = (int64_t)blockIdx.x * 256 + threadIdx.x;
    if (t >= tokens) return;
    const int64_t id = ids[t];
    if (id >= 0 && id < rows) e.order[e.start[id] + e.rank[t]] = (int)t;
}
template <typename T> __device__ __forceinline__ T plus(T held, float sum) {
    return bmt::Cvt<T>::from_f(bmt::Cvt<T>::to_f(held) + bmt::Cvt<T>::to_f(bmt::Cvt<T>::from_f(sum)));
}
// `team` threads (32 .. 256) per row.  ADD: the sums are added to what the table's gradient holds already, rounded first as the gradient
// they would be without: the bits of a gradient do not depend on whether zeros were there before.
// Then only rows that have tokens are touched, and there is a team per token instead, which works if its token is the first of its
// row: 4096 tokens, 50304 x 4096 bf16: 68 us for the whole table, and 190 us of autograd adding that up, became 14 us.
template <typename T, bool ADD>
__global__ void __launch_bounds__(256) emb_rows_kernel(int64_t items, int64_t rows, int64_t d, int team, const int64_t* __restrict__ ids,
                                                       const T* __restrict__ g, EmbScratch e, T* __restrict__ out) {
    bmt::after_previous();
    constexpr int V = bmt::Vec16<T>::N;
    int64_t r = (int64_t)blockIdx.x * (256 / team) + threadIdx.x / team;
    if (r >= items) return;
    if (ADD) {
        const int64_t id = ids[r];
        if (id < 0 || id >= rows || e.rank[r] != 0) return;
        r = id;
    }
    const int c = e.count[r];
    if (c > EMB_HOT) return;
    const int* __restrict__ tok = e.order + (c ? e.start[r] : 0);
    for (int64_t col = (threadIdx.x % team) * V; col < d; col += (int64_t)team * V) {
        float acc[V];
#pragma unroll
        for (int k = 0; k < V; ++k) acc[k] = 0.f;
#pragma unroll 4
        for (int i = 0; i < c; ++i) {
            const bmt::Vec16<T> v = bmt::ld16(g + (int64_t)tok[i] * d + col);
#pragma unroll
            for (int k = 0; k < V; ++k) acc[k] += bmt::Cvt<T>::to_f(v.v[k]);
        }
        bmt::Vec16<T> o;
        if (ADD) o = bmt::ld16(out + r * d + col);
#pragma unroll
        for (int k = 0; k < V; ++k) o.v[k] = ADD ? plus(o.v[k], acc[k]) : bmt::Cvt<T>::from_f(acc[k]);
        bmt::st16(out + r * d + col, o);
    }
}
template <typename T, bool ADD>
__global__ void __launch_bounds__(256) emb_hot_kernel(int64_t d, const T* __restrict__ g, EmbScratch e, T* __restrict__ out) {
    bmt::after_previous();
    constexpr int V = bmt::Vec16<T>::N;
    __shared__ float part[8][32 * V];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t segs = (d + 32 * V - 1) / (32 * V), items = (int64_t)*e.n_hot * segs;
    for (int64_t it = blockIdx.x; it < items; it += gridDim.x) {
        const int64_t r = e.hot[it / segs], col = (it % segs) * 32 * V + lane * V;
        const int c = e.count[r];
        const int* __restrict__ tok = e.order + e.start[r];
        float acc[V];
#pragma unroll
        for (int k = 0; k < V; ++k) acc[k] = 0.f;
        if (col < d) {
#pragma unroll 4
            for (int i = warp; i < c; i += 8) {
                const bmt::Vec16<T> v = bmt::ld16(g + (int64_t)tok[i] * d + col);
#pragma unroll
                for (int k = 0; k < V; ++k) acc[k] += bmt::Cvt<T>::to_f(v.v[k]);
            }
        }
        __syncthreads();                       // the previous item's sums have been read
#pragma unroll
        for (int k = 0; k < V; ++k) part[warp][lane * V + k] = acc[k];
        __syncthreads();
        if (warp == 0 && col < d) {
            bmt::Vec16<T> o;
            if (ADD) o = bmt::ld16(out + r * d + col);
#pragma unroll
            for (int k = 0; k < V; ++k) {
                float s = 0.f;
#pragma unroll
                for (int w = 0; w < 8; ++w) s += part[w][lane * V + k];
                o.v[k] = ADD ? plus(o.v[k], s) : bmt::Cvt<T>::from_f(s);
            }
            bmt::st16(out + r * d + col, o);
        }
    }
}

template <typename T, bool ADD>
void launch_rows(int64_t tokens, int64_t rows, int64_t d, const int64_t* ids, const void* g, const EmbScratch& e, void* out, cudaStream_t s) {
    constexpr int V = bmt::Vec16<T>::N;
    int team = 32;
    while (team < 256 && (int64_t)team * V < d) team *= 2;
    const int per = 256 / team;
    const int64_t items = ADD ? tokens : rows;
    bmt::launch(emb_rows_kernel<T, ADD>, (unsigned)((items + per - 1) / per), 256, 0, s, 1, items, rows, d, team, ids, (const T*)g, e, (T*)out);
    if (tokens > EMB_HOT) bmt::launch(emb_hot_kernel<T, ADD>, 296, 256, 0, s, 1, d, (const T*)g, e, (T*)out);
}

}  // namespace

// Many rows of one vector a thread are launched normally: such a block lives for less than a microsecond, and waiting for the kernel before it takes
// as long (65536 tokens, rows of 1024 16-bit values: 49 us so, 68 when launched early; 8192 of 256: 8.3 and 9.2, 4096 alike; 65536 of 5120: 195 and 192).
extern "C" int bmt_embedding_fwd(int64_t tokens, int64_t d, const void* ids, const void* weight, int dtype, void* out, void* stream) {
    if (tokens <= 0) return 0;
    cudaStream_t s = (cudaStream_t)stream;
    const auto run = [&](auto* zero) {
        using T = std::remove_pointer_t<decltype(zero)>;
        constexpr int V = bmt::Vec16<T>::N;
        if (d % V) return -3;
        if (d <= 128 * V && tokens > 4096) emb_fwd_kernel<T, false><<<(unsigned)tokens, 128, 0, s>>>(d, (const int64_t*)ids, (const T*)weight, (T*)out);
        else bmt::launch(emb_fwd_kernel<T, true>, (unsigned)tokens, 128, 0, s, 1, d, (const int64_t*)ids, (const T*)weight, (T*)out);
        return 0;
    };
    const int rc = dtype == BMT_DT_F32 ? run((float*)nullptr) : dtype == BMT_DT_F16 ? run((__half*)nullptr) : run((__nv_bfloat16*)nullptr);
    if (rc) return rc;
    bmt_count_launch(1);
    return (int)cudaGetLastError();
}

// 32-bit words of scratch that bmt_embedding_bwd needs.
extern "C" int64_t bmt_embedding_bwd_scratch(int64_t tokens, int64_t rows) { return 2 + 2 * rows + emb_hot_cap(tokens) + 2 * tokens; }

extern "C" int bmt_embedding_bwd_ex(int64_t tokens, int64_t d, int64_t rows, const void* ids, const void* grad, int dtype, void* out,
                                    int accumulate, void* scratch, void* stream) {
    if (rows <= 0 || (accumulate && tokens <= 0)) return 0;
    if (d % (dtype == BMT_DT_F32 ? 4 : 8) || tokens > 0x7fffffff || rows > 0x7fffffff) return -3;
    cudaStream_t s = (cudaStream_t)stream;
    const EmbScratch e = emb_scratch(scratch, tokens, rows);
    BMT_CUDA_OK(cudaMemsetAsync(e.total, 0, (size_t)(2 + rows) * sizeof(int), s));
    if (tokens > 0) {
        const unsigned tb = (unsigned)((tokens + 255) / 256);
        bmt::launch(emb_count_kernel, tb, 256, 0, s, 1, tokens, rows, (const int64_t*)ids, e);
        bmt::launch(emb_start_kernel, (unsigned)((rows + 255) / 256), 256, 0, s, 1, rows, e);
        bmt::launch(emb_order_kernel, tb, 256, 0, s, 1, tokens, rows, (const int64_t*)ids, e);
        bmt_count_launch(3);
    }
    const auto run = [&](auto zero) {
        using T = decltype(zero);
        if (accumulate) launch_rows<T, true>(tokens, rows, d, (const int64_t*)ids, grad, e, out, s);
        else launch_rows<T, false>(tokens, rows, d, (const int64_t*)ids, grad, e, out, s);
    };
    if (dtype == BMT_DT_F32) run(0.f);
    else if (dtype == BMT_DT_F16) run(__half());
    else run(__nv_bfloat16());
    bmt_count_launch(tokens > EMB_HOT ? 2 : 1);
    return (int)cudaGetLastError();
}
