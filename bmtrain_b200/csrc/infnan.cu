// Multi-tensor scans over gradient shards: inf/nan detection, sum of squares, in-place scaling.
// Replaces the reference's two-kernel-per-parameter any-reduce (csrc/cuda/has_inf_nan.cu:35-138) by one
// launch over up to 24 tensors with 128-bit loads; the flag is OR-ed with a single byte store.
#include "api.h"
#include "common.cuh"

namespace {

template <typename T> __device__ __forceinline__ bool bad(T v) {
    float f = bmt::Cvt<T>::to_f(v);
    return !(fabsf(f) <= 3.402823466e38f);  // true for inf and nan
}

// All three kernels walk the tensors as one list of chunks of THREADS * U 16-byte vectors, so a launch is as long as its bytes are,
// however they are spread over the tensors, and every thread has U loads in flight.  Bound by memory.  Measured on 300 M fp16 in eight
// tensors: scaling 543 -> 185 us (one element per load before; a block per chunk: a grid of resident blocks that loop loads, waits
// and stores in turn and copies at 0.92 of the rate); the scans 107 -> 92 us (resident blocks, so that there are few atomics; loads
// that leave no line in L1, 108 without that).
constexpr int THREADS = 256, SCAN_U = 8, SCAN_BLOCKS_PER_SM = 4, SCALE_U = 4;
constexpr int TABLE = sizeof(BmtPtrTable::p) / sizeof(void*);

struct ChunkTable {
    BmtPtrTable tab;
    int64_t first[TABLE + 1];   // chunk with which a tensor begins; the last entry in use is the number of chunks
};

// Elements before the first 16-byte boundary of a tensor: arbitrary sub-slices are taken.
template <typename T> __host__ __device__ __forceinline__ int64_t head_of(const void* p, int64_t n) {
    const int64_t head = (int64_t)(((16 - ((uintptr_t)p & 15)) & 15) / sizeof(T));
    return head < n ? head : n;
}

__device__ __forceinline__ void ld16_once(const void* p, void* to) {
    uint4 r;
    asm volatile("ld.global.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w) : "l"(p));
    *reinterpret_cast<uint4*>(to) = r;
}

// Calls `vec(pointer, data)` for every 16-byte vector and `one(pointer)` for the elements before and behind them.  `backwards` takes
// the chunks from the end.
template <typename T, int U, typename Vec, typename One>
__device__ __forceinline__ void walk(const ChunkTable& c, bool backwards, Vec vec, One one) {
    constexpr int V = bmt::Vec16<T>::N;
    const int64_t total = c.first[c.tab.count];
    for (int64_t k = blockIdx.x; k < total; k += gridDim.x) {
        const int64_t chunk = backwards ? total - 1 - k : k;
        int t = 0;
        while (c.first[t + 1] <= chunk) ++t;
        T* p = (T*)c.tab.p[t];
        const int64_t n = c.tab.n[t], head = head_of<T>(p, n), nvec = (n - head) / V;
        T* q = p + head;
        const int64_t v0 = (chunk - c.first[t]) * (THREADS * U) + threadIdx.x;
        bmt::Vec16<T> x[U];
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (v0 + u * THREADS < nvec) ld16_once(q + (v0 + u * THREADS) * V, &x[u]);
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (v0 + u * THREADS < nvec) vec(q + (v0 + u * THREADS) * V, x[u]);
        if (chunk == c.first[t]) {      // fewer than V elements on either side
            if ((int64_t)threadIdx.x < head) one(p + threadIdx.x);
            const int64_t tail = head + nvec * V + threadIdx.x;
            if (tail < n) one(p + tail);
        }
    }
}

template <typename T> __global__ void __launch_bounds__(THREADS) infnan_kernel(const __grid_constant__ ChunkTable c, unsigned char* out) {
    bool found = false;
    walk<T, SCAN_U>(c, false, [&](T*, const bmt::Vec16<T>& x) {
#pragma unroll
        for (int k = 0; k < bmt::Vec16<T>::N; ++k) found |= bad(x.v[k]);
    }, [&](T* p) { found |= bad(*p); });
    if (__syncthreads_or(found) && threadIdx.x == 0) *out = 1;
}

template <typename T> __global__ void __launch_bounds__(THREADS) sqnorm_kernel(const __grid_constant__ ChunkTable c, float* out) {
    __shared__ float scratch[33];
    float acc = 0.f;
    // a vector's squares come together first: added to the thread's sum one by one, some two thousand roundings of one sign were 1.4e-6 of
    // the result with 300 M fp16 values (now a few 1e-7)
    walk<T, SCAN_U>(c, false, [&](T*, const bmt::Vec16<T>& x) {
        constexpr int N = bmt::Vec16<T>::N;
        float s[N];
#pragma unroll
        for (int k = 0; k < N; ++k) s[k] = bmt::Cvt<T>::to_f(x.v[k]);
#pragma unroll
        for (int k = 0; k < N / 2; ++k) s[k] = fmaf(s[k], s[k], s[k + N / 2] * s[k + N / 2]);
#pragma unroll
        for (int n = N / 4; n > 0; n /= 2)
#pragma unroll
            for (int k = 0; k < n; ++k) s[k] += s[k + n];
        acc += s[0];
    }, [&](T* p) { const float f = bmt::Cvt<T>::to_f(*p); acc += f * f; });
    acc = bmt::block_allreduce<false>(acc, scratch);
    if (threadIdx.x == 0 && acc != 0.f) atomicAdd(out, acc);
}

// From the end: the norm has just been taken from the beginning, and the tail of what it read is still in L2; the overflow scan that
// follows finds the head there.
template <typename T> __global__ void __launch_bounds__(THREADS) scale_kernel(const __grid_constant__ ChunkTable c, const float* coef) {
    const float f = fminf(*coef, 1.f);
    if (f >= 1.f) return;
    walk<T, SCALE_U>(c, true, [&](T* p, bmt::Vec16<T>& x) {
#pragma unroll
        for (int k = 0; k < bmt::Vec16<T>::N; ++k) x.v[k] = bmt::Cvt<T>::from_f(bmt::Cvt<T>::to_f(x.v[k]) * f);
        bmt::st16(p, x);
    }, [&](T* p) { *p = bmt::Cvt<T>::from_f(bmt::Cvt<T>::to_f(*p) * f); });
}

// Zeros, by bytes.  Bound by the writes: 412 MB in one tensor 107 us with the framework's fill, 58 here.
__global__ void __launch_bounds__(THREADS) zero_kernel(const __grid_constant__ ChunkTable c) {
    const int64_t total = c.first[c.tab.count];
    for (int64_t k = blockIdx.x; k < total; k += gridDim.x) {
        int t = 0;
        while (c.first[t + 1] <= k) ++t;
        uint8_t* p = (uint8_t*)c.tab.p[t];
        const int64_t n = c.tab.n[t], head = head_of<uint8_t>(p, n), nvec = (n - head) / 16, v0 = (k - c.first[t]) * (THREADS * SCALE_U) + threadIdx.x;
#pragma unroll
        for (int u = 0; u < SCALE_U; ++u)
            if (v0 + u * THREADS < nvec) reinterpret_cast<uint4*>(p + head)[v0 + u * THREADS] = make_uint4(0, 0, 0, 0);
        if (k == c.first[t]) {          // fewer than 16 bytes on either side
            const int64_t tail = head + nvec * 16;
            if ((int64_t)threadIdx.x < head) p[threadIdx.x] = 0;
            if (tail + threadIdx.x < n) p[tail + threadIdx.x] = 0;
        }
    }
}

template <typename T> ChunkTable chunks_of(const BmtPtrTable* tab, int vectors) {
    ChunkTable c;
    c.tab = *tab;
    c.first[0] = 0;
    for (int i = 0; i < tab->count; ++i) {
        const int64_t n = tab->n[i] > 0 ? tab->n[i] : 0, nvec = (n - head_of<T>(tab->p[i], n)) / bmt::Vec16<T>::N;
        const int64_t chunks = bmt::ceil_div64(nvec, vectors);
        c.first[i + 1] = c.first[i] + (n == 0 ? 0 : chunks > 1 ? chunks : 1);
    }
    return c;
}

// `most`: blocks of the grid at most
template <typename T, typename Out>
int run(void (*kernel)(const ChunkTable, Out*), const BmtPtrTable* tab, int vectors, int64_t most, Out* out, void* stream) {
    const ChunkTable c = chunks_of<T>(tab, vectors);
    const int64_t total = c.first[tab->count];
    if (total == 0) return 0;
    kernel<<<(unsigned)(total < most ? total : most), THREADS, 0, (cudaStream_t)stream>>>(c, out);
    bmt_count_launch(1);
    return (int)cudaGetLastError();
}

template <typename T, typename Out> int scan(void (*kernel)(const ChunkTable, Out*), const BmtPtrTable* tab, Out* out, void* stream) {
    return run<T>(kernel, tab, THREADS * SCAN_U, (int64_t)bmt::sm_count() * SCAN_BLOCKS_PER_SM, out, stream);
}
template <typename T> int scale(const BmtPtrTable* tab, const float* coef, void* stream) {
    return run<T>(scale_kernel<T>, tab, THREADS * SCALE_U, INT32_MAX, coef, stream);
}

}  // namespace

extern "C" int bmt_has_inf_nan_multi(const BmtPtrTable* tab, int dtype, void* out, void* stream) {
    if (tab->count <= 0) return 0;
    unsigned char* o = (unsigned char*)out;
    if (dtype == BMT_DT_F16) return scan<__half>(infnan_kernel<__half>, tab, o, stream);
    if (dtype == BMT_DT_BF16) return scan<__nv_bfloat16>(infnan_kernel<__nv_bfloat16>, tab, o, stream);
    return scan<float>(infnan_kernel<float>, tab, o, stream);
}

extern "C" int bmt_sq_norm_multi(const BmtPtrTable* tab, int dtype, void* out, void* stream) {
    if (tab->count <= 0) return 0;
    float* o = (float*)out;
    if (dtype == BMT_DT_F16) return scan<__half>(sqnorm_kernel<__half>, tab, o, stream);
    if (dtype == BMT_DT_BF16) return scan<__nv_bfloat16>(sqnorm_kernel<__nv_bfloat16>, tab, o, stream);
    return scan<float>(sqnorm_kernel<float>, tab, o, stream);
}

extern "C" int bmt_scale_multi(const BmtPtrTable* tab, int dtype, const void* coef, void* stream) {
    if (tab->count <= 0) return 0;
    const float* o = (const float*)coef;
    if (dtype == BMT_DT_F16) return scale<__half>(tab, o, stream);
    if (dtype == BMT_DT_BF16) return scale<__nv_bfloat16>(tab, o, stream);
    return scale<float>(tab, o, stream);
}

// tab->n: bytes
extern "C" int bmt_zero_multi(const BmtPtrTable* tab, void* stream) {
    if (tab->count <= 0) return 0;
    const ChunkTable c = chunks_of<uint8_t>(tab, THREADS * SCALE_U);
    const int64_t total = c.first[tab->count];
    if (total == 0) return 0;
    zero_kernel<<<(unsigned)(total < INT32_MAX ? total : INT32_MAX), THREADS, 0, (cudaStream_t)stream>>>(c);
    bmt_count_launch(1);
    return (int)cudaGetLastError();
}
