// Shared device helpers for the sm_100a kernels: dtype traits, 128-bit vector
// access, warp / block reductions.  (Reference counterpart: csrc/cuda/reduce.cuh,
// which offers shuffle + 32-float shared-memory block reductions only.)
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#define BMT_DT_F16 0
#define BMT_DT_BF16 1
#define BMT_DT_F32 2

namespace bmt {

template <typename T> struct Cvt;
template <> struct Cvt<__half> {
    static __device__ __forceinline__ float to_f(__half v) { return __half2float(v); }
    static __device__ __forceinline__ __half from_f(float v) { return __float2half_rn(v); }
};
template <> struct Cvt<__nv_bfloat16> {
    static __device__ __forceinline__ float to_f(__nv_bfloat16 v) { return __bfloat162float(v); }
    static __device__ __forceinline__ __nv_bfloat16 from_f(float v) { return __float2bfloat16_rn(v); }
};
template <> struct Cvt<float> {
    static __device__ __forceinline__ float to_f(float v) { return v; }
    static __device__ __forceinline__ float from_f(float v) { return v; }
};

// A 16-byte packet of T (8 halves or 4 floats).
template <typename T> struct alignas(16) Vec16 {
    static constexpr int N = 16 / sizeof(T);
    T v[N];
};

template <typename T> __device__ __forceinline__ Vec16<T> ld16(const T* p) {
    return *reinterpret_cast<const Vec16<T>*>(p);
}
template <typename T> __device__ __forceinline__ void st16(T* p, const Vec16<T>& x) {
    *reinterpret_cast<Vec16<T>*>(p) = x;
}

// Two fp32 multiply-adds / adds in one instruction.
__device__ __forceinline__ uint64_t pack_f2(float a, float b) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void unpack_f2(uint64_t v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ uint64_t fma_f2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ uint64_t add_f2(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ uint64_t mul_f2(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
// Two 16-bit values that lie next to one another as a pair of fp32 values, and back.
template <typename T> __device__ __forceinline__ uint64_t to_f2(uint32_t two);
template <> __device__ __forceinline__ uint64_t to_f2<__half>(uint32_t two) {
    const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&two));
    return pack_f2(f.x, f.y);
}
template <> __device__ __forceinline__ uint64_t to_f2<__nv_bfloat16>(uint32_t two) {
    return pack_f2(__uint_as_float(two << 16), __uint_as_float(two & 0xffff0000u));
}
template <typename T> __device__ __forceinline__ uint32_t pack2(float a, float b);
template <> __device__ __forceinline__ uint32_t pack2<__half>(float a, float b) {
    __half2 h = __floats2half2_rn(a, b);
    return *reinterpret_cast<uint32_t*>(&h);
}
template <> __device__ __forceinline__ uint32_t pack2<__nv_bfloat16>(float a, float b) {
    __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<uint32_t*>(&h);
}
template <typename T> __device__ __forceinline__ uint32_t from_f2(uint64_t v) {
    float a, b;
    unpack_f2(v, a, b);
    return pack2<T>(a, b);
}
__device__ __forceinline__ float sum_f2(uint64_t v) {
    float a, b;
    unpack_f2(v, a, b);
    return a + b;
}

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// Block-wide all-reduce (every thread gets the result). `scratch` holds >= 33 floats.
template <bool IsMax> __device__ __forceinline__ float block_allreduce(float v, float* scratch) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = (blockDim.x + 31) >> 5;
    v = IsMax ? warp_max(v) : warp_sum(v);
    __syncthreads();  // scratch may still be read from a previous call
    if (lane == 0) scratch[warp] = v;
    __syncthreads();
    float r = (lane < nwarp) ? scratch[lane] : (IsMax ? -INFINITY : 0.f);
    r = IsMax ? warp_max(r) : warp_sum(r);
    return r;
}

__device__ __forceinline__ float rcp_approx_ftz(float x) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ float ex2_approx(float x) {
    float r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
// GELU.  The normal distribution function comes in two forms, neither with erff, which sets the pace of what uses it:
// Below 1.3: Phi(x) = 1/2 + x P(x^2), P fitted for this file in 64 bits behind its first coefficient, as that is rounded, weighted for the relative
// error of Phi on the negative side (3e-9).
// Above: Phi(-u) = t 2^(q(t)) exp(-u^2 / 2), t = 1 / (1 + 0.3 u), q fitted for this file in 64 bits (the form of the complementary error function in
// Press et al., Numerical Recipes, 6.2; largest error 7e-8).  It keeps its relative accuracy on the negative side (2e-6 at -5, where
// 1 + erf(x / sqrt 2) has 6e-2), but for small u it has errors of 5e-7.
// Largest errors between -1.3 and 1.3, as with erff: x Phi(x) 3.5e-7 relative, Phi(x) + x phi(x) 1.4e-7 absolute.
// One value or a pair at a time: pairs issue half as much, single ones take the constants as operands of the instructions (in pairs they sit in 30
// registers, which the GEMM's epilogue does not have: all forms of it took 2 % longer).
constexpr float HALF_LOG2E = 0.7213475204444817f, NORMAL_NEAR = 1.3f;
template <typename V> struct Lanes;
template <> struct Lanes<float> {
    static __device__ __forceinline__ float all(float a) { return a; }
    static __device__ __forceinline__ float fma(float a, float b, float c) { return fmaf(a, b, c); }
    static __device__ __forceinline__ float mul(float a, float b) { return __fmul_rn(a, b); }
    static __device__ __forceinline__ float abs(float a) { return fabsf(a); }
    static __device__ __forceinline__ float ex2(float a) { return ex2_approx(a); }
    static __device__ __forceinline__ float rcp(float a) { return rcp_approx_ftz(a); }
    // Phi(x) of its two forms: near(x), far(-|x|)
    static __device__ __forceinline__ float pick(float x, float near, float far) { return fabsf(x) < NORMAL_NEAR ? near : x >= 0.f ? 1.f - far : far; }
};
template <> struct Lanes<uint64_t> {
    typedef Lanes<float> One;
    template <typename F> static __device__ __forceinline__ uint64_t each(uint64_t v, F f) {
        float a, b;
        unpack_f2(v, a, b);
        return pack_f2(f(a), f(b));
    }
    static __device__ __forceinline__ uint64_t all(float a) { return pack_f2(a, a); }
    static __device__ __forceinline__ uint64_t fma(uint64_t a, uint64_t b, uint64_t c) { return fma_f2(a, b, c); }
    static __device__ __forceinline__ uint64_t mul(uint64_t a, uint64_t b) { return mul_f2(a, b); }
    static __device__ __forceinline__ uint64_t abs(uint64_t a) { return a & 0x7fffffff7fffffffull; }
    static __device__ __forceinline__ uint64_t ex2(uint64_t v) { return each(v, [](float a) { return ex2_approx(a); }); }
    static __device__ __forceinline__ uint64_t rcp(uint64_t v) { return each(v, [](float a) { return rcp_approx_ftz(a); }); }
    static __device__ __forceinline__ uint64_t pick(uint64_t x, uint64_t near, uint64_t far) {
        float a, b, na, nb, fa, fb;
        unpack_f2(x, a, b);
        unpack_f2(near, na, nb);
        unpack_f2(far, fa, fb);
        return pack_f2(One::pick(a, na, fa), One::pick(b, nb, fb));
    }
};
template <typename V> __device__ __forceinline__ V normal_near(V x) {
    typedef Lanes<V> L;
    const V s = L::mul(x, x);
    V p = L::all(5.271343753e-07f);
    p = L::fma(p, s, L::all(-9.379426047e-06f));
    p = L::fma(p, s, L::all(1.158123778e-04f));
    p = L::fma(p, s, L::all(-1.188031165e-03f));
    p = L::fma(p, s, L::all(9.974041022e-03f));
    p = L::fma(p, s, L::all(-6.649051607e-02f));
    p = L::fma(p, s, L::all(0.39894229173660278f));
    return L::fma(x, p, L::all(0.5f));
}
template <typename V> __device__ __forceinline__ V normal_far_log2(V t) {     // q, in units of log 2
    typedef Lanes<V> L;
    V q = L::all(0.1297198086977005f);
    q = L::fma(q, t, L::all(-0.041672442108392715f));
    q = L::fma(q, t, L::all(-0.49322715401649475f));
    q = L::fma(q, t, L::all(0.32053878903388977f));
    q = L::fma(q, t, L::all(0.087591201066970825f));
    q = L::fma(q, t, L::all(0.62215578556060791f));
    q = L::fma(q, t, L::all(1.4390027523040771f));
    return L::fma(q, t, L::all(-3.0625312328338623f));
}
// x Phi(x)
template <typename V> __device__ __forceinline__ V gelu(V x) {
    typedef Lanes<V> L;
    const V u = L::abs(x), t = L::rcp(L::fma(u, L::all(0.3f), L::all(1.f)));
    const V far = L::mul(t, L::ex2(L::fma(L::mul(u, L::all(-HALF_LOG2E)), u, normal_far_log2(t))));
    return L::mul(x, L::pick(x, normal_near(x), far));
}
// Phi(x) + x phi(x)
template <typename V> __device__ __forceinline__ V gelu_grad(V x) {
    typedef Lanes<V> L;
    const V u = L::abs(x), t = L::rcp(L::fma(u, L::all(0.3f), L::all(1.f))), e = L::ex2(L::mul(L::mul(u, L::all(-HALF_LOG2E)), u));
    const V far = L::mul(L::mul(t, e), L::ex2(normal_far_log2(t)));
    return L::fma(L::mul(x, L::all(0.3989422804014327f)), e, L::pick(x, normal_near(x), far));
}

// ---- dependent launches -------------------------------------------------------------------------------------------------------
// Kernels launched with `launch` may start while the kernel before them on the stream is still running: their CTAs take the SMs that
// it leaves, set up what does not touch global memory, and wait in `after_previous` until it has completed and its writes are visible.
// Every thread of such a kernel calls `after_previous` before its first access to global memory, and after it has allocated what it
// needs of the SM (tensor memory), since it also lets the next kernel begin.  A GEMM after a GEMM begins 2 us earlier this way
// (256 x 768 x 256: 6.2 -> 4.8 us from start to start, 1024 x 2560 x 2560: 18.5 -> 16.0).  Not for grids of resident CTAs that stride over
// their work with several to an SM: they count on being spread evenly, and CTAs that arrive while others still hold SMs pile up
// on the free ones (RMSNorm 16384 x 5120, both directions: 187 -> 204 us).  Those are launched normally and only let the next begin.
__device__ __forceinline__ void after_previous() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

template <typename... P, typename... A>
inline cudaError_t launch(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, int cluster, A&&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid; cfg.blockDim = block; cfg.dynamicSmemBytes = smem; cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = (unsigned)cluster; attr[1].val.clusterDim.y = 1; attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr; cfg.numAttrs = cluster > 1 ? 2 : 1;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

// SMs of the current device (148 on a B200, also where there is none to ask).
inline int sm_count() {
    static int sms[64] = {0};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 148;
    if (sms[dev] == 0 && cudaDeviceGetAttribute(&sms[dev], cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 148;
    return sms[dev];
}

__host__ __device__ __forceinline__ int64_t ceil_div64(int64_t a, int64_t b) { return (a + b - 1) / b; }

}  // namespace bmt

#define BMT_CUDA_OK(expr)                        \
    do {                                         \
        cudaError_t _e = (expr);                 \
        if (_e != cudaSuccess) return (int)_e;   \
    } while (0)
