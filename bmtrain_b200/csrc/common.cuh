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
