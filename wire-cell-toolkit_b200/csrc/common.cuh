// Shared device helpers for the DepoTransform kernels.
#pragma once

#include <cuda_runtime.h>
#include <cstdint>

namespace wctb200 {

__host__ __device__ __forceinline__ float2 cadd(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__host__ __device__ __forceinline__ float2 csub(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }
__host__ __device__ __forceinline__ float2 cmul(float2 a, float2 b)
{
    return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
// a * conj(b)
__host__ __device__ __forceinline__ float2 cmulc(float2 a, float2 b)
{
    return make_float2(a.x * b.x + a.y * b.y, a.y * b.x - a.x * b.y);
}
__host__ __device__ __forceinline__ float2 cconj(float2 a) { return make_float2(a.x, -a.y); }
__host__ __device__ __forceinline__ float2 cscale(float2 a, float s) { return make_float2(a.x * s, a.y * s); }
// multiply by -i (forward) or +i (inverse)
template <int SIGN>
__host__ __device__ __forceinline__ float2 cmul_i(float2 a)
{
    return SIGN < 0 ? make_float2(a.y, -a.x) : make_float2(-a.y, a.x);
}

// Order-preserving map of a double onto uint64 so atomicMin/atomicMax work on
// doubles bit-exactly (used for the reference's window min/max reductions).
__device__ __forceinline__ unsigned long long dkey(double v)
{
    unsigned long long u = (unsigned long long)__double_as_longlong(v);
    return (u & 0x8000000000000000ull) ? ~u : (u | 0x8000000000000000ull);
}
__host__ __device__ __forceinline__ double dkey_inv(unsigned long long k)
{
    unsigned long long u = (k & 0x8000000000000000ull) ? (k & 0x7fffffffffffffffull) : ~k;
#ifdef __CUDA_ARCH__
    return __longlong_as_double((long long)u);
#else
    double d;
    __builtin_memcpy(&d, &u, sizeof d);
    return d;
#endif
}

#ifdef __CUDACC__
// Whether a flagged charge wire lies within pad of wire W (all threads of the
// block call it): rows out of every charge's reach stay exactly zero, whatever
// rounding the convolution left in their spectra.
__device__ __forceinline__ bool row_reached(const unsigned char* __restrict__ flag, int nwires, int W, int pad)
{
    int any = 0;
    const int hi = min(nwires - 1, W + pad);
    for (int w = max(0, W - pad) + threadIdx.x; w <= hi; w += blockDim.x) any |= flag[w];
    return __syncthreads_or(any);
}

// Asynchronous 16-byte global -> shared copies (sm_80+ cp.async, no
// multicast): src_bytes = 0 fills the 16 bytes with zeros and reads nothing.
__device__ __forceinline__ void cp_async16(void* smem, const void* gmem, int src_bytes)
{
    const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(sa), "l"(gmem), "r"(src_bytes) : "memory");
}
// The 4-byte form.
__device__ __forceinline__ void cp_async4(void* smem, const void* gmem)
{
    const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(sa), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }
#endif

}  // namespace wctb200
