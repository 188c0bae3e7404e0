// Common device helpers for the cTDM GB300 kernels.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#define CTDM_PI_F 3.14159265358979323846f
#define CTDM_PI_D 3.14159265358979323846

__device__ __forceinline__ float2 cadd(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float2 csub(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ float2 cmul(float2 a, float2 b)
{
    return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
// a * conj(b)
__device__ __forceinline__ float2 cmulc(float2 a, float2 b)
{
    return make_float2(a.x * b.x + a.y * b.y, a.y * b.x - a.x * b.y);
}
__device__ __forceinline__ float2 cscale(float2 a, float s) { return make_float2(a.x * s, a.y * s); }
// multiply by -i (forward) or +i (inverse)
template <bool INV>
__device__ __forceinline__ float2 cmul_mi(float2 a)
{
    return INV ? make_float2(-a.y, a.x) : make_float2(a.y, -a.x);
}

// The same pointer, opaque to the compiler: loads through it stay behind this point (see
// chain_begin), and in a loop over line batches, where every thread's twiddles are
// loop-invariant, they are not kept in registers across it (15 complex values per radix-16
// stage cost more than reloading them from L1).
template <class T>
__device__ __forceinline__ T *fresh(T *p)
{
    asm volatile("" : "+l"(p));
    return p;
}

__device__ __forceinline__ int imod(int a, int b)
{
    int r = a % b;
    return r < 0 ? r + b : r;
}
