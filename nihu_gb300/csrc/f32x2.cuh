// Packed FP32 pairs: one instruction of sm_100 and later adds, multiplies or
// fuses two FP32 numbers, each rounded as by itself, in one issue slot.  An
// issue-bound FP32 kernel that works on two independent values per thread
// halves its arithmetic instructions with them.
#pragma once

#include <cuda_runtime.h>

namespace nihu {

struct f2 {
    unsigned long long v;  // low half: first value
};

__device__ __forceinline__ f2 f2_pack(float a, float b)
{
    f2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void f2_unpack(f2 x, float &a, float &b)
{
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(x.v));
}
__device__ __forceinline__ f2 f2_dup(float a) { return f2_pack(a, a); }
__device__ __forceinline__ f2 operator+(f2 a, f2 b)
{
    f2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ f2 operator*(f2 a, f2 b)
{
    f2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
// a b + c
__device__ __forceinline__ f2 f2_fma(f2 a, f2 b, f2 c)
{
    f2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
    return r;
}
__device__ __forceinline__ f2 f2_rsqrt(f2 x)
{
    float a, b;
    f2_unpack(x, a, b);
    return f2_pack(rsqrtf(a), rsqrtf(b));
}

// sincos_reduced (common.cuh) of two arguments: the nearest multiple of 2 pi by
// the rounding of the FP32 sum with 1.5 x 2^23
__device__ __forceinline__ void f2_sincos_reduced(f2 x, f2 &s, f2 &c)
{
    const f2 big = f2_dup(12582912.0f), nbig = f2_dup(-12582912.0f);
    const f2 n = f2_fma(x, f2_dup(0.159154943091895335769f), big) + nbig;
    float a, b, sa, sb, ca, cb;
    f2_unpack(f2_fma(f2_dup(-6.28318530717958647692f), n, x), a, b);
    __sincosf(a, &sa, &ca);
    __sincosf(b, &sb, &cb);
    s = f2_pack(sa, sb);
    c = f2_pack(ca, cb);
}

}  // namespace nihu
