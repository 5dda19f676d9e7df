// Float-float arithmetic: a value is the unevaluated sum h + l of two FP32
// numbers with |l| <= ulp(h) / 2, about 48 significand bits (Dekker 1971,
// Knuth's two-sum).
//
// GB300 issues 128 FP32 operations per SM and cycle but only 2 FP64 ones, so
// a float-float product (7 FP32 instructions) or sum (11) costs 0.05 - 0.09
// of the SM's time of one FP64 instruction.  Sums whose result is rounded to
// FP32, and which FP32 alone would leave with cancellation error, are formed
// here: the functions below hold about 1e-12 relative (sin, cos, log and the
// angle) or better, four orders below the rounding of an FP32 result.
//
// The additions and products are written with the rounding intrinsics, so
// that no contraction to a fused multiply-add changes the error terms.
#pragma once

#include <cuda_runtime.h>

#include "common.cuh"

namespace nihu {

struct ff {
    float h, l;
};

__device__ __forceinline__ ff ff_quick(float a, float b)  // |a| >= |b| or a = 0
{
    const float s = __fadd_rn(a, b);
    return {s, __fsub_rn(b, __fsub_rn(s, a))};
}

__device__ __forceinline__ ff ff_two_sum(float a, float b)
{
    const float s = __fadd_rn(a, b);
    const float bb = __fsub_rn(s, a);
    return {s, __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb))};
}

__device__ __forceinline__ ff ff_two_prod(float a, float b)
{
    const float p = __fmul_rn(a, b);
    return {p, __fmaf_rn(a, b, -p)};
}

__device__ __forceinline__ ff ff_from(double x)
{
    const float h = (float)x;
    return {h, (float)(x - (double)h)};
}

__device__ __forceinline__ double ff_double(ff a) { return (double)a.h + (double)a.l; }
__device__ __forceinline__ ff ff_neg(ff a) { return {-a.h, -a.l}; }
// times a power of two (exact)
__device__ __forceinline__ ff ff_scale(ff a, float s) { return {a.h * s, a.l * s}; }

__device__ __forceinline__ ff ff_add(ff a, ff b)
{
    const ff s = ff_two_sum(a.h, b.h);
    return ff_quick(s.h, __fadd_rn(s.l, __fadd_rn(a.l, b.l)));
}

__device__ __forceinline__ ff ff_sub(ff a, ff b) { return ff_add(a, ff_neg(b)); }

__device__ __forceinline__ ff ff_mul(ff a, ff b)
{
    const ff p = ff_two_prod(a.h, b.h);
    return ff_quick(p.h, __fmaf_rn(a.h, b.l, __fmaf_rn(a.l, b.h, p.l)));
}

// 1 / a: the FP32 reciprocal and one Newton step on the float-float residual
__device__ __forceinline__ ff ff_recip(ff a)
{
    const float y = __fdividef(1.0f, a.h);
    const float r = __fmaf_rn(-a.l, y, __fmaf_rn(-a.h, y, 1.0f));
    return ff_quick(y, __fmul_rn(y, __fmaf_rn(r, r, r)));
}

// 1 / sqrt(a), a > 0: rsqrtf and one Newton step
__device__ __forceinline__ ff ff_rsqrt(ff a)
{
    const float y = rsqrtf(a.h);
    const ff p = ff_mul(a, ff_two_prod(y, y));
    const float r = __fsub_rn(__fsub_rn(1.0f, p.h), p.l);
    return ff_quick(y, __fmul_rn(y, __fmul_rn(r, __fmaf_rn(0.375f, r, 0.5f))));
}

// sin and cos of n / 16, n = 0..26, and 1 / c, -log(1 / c) of the FP32
// reciprocals 1 / c of c = 1 + (i + 1/2) / 128, i = 0..127, as float-float
// (Taylor series and the atanh series, summed in FP64 at compile time)
struct FfTables {
    float4 sc[27];   // (sin hi, sin lo, cos hi, cos lo)
    float4 lg[128];  // (1/c, log hi, log lo, 0)
    constexpr FfTables() : sc(), lg()
    {
        for (int n = 0; n < 27; ++n) {
            const double x = n / 16.0;
            double s = 0.0, c = 0.0, t = 1.0;
            for (int k = 0; k < 30; ++k) {  // t = x^k / k!
                const double g = (k & 2) ? -t : t;
                if (k & 1) s += g;
                else c += g;
                t *= x / (k + 1);
            }
            sc[n].x = (float)s;
            sc[n].y = (float)(s - (double)(float)s);
            sc[n].z = (float)c;
            sc[n].w = (float)(c - (double)(float)c);
        }
        for (int i = 0; i < 128; ++i) {
            const float ic = (float)(1.0 / (1.0 + (i + 0.5) / 128.0));
            const double z = (1.0 - (double)ic) / (1.0 + (double)ic);  // -log(ic) = 2 atanh z
            double l = 0.0, p = z;
            for (int k = 0; k < 30; ++k) {
                l += 2.0 * p / (2 * k + 1);
                p *= z * z;
            }
            lg[i].x = ic;
            lg[i].y = (float)l;
            lg[i].z = (float)(l - (double)(float)l);
            lg[i].w = 0.0f;
        }
    }
};
static __device__ const FfTables FF_TAB{};

// sin and cos for |x| <= 1.6: x = n / 16 + r, |r| <= 1/32 (r exact), the
// series of r with its small terms in FP32, and the table's sin and cos of n / 16
__device__ __forceinline__ void ff_sincos(ff x, ff &s, ff &c)
{
    const float n = rintf(x.h * 16.0f);
    const float r = __fmaf_rn(-0.0625f, n, x.h);
    const float4 t = FF_TAB.sc[(int)fabsf(n)];
    const float sg = n < 0.0f ? -1.0f : 1.0f;
    const ff S{t.x * sg, t.y * sg}, C{t.z, t.w};
    const ff p = ff_two_prod(r, r);
    const float corr = __fmul_rn(__fmul_rn(r, p.h), __fmaf_rn(p.h, 1.0f / 120.0f, -1.0f / 6.0f));
    const ff sr = ff_quick(r, __fadd_rn(corr, __fmaf_rn(-0.5f * p.h, x.l, x.l)));
    const ff cm = ff_quick(-0.5f * p.h, __fmaf_rn(__fmul_rn(p.h, p.h), __fmaf_rn(p.h, -1.0f / 720.0f, 1.0f / 24.0f),
                                                 __fmaf_rn(-r, x.l, -0.5f * p.l)));
    s = ff_add(S, ff_add(ff_mul(S, cm), ff_mul(C, sr)));
    c = ff_add(C, ff_sub(ff_mul(C, cm), ff_mul(S, sr)));
}

// atan2(u, s) for s >= 0, the angle in [-pi/2, pi/2] (0 for u = s = 0): the
// FP32 angle a and the rotation of (s, u) by -a, whose remaining angle is
// below 1e-6 (its tangent differs from it by less than 1e-18)
__device__ __forceinline__ ff ff_angle(ff u, ff s)
{
    const float a = atan2f(u.h, s.h);
    ff sa, ca;
    ff_sincos(ff{a, 0.0f}, sa, ca);
    const ff num = ff_sub(ff_mul(u, ca), ff_mul(s, sa));
    const float den = __fmaf_rn(s.h, ca.h, u.h * sa.h);
    return ff_quick(a, den > 0.0f ? num.h / den : 0.0f);
}

// log(v 2^e) for v > 0: v = 2^k m, m / c - 1 = r exactly formed, |r| <= 1/256
__device__ __forceinline__ ff ff_log(ff v, int e)
{
    const int b = __float_as_int(v.h);
    const int k = (b >> 23) - 127;
    const float m = __int_as_float((b & 0x007fffff) | 0x3f800000);
    const float sc = __int_as_float((127 - k) << 23);  // 2^-k
    const float4 t = FF_TAB.lg[(b >> 16) & 127];
    const ff p = ff_two_prod(m, t.x);
    const ff r = ff_quick(__fsub_rn(p.h, 1.0f), __fmaf_rn(v.l * sc, t.x, p.l));
    const float tail = __fmul_rn(__fmul_rn(r.h, r.h),
                                 __fmaf_rn(r.h, __fmaf_rn(r.h, __fmaf_rn(r.h, 0.2f, -0.25f), 1.0f / 3.0f), -0.5f));
    // ln 2 in 13 + 24 bits: n LN2_HI is exact for |n| < 2^11
    constexpr float LN2_HI = 0.693115234375f;  // 5678 / 8192
    constexpr float LN2_LO = (float)(0.69314718055994530942 - 0.693115234375);
    constexpr float LN2_LO2 = (float)(0.69314718055994530942 - 0.693115234375 - (double)LN2_LO);
    const float n = (float)(k + e);
    const ff ln = ff_add(ff{n * LN2_HI, 0.0f}, ff_add(ff_two_prod(n, LN2_LO), ff{n * LN2_LO2, 0.0f}));
    return ff_add(ff_add(ln, ff{t.y, t.z}), ff_quick(r.h, __fadd_rn(r.l, tail)));
}

// sin and cos of any x of moderate size: x less the nearest multiple n of pi/2
// in three parts (exact products for |n| < 2^9), then ff_sincos and the quadrant
__device__ __forceinline__ void ff_sincos_any(ff x, ff &s, ff &c)
{
    constexpr double HP = 1.57079632679489661923;
    constexpr float P1 = 1.5703125f;  // 201 / 128
    constexpr float P2 = (float)(HP - 1.5703125);
    constexpr float P3 = (float)(HP - 1.5703125 - (double)P2);
    const float n = rintf(x.h * 0.636619772367581343f);
    ff r = ff_add(x, ff{__fmul_rn(-n, P1), 0.0f});
    r = ff_add(r, ff_two_prod(-n, P2));
    r = ff_add(r, ff{__fmul_rn(-n, P3), 0.0f});
    ff sr, cr;
    ff_sincos(r, sr, cr);
    const int q = (int)n & 3;
    s = (q & 1) ? cr : sr;
    c = (q & 1) ? sr : cr;
    if (q & 2) s = ff_neg(s);
    if (q == 1 || q == 2) c = ff_neg(c);
}

// e^x for |x| < 80: x = n ln 2 / 16 + f, |f| <= ln 2 / 32, the 16 powers
// 2^{j/16} from a table, the series of f with its small terms in FP32
struct FfExp2 {
    float h[16], l[16];
    constexpr FfExp2() : h(), l()
    {
        for (int j = 0; j < 16; ++j) {
            const double x = 0.69314718055994530942 * j / 16.0;
            double v = 0.0, t = 1.0;
            for (int k = 0; k < 30; ++k) {
                v += t;
                t *= x / (k + 1);
            }
            h[j] = (float)v;
            l[j] = (float)(v - (double)(float)v);
        }
    }
};
static __device__ const FfExp2 FF_EXP2{};

__device__ __forceinline__ ff ff_exp(ff x)
{
    constexpr double L = 0.69314718055994530942 / 16.0;
    constexpr float L1 = 0.043304443359375f;  // 1419 / 32768
    constexpr float L2 = (float)(L - 0.043304443359375);
    constexpr float L3 = (float)(L - 0.043304443359375 - (double)L2);
    const float n = rintf(x.h * 23.0831206542234142f);
    ff f = ff_add(x, ff{__fmul_rn(-n, L1), 0.0f});
    f = ff_add(f, ff_two_prod(-n, L2));
    f = ff_add(f, ff{__fmul_rn(-n, L3), 0.0f});
    const ff f2 = ff_mul(f, f);
    const float tail = __fmul_rn(__fmul_rn(f2.h, f.h),
                                 __fmaf_rn(f.h, __fmaf_rn(f.h, 1.0f / 120.0f, 1.0f / 24.0f), 1.0f / 6.0f));
    const ff em1 = ff_add(f, ff_quick(0.5f * f2.h, __fadd_rn(0.5f * f2.l, tail)));  // e^f - 1
    const int i = (int)n, j = i & 15;
    const ff t{FF_EXP2.h[j], FF_EXP2.l[j]};
    return ff_scale(ff_add(t, ff_mul(t, em1)), __int_as_float(((i >> 4) + 127) << 23));
}

// an n-point Gauss-Legendre rule's non-negative half as float-float:
// nodes x (decreasing) and weights, the last node 0 when n is odd
template <int N>
struct GaussHalfFF {
    static constexpr int HALF = N / 2;
    float xh[(N + 1) / 2], xl[(N + 1) / 2], wh[(N + 1) / 2], wl[(N + 1) / 2];
    constexpr GaussHalfFF() : xh(), xl(), wh(), wl()
    {
        constexpr double d[NIHU_GAUSS_DATA_LEN] = NIHU_GAUSS_DATA;
        constexpr int off[NIHU_GAUSS_MAX_N] = NIHU_GAUSS_OFFSETS;
        for (int q = 0; q < (N + 1) / 2; ++q) {
            const double x = q == HALF ? 0.0 : d[2 * (off[N - 1] + N - 1 - q)], w = d[2 * (off[N - 1] + N - 1 - q) + 1];
            xh[q] = (float)x;
            xl[q] = (float)(x - (double)(float)x);
            wh[q] = (float)w;
            wl[q] = (float)(w - (double)(float)w);
        }
    }
};
// the 42-point degree-14 triangle rule: (xi hi, xi lo, eta hi, eta lo) and (w hi, w lo)
struct Tri14FF {
    float4 x[42];
    float2 w[42];
    constexpr Tri14FF() : x(), w()
    {
        constexpr double d[NIHU_TRI_DATA_LEN] = NIHU_TRI_DATA;
        constexpr int off[15] = NIHU_TRI_OFFSETS;
        for (int q = 0; q < 42; ++q) {
            const double a = d[3 * (off[14] + q)], b = d[3 * (off[14] + q) + 1], c = d[3 * (off[14] + q) + 2];
            x[q].x = (float)a;
            x[q].y = (float)(a - (double)(float)a);
            x[q].z = (float)b;
            x[q].w = (float)(b - (double)(float)b);
            w[q].x = (float)c;
            w[q].y = (float)(c - (double)(float)c);
        }
    }
};
static __device__ const Tri14FF TRI14_FF{};

static __device__ const GaussHalfFF<6> GAUSS6_FF{};
static __device__ const GaussHalfFF<8> GAUSS8_FF{};
static __device__ const GaussHalfFF<21> GAUSS21_FF{};

}  // namespace nihu
