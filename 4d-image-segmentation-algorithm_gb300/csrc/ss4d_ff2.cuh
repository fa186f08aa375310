// ss4d_ff2.cuh — float-float arithmetic on two values at a time with the
// packed FP32 instructions (add/sub/mul/fma.rn.f32x2, two FP32 results per
// instruction, each rounded as the scalar instruction rounds it).  A probe on
// GB300 gave 128 FP32 results per clock and SM either way, but the packed form issues half the
// instructions, and the float-float kernels are bound by issue: their loads,
// index arithmetic and integer work (62 to 97 results per clock) share the
// slots.  The formulas are those of ss4d_ff.cuh.
#pragma once

#include "ss4d_ff.cuh"

namespace ss4d {
namespace ffa {

// two floats in one 64-bit register pair
struct f2 {
    unsigned long long v;
};

__device__ __forceinline__ f2 mk2(float a, float b)
{
    f2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float lo2(f2 a)
{
    float x, y;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(a.v));
    return x;
}
__device__ __forceinline__ float hi2(f2 a)
{
    float x, y;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(a.v));
    return y;
}
__device__ __forceinline__ f2 both(float a)
{
    return mk2(a, a);
}
__device__ __forceinline__ f2 add2(f2 a, f2 b)
{
    f2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ f2 sub2(f2 a, f2 b)
{
    f2 r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ f2 mul2(f2 a, f2 b)
{
    f2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c)
{
    f2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
    return r;
}
__device__ __forceinline__ f2 neg2(f2 a)
{
    return mk2(-lo2(a), -hi2(a));
}

// two float-float values
struct ff2 {
    f2 h, l;
};

__device__ __forceinline__ ff2 both(ff a)
{
    return ff2{both(a.h), both(a.l)};
}
__device__ __forceinline__ ff2 neg2(ff2 a)
{
    return ff2{neg2(a.h), neg2(a.l)};
}
// |a| >= |b| (or a == 0)
__device__ __forceinline__ ff2 fast_two_sum2(f2 a, f2 b)
{
    const f2 s = add2(a, b);
    return ff2{s, sub2(b, sub2(s, a))};
}
__device__ __forceinline__ ff2 two_sum2(f2 a, f2 b)
{
    const f2 s = add2(a, b), v = sub2(s, a);
    return ff2{s, add2(sub2(a, sub2(s, v)), sub2(b, v))};
}
__device__ __forceinline__ ff2 two_diff2(f2 a, f2 b)
{
    const f2 s = sub2(a, b), v = sub2(s, a);
    return ff2{s, sub2(sub2(a, sub2(s, v)), add2(b, v))};
}
__device__ __forceinline__ ff2 ff_add2(ff2 a, ff2 b)
{
    const ff2 s = two_sum2(a.h, b.h);
    return fast_two_sum2(s.h, add2(s.l, add2(a.l, b.l)));
}
__device__ __forceinline__ ff2 ff_sub2(ff2 a, ff2 b)
{
    const ff2 s = two_diff2(a.h, b.h);
    return fast_two_sum2(s.h, add2(s.l, sub2(a.l, b.l)));
}
// without renormalising (ff_add_nr)
__device__ __forceinline__ ff2 ff_add_nr2(ff2 a, ff2 b)
{
    const ff2 s = two_sum2(a.h, b.h);
    return ff2{s.h, add2(s.l, add2(a.l, b.l))};
}
__device__ __forceinline__ ff2 ff_sub_nr2(ff2 a, ff2 b)
{
    const ff2 s = two_diff2(a.h, b.h);
    return ff2{s.h, add2(s.l, sub2(a.l, b.l))};
}
__device__ __forceinline__ ff2 ff_norm2(ff2 a)
{
    return fast_two_sum2(a.h, a.l);
}
// a b; _nr: the product's error stays in the low part
__device__ __forceinline__ ff2 ff_mul_nr2(ff2 a, ff2 b)
{
    const f2 p = mul2(a.h, b.h);
    return ff2{p, fma2(a.l, b.h, fma2(a.h, b.l, fma2(a.h, b.h, neg2(p))))};
}
__device__ __forceinline__ ff2 ff_mul2(ff2 a, ff2 b)
{
    return ff_norm2(ff_mul_nr2(a, b));
}
// a^2 of a pair whose low part may reach the size of the high one (an
// unnormalised sum that cancelled): the low part's own square is kept
__device__ __forceinline__ ff2 ff_sqr_nr2(ff2 a)
{
    const f2 p = mul2(a.h, a.h);
    return ff2{p, fma2(add2(a.h, a.h), a.l, fma2(a.l, a.l, fma2(a.h, a.h, neg2(p))))};
}

// 16 bytes {h of value 0, h of value 1, l of value 0, l of value 1}: both
// parts are register pairs as they come
__device__ __forceinline__ ff2 unpack4(float4 v)
{
    return ff2{mk2(v.x, v.y), mk2(v.z, v.w)};
}
__device__ __forceinline__ float4 pack4(ff2 a)
{
    return make_float4(lo2(a.h), hi2(a.h), lo2(a.l), hi2(a.l));
}

} // namespace ffa
} // namespace ss4d
