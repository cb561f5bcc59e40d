// Packed FP32 pairs (two lanes in one 64-bit register pair) and the
// double-float arithmetic of dfloat.cuh on them.
//
// sm_103a issues one FMA-pipe warp instruction per clock and scheduler; the
// packed forms do two lanes' work per issue slot at the same rate per lane
// (measured on a GB300: fma.rn.f32 118 lanes/clock/SM, fma.rn.f32x2 2 x 62),
// so a kernel bound by issue slots gains what its loads, shared-memory
// accumulators, compares and moves took from the FMA pipe.
//
// ptxas fuses a packed multiply that feeds a packed add or subtract into one
// fma even where both are written .rn (measured; -fmad=false does not stop
// it).  Products whose rounded value an error term depends on are therefore
// written as fma(a, b, nz) with nz = -0 from memory the compiler cannot see
// through (kNegZero2): the sum is the rounded product, and there is no
// multiply left to fuse.
#pragma once
#include <cuda_runtime.h>

#include "dfloat.cuh"
#include "rmw_common.cuh"

namespace rmw {

typedef float2 f2;

static __constant__ float2 kNegZero2 = {-0.0f, -0.0f};

__device__ __forceinline__ unsigned long long f2_bits(f2 a)
{
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a.x), "f"(a.y));
    return r;
}
__device__ __forceinline__ f2 f2_of(unsigned long long r)
{
    f2 a;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a.x), "=f"(a.y) : "l"(r));
    return a;
}

__device__ __forceinline__ f2 f2_dup(float a) { return make_float2(a, a); }
__device__ __forceinline__ f2 f2_neg(f2 a) { return make_float2(-a.x, -a.y); }
__device__ __forceinline__ f2 f2_add(f2 a, f2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ f2 f2_sub(f2 a, f2 b)
{
    unsigned long long r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(f2_bits(a)), "l"(f2_bits(b)));
    return f2_of(r);
}
__device__ __forceinline__ f2 f2_fma(f2 a, f2 b, f2 c) { return __ffma2_rn(a, b, c); }
// product consumed by fma operands only (may be fused into a following add)
__device__ __forceinline__ f2 f2_mul(f2 a, f2 b) { return __fmul2_rn(a, b); }
// product rounded on its own
__device__ __forceinline__ f2 f2_mulr(f2 a, f2 b) { return __ffma2_rn(a, b, kNegZero2); }

// ---- double-float on packed lanes (names and contracts as in dfloat.cuh) ----
struct df2 {
    f2 hi, lo;
};

__device__ __forceinline__ df2 df2_dup(df a) { return {f2_dup(a.hi), f2_dup(a.lo)}; }
__device__ __forceinline__ df2 df2_pack(df a, df b) { return {make_float2(a.hi, b.hi), make_float2(a.lo, b.lo)}; }
__device__ __forceinline__ df2 df2_zero() { return {f2_dup(0.f), f2_dup(0.f)}; }

// |a| >= |b| lane by lane (or a = 0)
__device__ __forceinline__ df2 fast_two_sum(f2 a, f2 b)
{
    const f2 s = f2_add(a, b);
    return {s, f2_sub(b, f2_sub(s, a))};
}
__device__ __forceinline__ df2 two_sum_df(f2 a, f2 b)
{
    const f2 s = f2_add(a, b);
    const f2 bb = f2_sub(s, a);
    return {s, f2_add(f2_sub(a, f2_sub(s, bb)), f2_sub(b, bb))};
}
__device__ __forceinline__ df2 operator-(df2 a) { return {f2_neg(a.hi), f2_neg(a.lo)}; }
__device__ __forceinline__ df2 scale2(df2 a, float p2)
{
    return {f2_mul(a.hi, f2_dup(p2)), f2_mul(a.lo, f2_dup(p2))};  // exact: fused or not is the same
}

__device__ __forceinline__ df2 mul_u(df2 a, df2 b)
{
    const f2 p = f2_mulr(a.hi, b.hi);
    f2 e = f2_fma(a.hi, b.hi, f2_neg(p));
    e = f2_fma(a.hi, b.lo, e);
    return {p, f2_fma(a.lo, b.hi, e)};
}
__device__ __forceinline__ df2 mul_u(df2 a, float b)
{
    const f2 bb = f2_dup(b), p = f2_mulr(a.hi, bb);
    const f2 e = f2_fma(a.hi, bb, f2_neg(p));
    return {p, f2_fma(a.lo, bb, e)};
}
__device__ __forceinline__ df2 sqr_u(df2 a)
{
    const f2 p = f2_mulr(a.hi, a.hi);
    const f2 e = f2_fma(a.hi, a.hi, f2_neg(p));
    return {p, f2_fma(f2_add(a.hi, a.hi), a.lo, e)};
}
__device__ __forceinline__ df2 norm(df2 a) { return fast_two_sum(a.hi, a.lo); }
__device__ __forceinline__ df2 operator*(df2 a, df2 b) { return norm(mul_u(a, b)); }
__device__ __forceinline__ df2 sqr(df2 a) { return norm(sqr_u(a)); }

__device__ __forceinline__ df2 add_u(df2 a, df2 b)
{
    const df2 s = two_sum_df(a.hi, b.hi);
    return {s.hi, f2_add(s.lo, f2_add(a.lo, b.lo))};
}
__device__ __forceinline__ df2 sub_u(df2 a, df2 b)
{
    const f2 s = f2_sub(a.hi, b.hi);
    const f2 bb = f2_sub(s, a.hi);  // -(b as it entered the sum)
    const f2 t = f2_sub(f2_sub(a.hi, f2_sub(s, bb)), f2_add(b.hi, bb));
    return {s, f2_add(t, f2_sub(a.lo, b.lo))};
}
__device__ __forceinline__ df2 operator+(df2 a, df2 b) { return norm(add_u(a, b)); }
__device__ __forceinline__ df2 operator-(df2 a, df2 b) { return norm(sub_u(a, b)); }

// a + b, unnormalised, where |a.hi| >= |b.hi| (lane by lane)
__device__ __forceinline__ df2 add_fast_u(df2 a, df2 b)
{
    const df2 s = fast_two_sum(a.hi, b.hi);
    return {s.hi, f2_add(s.lo, f2_add(a.lo, b.lo))};
}
// c + b, unnormalised, for a float c >= |b|
__device__ __forceinline__ df2 add_fast_u(float c, df2 b)
{
    const df2 s = fast_two_sum(f2_dup(c), b.hi);
    return {s.hi, f2_add(s.lo, b.lo)};
}
// a + c, unnormalised, for a float c <= |a|
__device__ __forceinline__ df2 add_fast_u(df2 a, float c)
{
    const df2 s = fast_two_sum(a.hi, f2_dup(c));
    return {s.hi, f2_add(s.lo, a.lo)};
}

// a b + c d, unnormalised
__device__ __forceinline__ df2 mad2_u(df2 a, df2 b, df2 c, df2 d) { return add_u(mul_u(a, b), mul_u(c, d)); }

// acc += a b + c d without renormalising acc (acc_dot2 of dfloat.cuh)
__device__ __forceinline__ void acc_dot2(df2 &acc, df2 a, df2 b, df2 c, df2 d)
{
    const df2 p = mul_u(a, b), q = mul_u(c, d);
    const df2 t1 = two_sum_df(acc.hi, p.hi);
    const df2 t2 = two_sum_df(t1.hi, q.hi);
    acc.hi = t2.hi;
    acc.lo = f2_add(acc.lo, f2_add(f2_add(t1.lo, t2.lo), f2_add(p.lo, q.lo)));
}

// acc += a b (+ c d + e f) without renormalising acc
__device__ __forceinline__ void acc_dot1(df2 &acc, df2 a, df2 b)
{
    const df2 p = mul_u(a, b);
    const df2 t = two_sum_df(acc.hi, p.hi);
    acc.hi = t.hi;
    acc.lo = f2_add(acc.lo, f2_add(t.lo, p.lo));
}
__device__ __forceinline__ void acc_dot3(df2 &acc, df2 a, df2 b, df2 c, df2 d, df2 e, df2 f)
{
    const df2 p = mul_u(a, b), q = mul_u(c, d), r = mul_u(e, f);
    const df2 t1 = two_sum_df(acc.hi, p.hi);
    const df2 t2 = two_sum_df(t1.hi, q.hi);
    const df2 t3 = two_sum_df(t2.hi, r.hi);
    acc.hi = t3.hi;
    const f2 lo = f2_add(f2_add(t1.lo, t2.lo), t3.lo);
    acc.lo = f2_add(acc.lo, f2_add(lo, f2_add(f2_add(p.lo, q.lo), r.lo)));
}

// 1/sqrt(x) from the estimate y, as rsqrt_df
__device__ __forceinline__ df2 rsqrt_df(df2 x, f2 y)
{
    const f2 h = f2_mul(f2_dup(-0.5f), x.hi);
    y = f2_mulr(y, f2_fma(h, f2_mul(y, y), f2_dup(1.5f)));
    const f2 p = f2_mulr(y, y);
    const df2 t = mul_u(x, df2{p, f2_fma(y, y, f2_neg(p))});
    const f2 e = f2_sub(f2_sub(f2_dup(1.0f), t.hi), t.lo);
    return fast_two_sum(y, f2_mul(f2_mul(y, e), f2_fma(f2_dup(0.375f), e, f2_dup(0.5f))));
}
__device__ __forceinline__ df2 rsqrt_df(df2 x) { return rsqrt_df(x, make_float2(rsqrtf(x.hi.x), rsqrtf(x.hi.y))); }
// for x far above the smallest normal float (squared distances to images: at least 4)
__device__ __forceinline__ df2 rsqrt_far_df(df2 x)
{
    return rsqrt_df(x, make_float2(rsqrt_approx(x.hi.x), rsqrt_approx(x.hi.y)));
}

}  // namespace rmw
