// FP64 products and reciprocal square roots on the integer pipes.
//
// An FP64 warp instruction holds its SM partition's pipe for 64 clocks
// (measured: 0.53 T FP64 instructions/s on 152 SMs), during which the same
// partition issues about 60 integer instructions.  The FP64 pair kernels are
// bound by that pipe alone, so the operations whose operands are known to be
// finite and normal leave it: 53 x 53-bit schoolbook products from 32-bit
// halves (22 to 28 integer instructions) and 1/sqrt as one third-order Newton
// step in fixed point (about 45).  M_UF at 10,752 blobs 8.1 -> 5.5 ms with
// products and roots, 4.36 ms with multiply-adds of positive terms and the
// products with the vectors, 3.69 ms with seven of mixed signs
// (3.73 with the scaling of the separations).
//
// Error bounds, tested against exact arithmetic: int_mul 0.504 ulp (the
// product of the low halves, below 2^-62 of the result, and the order of ties
// are left out; the FP64 pipe's 0.5), int_fma_pos 0.51 ulp, int_fma half an
// ulp and 2^-59 of the larger term (the pipe's: half an ulp, also where the
// terms cancel; their own roundings are 2^-53 of them), int_rsqrt 0.51 ulp
// (rsqrt64 1 ulp).  The products' errors against 64 bits are no larger than
// with the pipe's operations alone.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "rmw_common.cuh"

namespace rmw {

__device__ __forceinline__ uint64_t u64_of(uint32_t hi, uint32_t lo) { return ((uint64_t)hi << 32) | lo; }

// 53-bit significand of a normal x, leading bit at bit 63
__device__ __forceinline__ void int_significand(double x, uint32_t &h, uint32_t &l)
{
    const uint32_t hi = (uint32_t)__double2hiint(x), lo = (uint32_t)__double2loint(x);
    h = __funnelshift_l(lo, hi, 11) | 0x80000000u;
    l = lo << 11;
}
// top 64 bits of a 64 x 64-bit product, at most 3 units below the exact value
__device__ __forceinline__ uint64_t int_mulhi(uint32_t ah, uint32_t al, uint32_t bh, uint32_t bl)
{
    return (uint64_t)ah * bh + __umulhi(ah, bl) + __umulhi(al, bh);
}
// |a b| with the sign bits of the high word passed in; exponents must not leave the normal range
__device__ __forceinline__ double int_mul_core(double a, double b, uint32_t ea, uint32_t eb, uint32_t sign)
{
    uint32_t ah, al, bh, bl;
    int_significand(a, ah, al);
    int_significand(b, bh, bl);
    const uint64_t r = int_mulhi(ah, al, bh, bl);  // in [2^62, 2^64 - 2^12]
    const uint32_t top = (uint32_t)(r >> 63);
    const uint64_t q = (r + (512u << top)) >> (10 + top);  // in [2^52, 2^53], rounded to nearest
    const uint32_t hi = (uint32_t)(q >> 32) + ea + eb + (top << 20) - (1024u << 20) + sign;  // q's leading bit adds one
    return __hiloint2double((int)hi, (int)(uint32_t)q);
}
// a b of positive normal numbers whose product is normal
__device__ __forceinline__ double int_mul(double a, double b)
{
    return int_mul_core(a, b, (uint32_t)__double2hiint(a) & 0x7ff00000u, (uint32_t)__double2hiint(b) & 0x7ff00000u, 0u);
}
// a b of finite numbers below 2^400 in magnitude; factors below 2^-400 count as zero
__device__ __forceinline__ double int_mul_signed(double a, double b)
{
    const uint32_t ha = (uint32_t)__double2hiint(a), hb = (uint32_t)__double2hiint(b);
    const uint32_t ea = ha & 0x7ff00000u, eb = hb & 0x7ff00000u;
    const double p = int_mul_core(a, b, ea, eb, (ha ^ hb) & 0x80000000u);
    return min(ea, eb) < (623u << 20) ? 0.0 : p;
}

// 1/sqrt(x) in FP64 from an estimate y of relative error below 2^-20: one
// third-order Householder step, y + y e (1/2 + 3 e / 8) with e = 1 - x y^2.
// What the step leaves out is 5/16 e^3 < 2^-57.  The rounding of y^2 moves e by 2^-53 and
// the result by half an ulp at most, the last fma rounds by another half:
// 1 ulp, as the library's rsqrt.
__device__ __forceinline__ double rsqrt64_step(double x, double y)
{
    const double e = fma(-x, y * y, 1.0);
    return fma(y * e, fma(0.375, e, 0.5), y);
}

// 1/sqrt(x) of a positive normal x.  m = x 4^-h in [1, 4); y0 = 1/sqrt(m) to
// 2^-22 in units 2^-31, e = 1 - m y0^2 and y0 (1 + e/2 + 3 e^2/8), rounded once.
__device__ __forceinline__ double int_rsqrt(double x)
{
    const uint32_t hi = (uint32_t)__double2hiint(x), lo = (uint32_t)__double2loint(x);
    const int ex = (int)(hi >> 20);
    const int odd = (ex & 1) ^ 1;  // the exponent ex - 1023 is odd
    const uint32_t xh = __funnelshift_l(lo, (hi & 0xfffffu) | 0x100000u, 10 + odd), xl = lo << (10 + odd);  // 2^-62
    const float y = rsqrt_approx((float)xh);  // 2^-15 / sqrt(m)
    const uint32_t y0 = min(__float2uint_rn(y * 70368744177664.0f), 0x7fffffffu);  // 2^46 y
    const uint64_t q = (uint64_t)y0 * y0;                                           // 2^-62
    const int64_t e = (int64_t)((1ull << 60) - int_mulhi(xh, xl, (uint32_t)(q >> 32), (uint32_t)q));  // 2^-60
    const int e51 = (int)(e >> 9);                                                  // |e| < 2^-21
    const int64_t f = e + ((__mulhi(e51, e51) * 3) >> 12);                          // e + 3/4 e^2, 2^-60
    // y0 f / 2: the product's units 2^-91, its high part's 2^-59, halved 2^-60
    const int64_t d = (int64_t)(int)y0 * (int)(f >> 32) + (int64_t)__umulhi(y0, (uint32_t)f);
    const uint64_t s = ((uint64_t)y0 << 29) + (uint64_t)d;                          // y, 2^-60, in (2^59, 2^60]
    const uint64_t m = (s + 64) >> 7;                                               // in [2^52, 2^53]
    const int h = (ex - 1023 - odd) >> 1;
    return __hiloint2double((int)((uint32_t)(m >> 32) + ((uint32_t)(1021 - h) << 20)), (int)(uint32_t)m);
}

// a b + c of non-negative numbers below 2^400 in magnitude (signs ignored; zero allowed): factors or addends 2^62 below
// the other term count as zero.  0.51 ulp; 0 0 + 0 is 0 (squares of stacked blobs' separations), and the sum of two
// zero terms otherwise below 2^-600.
__device__ __forceinline__ double int_fma_pos(double a, double b, double c)
{
    uint32_t ah, al, bh, bl, ch, cl;
    int_significand(a, ah, al);
    int_significand(b, bh, bl);
    int_significand(c, ch, cl);
    const int ec = (__double2hiint(c) & 0x7fffffff) >> 20;
    const int ep = ((__double2hiint(a) & 0x7fffffff) >> 20) + ((__double2hiint(b) & 0x7fffffff) >> 20) - 1023;
    const uint64_t p = int_mulhi(ah, al, bh, bl) >> 1, s = u64_of(ch, cl) >> 2;  // units 2^-61 of their exponents
    const int d = ep - ec;
    const uint64_t big = d >= 0 ? p : s, small = d >= 0 ? s : p;
    const uint64_t t = big + (small >> min(abs(d), 63));  // in [2^61, 2^64)
    const int z = __clz((int)(t >> 32));                  // 0 to 2
    const uint64_t q = t << z, m = (q >> 11) + ((q >> 10) & 1);
    const uint32_t hi = (uint32_t)(m >> 32) + ((uint32_t)(max(ep, ec) + 1 - z) << 20);
    return __hiloint2double((int)hi, (int)(uint32_t)m);
}

// a b + c of finite numbers below 2^400 in magnitude; terms below 2^-400 count
// as zero.  Half an ulp and 2^-59 of the larger term, which counts where the
// terms cancel.
__device__ __forceinline__ double int_fma(double a, double b, double c)
{
    const uint32_t ha = (uint32_t)__double2hiint(a), hb = (uint32_t)__double2hiint(b), hc = (uint32_t)__double2hiint(c);
    uint32_t ah, al, bh, bl, ch, cl;
    int_significand(a, ah, al);
    int_significand(b, bh, bl);
    int_significand(c, ch, cl);
    const int ec = (int)(hc >> 20 & 0x7ffu), ep = (int)(ha >> 20 & 0x7ffu) + (int)(hb >> 20 & 0x7ffu) - 1023;
    const int d = ep - ec;
    const bool sw = d < 0;
    const uint64_t p = int_mulhi(ah, al, bh, bl) >> 2, s = u64_of(ch, cl) >> 3;  // units 2^-60 of their exponents
    const int64_t big = (int64_t)(sw ? s : p), small = (int64_t)((sw ? p : s) >> min(abs(d), 63));
    const uint32_t sp = ha ^ hb;
    const int64_t t = (int32_t)(sp ^ hc) < 0 ? big - small : big + small;
    const uint64_t m0 = (uint64_t)(t < 0 ? -t : t);
    const int z = __clzll((long long)m0);
    const uint64_t q = m0 << (z & 63), m = (q >> 11) + ((q >> 10) & 1);
    const uint32_t sign = ((sw ? hc : sp) ^ (uint32_t)(t >> 32)) & 0x80000000u;
    const int e = max(ep, ec) + 2 - z;
    const uint32_t hi = (uint32_t)(m >> 32) + ((uint32_t)e << 20) + sign;
    return t == 0 || e < 560 ? 0.0 : __hiloint2double((int)hi, (int)(uint32_t)m);
}

// x in [2^-64, 2^64): what the pair kernels' integer forms ask of the squared distances
__device__ __forceinline__ bool int_range(double x)
{
    return (uint32_t)__double2hiint(x) - (959u << 20) < (128u << 20);
}

// |d| < 2^400, for separations before they are scaled (false for NaN and infinities)
__device__ __forceinline__ bool int_range_mag(double x, double y, double z)
{
    const uint32_t a = (uint32_t)__double2hiint(x) & 0x7fffffffu, b = (uint32_t)__double2hiint(y) & 0x7fffffffu;
    return max(max(a, b), (uint32_t)__double2hiint(z) & 0x7fffffffu) < (1423u << 20);
}
// |d| < 2^32, for separations (false for NaN and infinities)
__device__ __forceinline__ bool int_range_sep(double dx, double dy, double dz)
{
    const uint32_t a = (uint32_t)__double2hiint(dx) & 0x7fffffffu, b = (uint32_t)__double2hiint(dy) & 0x7fffffffu;
    return max(max(a, b), (uint32_t)__double2hiint(dz) & 0x7fffffffu) < (1055u << 20);
}
// zero or 2^-E <= |v| < 2^300.  Factors below 2^-400 count as zero, so what the pair kernels multiply has to stay above:
// coordinates (E = 130) differ by nothing or by 2^-182, separations in radii are 2^-246 at least, their products
// with vectors (E = 150) 2^-396.
template <int E = 300> __device__ __forceinline__ bool int_range_vec(double v)
{
    return ((uint32_t)__double2hiint(v) & 0x7fffffffu) - ((uint32_t)(1023 - E) << 20) < ((uint32_t)(300 + E) << 20) ||
           v == 0.0;
}
template <int E = 300> __device__ __forceinline__ bool int_range_vec(double x, double y, double z)
{
    return int_range_vec<E>(x) && int_range_vec<E>(y) && int_range_vec<E>(z);
}
__device__ __forceinline__ bool int_range_blob(double x, double y, double z, double vx, double vy, double vz)
{
    return int_range_vec<130>(x, y, z) && int_range_vec<150>(vx, vy, vz);
}

// Products of the pair blocks in plain arithmetic (MulPipe) or on the integer
// pipes (MulInt).  pos: both factors positive; mul: any sign; fma_pos: a b + c
// of non-negative terms; fma_any: of any sign.
template <typename T> struct MulPipe {
    static __device__ __forceinline__ T pos(T a, T b) { return a * b; }
    static __device__ __forceinline__ T mul(T a, T b) { return a * b; }
    static __device__ __forceinline__ T fma_pos(T a, T b, T c) { return fma(a, b, c); }
    static __device__ __forceinline__ T fma_any(T a, T b, T c) { return fma(a, b, c); }
    static __device__ __forceinline__ bool le4(T x) { return !(x > T(4)); }
    static __device__ __forceinline__ bool lt4(T x) { return !(x >= T(4)); }
};
using MulFp64 = MulPipe<double>;
struct MulInt {
    static __device__ __forceinline__ double pos(double a, double b) { return int_mul(a, b); }
    static __device__ __forceinline__ double mul(double a, double b) { return int_mul_signed(a, b); }
    static __device__ __forceinline__ double fma_pos(double a, double b, double c) { return int_fma_pos(a, b, c); }
    static __device__ __forceinline__ double fma_any(double a, double b, double c) { return int_fma(a, b, c); }
    static __device__ __forceinline__ bool le4(double x) { return __double_as_longlong(x) <= 0x4010000000000000ll; }
    static __device__ __forceinline__ bool lt4(double x) { return __double_as_longlong(x) < 0x4010000000000000ll; }
};

}  // namespace rmw
