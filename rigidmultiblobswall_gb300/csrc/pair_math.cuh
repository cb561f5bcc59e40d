// Pair formulas of the single-wall RPY mobility blocks (shared by the
// all-pairs product kernels and the dense per-body mobility of the
// preconditioner).
#pragma once
#include <type_traits>

#include "f32x2.cuh"
#include "fp64_int.cuh"
#include "rmw_common.cuh"

namespace rmw {

// 1/sqrt(x) in FP64: the hardware's estimate (relative error below 2^-20) and
// rsqrt64_step, five FP64 instructions and no special-case branch (zero,
// infinite and subnormal x give non-finite values; no pair of distinct blobs
// has one).
__device__ __forceinline__ double rsqrt64(double x)
{
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    return rsqrt64_step(x, y);
}

// pair math.  (dx,dy,dz) = (r_i - r_j)/a; Rz = (z_i + z_j)/a; hi = z_i/a; hj = z_j/a.
template <typename T> __device__ __forceinline__ T rsq(T x);
template <> __device__ __forceinline__ double rsq<double>(double x) { return rsqrt64(x); }
template <> __device__ __forceinline__ float rsq<float>(float x) { return rsqrt_approx(x); }

// The reference builds each 3x3 block from unit vectors e = (dx, dy, Rz)/R and
// then multiplies by v.  Here the products are regrouped so that e never
// appears: with s = 1/R, W = dx vx + dy vy + Rz vz and Q = dy vx - dx vy,
//   (f2 (e.v) + f3 vz) e  = (f2 W s^2 + f3 vz s) (dx, dy, Rz)
// and the RPY term Bc (d.v) d shares dx vx + dy vy with W.  h_hat never
// appears either (h_hat e_z = h_j s, (1 - h_hat) e_z = h_i s).
template <int KIND, typename T>
__device__ __forceinline__ void pair_contrib(T dx, T dy, T dz, T Rz, T hi, T hj, T vx, T vy, T vz, T &ux, T &uy,
                                             T &uz)
{
    const T rho2 = dx * dx + dy * dy;
    const T r2 = rho2 + dz * dz;
    const T invr = rsq<T>(r2);
    const T r = r2 * invr;
    const T Rz2 = Rz * Rz;
    const T s = rsq<T>(rho2 + Rz2);
    const T s2 = s * s;
    const T s3 = s2 * s;
    const T E = Rz2 * s2;  // e_z^2
    const T Pxy = dx * vx + dy * vy;
    if (KIND == RMW_UF) {
        const T invr2 = invr * invr;
        // far branch always; the near (r <= 2) branch only when some lane of the
        // warp needs it (rare: touching blobs), so warps stay convergent
        T A = (T(1) + T(2.0 / 3.0) * invr2) * invr;
        T Bc = (T(1) - T(2) * invr2) * invr2 * invr;
        const bool near = !(r > T(2));
        if (__any_sync(__activemask(), near)) {
            if (near) {
                A = T(4.0 / 3.0) * (T(1) - T(0.28125) * r);
                Bc = T(0.125) * invr;
            }
        }
        const T dv = Pxy + dz * vz;
        const T W = Pxy + Rz * vz;
        const T s5 = s3 * s2;
        const T hh = hi * hj * s2;
        const T ez = Rz * s;
        const T q5 = (T(1) - T(5) * E) * s3;
        const T f1 = -((T(1) + T(2) * hh) * s + T(2.0 / 3.0) * ((T(1) - T(3) * E) * s3 - q5 * s2));
        const T f2 = -((T(1) - T(6) * hh) * s - T(2) * q5 + T(10.0 / 3.0) * (T(1) - T(7) * E) * s5);
        const T f3 = T(2.0 / 3.0) * (T(3) * hj * s2 - T(18) * hh * ez * s +
                                     ez * (T(10) * (T(2) - T(7) * E) * s5 - T(6) * q5));
        const T f4 = T(2.0 / 3.0) * (T(3) * hj * s2 - T(10) * ez * s5);
        const T f5 = T(-4.0 / 3.0) * (T(3) * (hj * hj + E) * s3 + (T(2) - T(15) * E) * s5);
        const T Af = A + f1;
        const T Gr = Bc * dv;
        const T Gw = (f2 * W * s + f3 * vz) * s;
        const T G = Gr + Gw;
        ux += Af * vx + G * dx;
        uy += Af * vy + G * dy;
        uz += Af * vz + Gr * dz + Gw * Rz + f4 * W * s + f5 * vz;
    } else if (KIND == RMW_UT || KIND == RMW_WF) {
        T c = invr * invr * invr;
        const bool near = !(r >= T(2));
        if (__any_sync(__activemask(), near)) {
            if (near) c = T(0.5) * (T(1) - T(0.375) * r);
        }
        const T Q = dy * vx - dx * vy;  // (v x d)_z
        // RPY part: c (v x d)
        T ax = c * (vy * dz - vz * dy);
        T ay = c * (vz * dx - vx * dz);
        T az = c * Q;
        const T s4 = s2 * s2;
        const T ez = Rz * s;
        const T h = (KIND == RMW_UT) ? hi : hj;  // UT evaluates the wall term with i and j swapped
        const T hs3 = h * s3;
        const T ezs4 = ez * s4;
        const T f2 = T(2) * (T(6) * hs3 * ez + (T(1) - T(10) * E) * s4);
        const T f3 = T(-2) * (T(3) * hs3 - T(5) * ezs4);
        const T f4 = T(-2) * (hs3 - ezs4);
        const T p = s2 * ez + f4;  // f1 = s^2
        if (KIND == RMW_UT) {
            const T F3 = f3 * s2 * Q;
            const T F1 = s3 * vz;
            const T g = s2 + f2 + f3 * ez;
            ax += F3 * dx + p * vy + F1 * dy;
            ay += F3 * dy - p * vx - F1 * dx;
            az -= g * s * Q;
        } else {
            const T g = s2 + f2 + f3 * ez;
            const T H = f3 * s2 * Pxy + g * s * vz;
            ax += H * dy - p * vy;
            ay += p * vx - H * dx;
            az -= s3 * Q;
        }
        ux += ax;
        uy += ay;
        uz += az;
    } else {  // RMW_WT
        const T invr2 = invr * invr;
        const T invr3 = invr2 * invr;
        T A = T(-0.5) * invr3;
        T Bc = T(1.5) * invr2 * invr3;
        const bool near = !(r >= T(2));
        if (__any_sync(__activemask(), near)) {
            if (near) {
                A = T(1) - T(0.84375) * r + T(0.078125) * r * r2;
                Bc = T(0.28125) * invr - T(0.046875) * r;
            }
        }
        const T dv = Pxy + dz * vz;
        const T W = Pxy + Rz * vz;
        const T Q = dy * vx - dx * vy;
        const T s5 = s3 * s2;
        const T Af = A + T(0.5) * (T(1) - T(6) * E) * s3;
        const T Gw = T(-1.5) * s5 * W;
        const T Tq = T(3) * s5 * Q;
        const T Gr = Bc * dv;
        ux += Af * vx + (Gr + Gw) * dx + Tq * dy;
        uy += Af * vy + (Gr + Gw) * dy - Tq * dx;
        uz += Af * vz + Gr * dz - Gw * Rz;
    }
}

// Vector-independent part of one M_UF block, times 3/2 (the consumers'
// finalize kernels multiply the pair sums by 2/3 in FP64), for the FP32 pair
// kernels:  (3/2) M v = Af v + (Bc (d.v) + c2 W + c3 vz) (dx, dy, .) ...
// with W = dx vx + dy vy + Rz vz (see uf_apply).  The 3/2 turns the RPY and
// Swan-Brady constants into the small integers and halves below:
//   (3/2) A  = 3/(2r) + 1/r^3,          (3/2) Bc = (3/2 - 3/r^2) / r^3
//   (3/2) f1 = -(3/2 + 3 hh) s - [(1 - 3E) t - (1 - 5E) p]
//   (3/2) f2 = -(3/2 - 9 hh) s + 3 (1 - 5E) t - 5 (1 - 7E) p
//   c3 = (3/2) f3 s = 3 h_j t - 18 hh Rz t + Rz s^2 [10 (2 - 7E) p - 6 (1 - 5E) t]
//   c4 = (3/2) f4 s = 3 h_j t - 10 Rz s^2 p
//   (3/2) f5 = -2 [3 (h_j^2 + E) t + (2 - 15E) p]
// with t = s^3, p = s^5, E = (Rz s)^2, hh = h_i h_j s^2; for r <= 2
// (3/2) A = 2 (1 - 9r/32), (3/2) Bc = 3 / (16 r).
constexpr double kUFCoeffScale = 2.0 / 3.0;  // undoes the 3/2
struct UFCoeffs {
    float Af, Bc, c2, c3, c4, Af5;  // Af5 = Af + f5, the zz diagonal
};

__device__ __forceinline__ UFCoeffs uf_coeffs(float dx, float dy, float dz, float Rz, float hi, float hj)
{
    const float rho2 = dx * dx + dy * dy;
    const float r2 = rho2 + dz * dz;
    const float invr = rsqrt_approx(r2);
    const float Rz2 = Rz * Rz;
    const float s = rsqrt_approx(rho2 + Rz2);
    const float u = s * s;
    const float t = u * s;
    const float p = t * u;
    const float E = Rz2 * u;
    const float invr2 = invr * invr;
    const float invr3 = invr2 * invr;
    float A = 1.5f * invr + invr3;
    float Bc = (1.5f - 3.0f * invr2) * invr3;
    const bool near = !(r2 > 4.0f);  // r <= 2
    if (__any_sync(__activemask(), near)) {
        if (near) {
            const float r = r2 * invr;
            A = 2.0f - 0.5625f * r;
            Bc = 0.1875f * invr;
        }
    }
    const float hh = hi * hj * u;
    const float q5 = (1.0f - 5.0f * E) * t;
    const float Ru = Rz * u;
    const float hjt3 = 3.0f * hj * t;
    const float f1 = -((1.5f + 3.0f * hh) * s + ((1.0f - 3.0f * E) * t - q5 * u));
    const float f2 = 3.0f * q5 - (1.5f - 9.0f * hh) * s - 5.0f * (1.0f - 7.0f * E) * p;
    const float c3 = hjt3 - 18.0f * hh * Rz * t + Ru * (10.0f * (2.0f - 7.0f * E) * p - 6.0f * q5);
    const float c4 = hjt3 - 10.0f * Ru * p;
    const float f5 = -2.0f * (3.0f * (hj * hj + E) * t + (2.0f - 15.0f * E) * p);
    const float Af = A + f1;
    return {Af, Bc, f2 * u, c3, c4, Af + f5};
}

// (M v) of uf_coeffs: every term chained into the accumulator by an FMA (two plain
// multiplies and one subtraction per application)
__device__ __forceinline__ void uf_apply(const UFCoeffs &c, float dx, float dy, float dz, float Rz, float vx, float vy,
                                         float vz, float &ux, float &uy, float &uz)
{
    // with dv = d.v, G = Bc dv + Gw and Rz - dz = 2 h_j:
    // (M v)_z = Af5 vz + G dz + Gw (Rz - dz) + c4 W
    const float h2 = Rz - dz;
    const float dv = fmaf(dz, vz, fmaf(dy, vy, dx * vx));
    const float W = fmaf(h2, vz, dv);
    const float Gw = fmaf(c.c2, W, c.c3 * vz);
    const float G = fmaf(c.Bc, dv, Gw);
    ux = fmaf(c.Af, vx, fmaf(G, dx, ux));
    uy = fmaf(c.Af, vy, fmaf(G, dy, uy));
    uz = fmaf(c.Af5, vz, fmaf(G, dz, fmaf(Gw, h2, fmaf(c.c4, W, uz))));
}

// uf_coeffs for two pairs in packed lanes: every operation written out
// with the contractions the compiler gives the scalar form (products that
// feed a sum fused into it, the operands of other products rounded), so a
// mixed product is the same to the bit whichever form forms its blocks.
// FUSED_R2: R^2 = fma(Rz, Rz, rho^2) instead of rho^2 + Rz^2 rounded, which
// the scalar form came out as in every second step of an unrolled loop.
struct UFCoeffs2 {
    f2 Af, Bc, c2, c3, c4, Af5;
};
__device__ __forceinline__ f2 f2_c(float a, f2 b, f2 c) { return f2_fma(f2_dup(a), b, c); }  // a b + c
__device__ __forceinline__ f2 f2_c(float a, f2 b, float c) { return f2_fma(f2_dup(a), b, f2_dup(c)); }
__device__ __forceinline__ f2 f2_s(float a, f2 b) { return f2_mul(f2_dup(a), b); }

template <bool FUSED_R2>
__device__ __forceinline__ UFCoeffs2 uf_coeffs_f2(f2 dx, f2 dy, f2 dz, f2 Rz, f2 hi, f2 hj)
{
    const f2 rho2 = f2_fma(dx, dx, f2_mul(dy, dy));
    const f2 r2 = f2_fma(dz, dz, rho2);
    const f2 invr = make_float2(rsqrt_approx(r2.x), rsqrt_approx(r2.y));
    const f2 Rz2 = f2_mulr(Rz, Rz);
    const f2 R2 = FUSED_R2 ? f2_fma(Rz, Rz, rho2) : f2_add(rho2, Rz2);
    const f2 s = make_float2(rsqrt_approx(R2.x), rsqrt_approx(R2.y));
    const f2 u = f2_mul(s, s), t = f2_mul(u, s), p = f2_mul(t, u), E = f2_mul(Rz2, u);
    const f2 invr2 = f2_mul(invr, invr), invr3 = f2_mul(invr2, invr);
    f2 A = f2_c(1.5f, invr, invr3);
    f2 Bc = f2_mul(f2_c(-3.0f, invr2, 1.5f), invr3);
    const bool na = !(r2.x > 4.0f), nb = !(r2.y > 4.0f);  // r <= 2
    if (__any_sync(__activemask(), na || nb)) {
        if (na) {
            A.x = fmaf(-0.5625f, __fmul_rn(r2.x, invr.x), 2.0f);
            Bc.x = __fmul_rn(0.1875f, invr.x);
        }
        if (nb) {
            A.y = fmaf(-0.5625f, __fmul_rn(r2.y, invr.y), 2.0f);
            Bc.y = __fmul_rn(0.1875f, invr.y);
        }
    }
    const f2 hh = f2_mul(f2_mul(hi, hj), u);
    const f2 q5 = f2_mul(f2_c(-5.0f, E, 1.0f), t);
    const f2 Ru = f2_mul(Rz, u);
    const f2 hjt3 = f2_mul(f2_s(3.0f, hj), t);
    const f2 e7 = f2_c(-7.0f, E, 1.0f);
    // -f1
    const f2 g1 = f2_fma(f2_c(3.0f, hh, 1.5f), s, f2_fma(f2_c(-3.0f, E, 1.0f), t, f2_neg(f2_mul(q5, u))));
    const f2 x2 = f2_c(3.0f, q5, f2_neg(f2_mul(f2_c(-9.0f, hh, 1.5f), s)));
    const f2 f2c = f2_fma(f2_neg(f2_s(5.0f, e7)), p, x2);
    const f2 in = f2_fma(f2_s(10.0f, f2_c(-7.0f, E, 2.0f)), p, f2_neg(f2_s(6.0f, q5)));
    const f2 f5 = f2_fma(f2_s(3.0f, f2_fma(hj, hj, E)), t, f2_mul(f2_c(-15.0f, E, 2.0f), p));
    UFCoeffs2 c;
    c.Af = f2_sub(A, g1);
    c.Bc = Bc;
    c.c2 = f2_mulr(f2c, u);
    c.c3 = f2_fma(Ru, in, f2_fma(f2_neg(f2_mul(f2_s(18.0f, hh), Rz)), t, hjt3));
    c.c4 = f2_fma(f2_neg(f2_s(10.0f, Ru)), p, hjt3);
    c.Af5 = f2_c(-2.0f, f5, c.Af);
    return c;
}

// uf_apply in packed lanes
__device__ __forceinline__ void uf_apply_f2(const UFCoeffs2 &c, f2 c3, f2 c4, f2 dx, f2 dy, f2 dz, f2 h2, f2 vx, f2 vy,
                                            f2 vz, f2 &ux, f2 &uy, f2 &uz)
{
    const f2 dv = f2_fma(dz, vz, f2_fma(dy, vy, f2_mul(dx, vx)));
    const f2 W = f2_fma(h2, vz, dv);
    const f2 Gw = f2_fma(c.c2, W, f2_mul(c3, vz));
    const f2 G = f2_fma(c.Bc, dv, Gw);
    ux = f2_fma(c.Af, vx, f2_fma(G, dx, ux));
    uy = f2_fma(c.Af, vy, f2_fma(G, dy, uy));
    uz = f2_fma(c.Af5, vz, f2_fma(G, dz, f2_fma(Gw, h2, f2_fma(c4, W, uz))));
}

// The explicit 3x3 block of uf_coeffs, for products with several right-hand
// sides: nine FMAs per right-hand side instead of sixteen.  With d = (dx, dy,
// dz), e = (dx, dy, Rz) and z the wall normal,
//   M = Af I + Bc d d^T + c2 e e^T + c3 e z^T + c4 z e^T + f5 z z^T,
// so M_xy = M_yx = (Bc + c2) dx dy, M_xz = dx t3, M_zx = dx t4 with
// t3,4 = Bc dz + c2 Rz + c3,4, and M_zz = Af + f5 + Bc dz^2 + (c2 Rz + c3 + c4) Rz.
// Two pairs (sources) in packed lanes.
struct UFBlock2 {
    f2 xx, xy, xz, yy, yz, zx, zy, zz;  // M_yx = M_xy
};

__device__ __forceinline__ UFBlock2 uf_block_f2(const UFCoeffs2 &c, f2 dx, f2 dy, f2 dz, f2 Rz)
{
    const f2 b2 = f2_add(c.Bc, c.c2);
    const f2 t = f2_fma(c.Bc, dz, f2_mul(c.c2, Rz));
    const f2 t3 = f2_add(t, c.c3), t4 = f2_add(t, c.c4);
    const f2 px = f2_mul(b2, dx);
    UFBlock2 m;
    m.xx = f2_fma(px, dx, c.Af);
    m.xy = f2_mul(px, dy);
    m.yy = f2_fma(f2_mul(b2, dy), dy, c.Af);
    m.xz = f2_mul(dx, t3);
    m.yz = f2_mul(dy, t3);
    m.zx = f2_mul(dx, t4);
    m.zy = f2_mul(dy, t4);
    m.zz = f2_fma(f2_fma(c.c2, Rz, f2_add(c.c3, c.c4)), Rz, f2_fma(f2_mul(c.Bc, dz), dz, c.Af5));
    return m;
}

// The explicit M_UF block in FP64, times 3/2: the formulas of uf_block_df
// (pair_math_df.cuh), where they are derived.  73 operations a pair, both
// ways, against 93 of uf_coeffs / uf_apply: the FP64 pipe (1/64 of the FP32
// rate) bounds the kernels that use it, so MulInt takes 42 of them to the
// integer pipes (fp64_int.cuh): the products and positive sums of the
// geometry, seven multiply-adds of mixed signs and the products with the
// vectors.  10,752 blobs 8.1 -> 3.73 ms.
// ZPER: dz is an image's and not h_i - h_j.
struct PairGeoD {
    double r2, invr, i2, u, s, t, p;
};
// MUL = MulInt needs r2 and R2 (the squared distances of a pair, the second to
// the mirror image) within int_range.
template <class MUL>
__device__ __forceinline__ PairGeoD pair_geo_d(double r2, double R2)
{
    constexpr bool I = std::is_same<MUL, MulInt>::value;
    PairGeoD g;
    g.r2 = r2;
    g.invr = I ? int_rsqrt(r2) : rsqrt64(r2);
    g.s = I ? int_rsqrt(R2) : rsqrt64(R2);
    g.i2 = MUL::pos(g.invr, g.invr);
    g.u = MUL::pos(g.s, g.s);
    g.t = MUL::pos(g.u, g.s);
    g.p = MUL::pos(g.t, g.u);
    return g;
}
// The separations (ex, ey, ez) times scale, their squared distances and
// f(geometry, dx, dy, dz, MUL()): the integer forms where allow is set and every lane's pair permits them (all
// but dummies, coincident blobs and distances beyond 2^32 radii), else the FP64 ones.  ZPER pairs (dz an image's) take
// the latter.  SCALE: positions are subtracted before they are scaled to radii, so that blobs near each other and far
// from the origin keep their separation to the last bit (scaled first, it would carry the rounding of x / a: at 504
// blobs near the origin 5.4e-16 of M_UF against 2.3e-16, by extended precision); false:
// scale is 1.  Every lane of the warp calls this together (the choice of the form is the warp's, and with it the
// rounding: it must not depend on which lanes happen to run in step).  allow also stands for a scale within 2^+-64.  Three integer products a pair: M_UF of 10,752 blobs
// 3.69 -> 3.77 ms (4.03 with FP64 multiplies; 3.73 since the vote is the whole warp's).
template <bool ZPER, bool SCALE, class F>
__device__ __forceinline__ void with_pair_geo_d(double ex, double ey, double ez, double scale, double Rz, double hi,
                                                double hj, bool allow, F &&f)
{
    if (!ZPER && allow) {
        const double dx = SCALE ? int_mul_signed(ex, scale) : ex, dy = SCALE ? int_mul_signed(ey, scale) : ey,
                     dz = SCALE ? int_mul_signed(ez, scale) : ez;
        const double q2 = int_fma_pos(dz, dz, int_fma_pos(dx, dx, int_mul_signed(dy, dy)));
        if (__all_sync(0xffffffffu, int_range_mag(ex, ey, ez) && int_range_sep(Rz, Rz, Rz) && int_range(q2))) {
            f(pair_geo_d<MulInt>(q2, int_fma_pos(4.0 * hi, hj, q2)), dx, dy, dz, MulInt());
            return;
        }
    }
    const double dx = SCALE ? ex * scale : ex, dy = SCALE ? ey * scale : ey, dz = SCALE ? ez * scale : ez;
    const double rho2 = fma(dx, dx, dy * dy), r2 = fma(dz, dz, rho2);
    f(pair_geo_d<MulFp64>(r2, ZPER ? fma(Rz, Rz, rho2) : fma(4.0 * hi, hj, r2)), dx, dy, dz, MulFp64());
}
struct UFBlockD {
    double Af, b2, t3, t4, zz;
};
template <bool ZPER, class MUL = MulFp64>
__device__ __forceinline__ UFBlockD uf_block_d(const PairGeoD &g, double dz, double Rz, double hi, double hj,
                                               MUL = MUL())
{
    const double k1 = MUL::fma_pos(3.0 * hi, hj, 1.0), z2 = MUL::pos(Rz, Rz);  // 3 h_i h_j + 1
    double ia = g.invr, a3 = MUL::pos(g.i2, g.invr);
    double Bc = MUL::pos(MUL::fma_any(g.i2, -3.0, 1.5), a3);  // positive where it is used (r > 2)
    const bool near = MUL::le4(g.r2);                // r <= 2
    if (__any_sync(__activemask(), near)) {
        if (near) {
            ia = 0.0;
            a3 = fma(-0.5625, g.r2 * g.invr, 2.0);
            Bc = 0.1875 * g.invr;
        }
    }
    const double s = g.s, u = g.u, t = g.t, p = g.p;
    const double E = MUL::pos(z2, u);
    const double b1 = MUL::fma_pos(z2, 3.0, 1.0);
    const double w5 = MUL::fma_any(E, -5.0, b1), w7 = MUL::fma_any(E, -7.0, b1);
    const double Y = MUL::fma_any(MUL::mul(u, w7), -5.0, MUL::fma_pos(9.0 * hi, hj, 3.0));
    const double Y10 = MUL::fma_any(u, -10.0, Y);
    const double Z = fma(z2, fma(-20.0, u, Y10) + 6.0, 4.0);
    const double X = MUL::mul(MUL::pos(Rz, p), Y10);
    UFBlockD m;
    m.Af = fma(p, w5, fma(-k1, t, fma(1.5, ia - s, a3)));
    const double F = MUL::fma_any(t, -1.5, Bc);
    m.b2 = MUL::fma_any(p, Y, F);
    double G, dG;  // dz F, dz^2 F
    if constexpr (ZPER) {
        const double dw = hi - hj, x = dz * Bc, w = -1.5 * t * dw;
        G = x + w;
        dG = fma(dz, x, dw * w);
    } else {
        G = MUL::mul(dz, F);
        dG = MUL::mul(dz, G);
    }
    m.t3 = G - X;
    m.t4 = G + X;
    m.zz = fma(-p, Z, m.Af + dG);
    return m;
}
// (ux, uy, uz) += (3/2) M v; with t3 and t4 exchanged, the transposed block.
// V: MulInt where all vectors are within int_range_vec.
template <class V>
__device__ __forceinline__ void uf_block_acc_d(const UFBlockD &m, double t3, double t4, double dx, double dy,
                                               double vx, double vy, double vz, double &ux, double &uy, double &uz)
{
    const double P = fma(dy, vy, V::mul(dx, vx));
    const double G = fma(t3, vz, V::mul(m.b2, P));
    ux = fma(G, dx, fma(m.Af, vx, ux));
    uy = fma(G, dy, fma(m.Af, vy, uy));
    uz = fma(t4, P, fma(m.zz, vz, uz));
}

// UT, WF and WT for both orders of a pair in FP64, the formulas of
// rot_block_df and wt_block_df (pair_math_df.cuh), where they are derived: 64
// (UT, WF) and 62 (WT) operations a pair against 91 and 74 of the tensor
// forms, about half of them on the integer pipes (MulInt).  10,752 blobs: UT
// 9.82 -> 3.98 ms, WF 9.97 -> 4.10, WT 8.08 -> 3.80.  UF32: the blocks times 3/2, as the UF block (for sums of both).
struct RotBlockD {
    double a, ar, b, ei, ej, wi, wj;
};
template <bool UF32 = false, class MUL = MulFp64>
__device__ __forceinline__ RotBlockD rot_block_d(const PairGeoD &g, double dz, double Rz, double hi, double hj,
                                                 MUL = MUL())
{
    constexpr double f = UF32 ? 1.5 : 1.0;
    double c = MUL::pos(g.i2, g.invr);
    const bool near = MUL::lt4(g.r2);  // r < 2
    if (__any_sync(__activemask(), near)) {
        if (near) c = fma(-0.1875, g.r2 * g.invr, 0.5);
    }
    RotBlockD k;
    k.b = UF32 ? 1.5 * (g.t - c) : g.t - c;
    const double m = MUL::mul(dz, k.b), Rp = MUL::pos(Rz, g.p), Ru = MUL::pos(Rz, g.u);
    k.a = fma(2.0 * f, Rp, -m);
    k.ar = fma(2.0 * f, Rp, m);
    const double R10 = 10.0 * f * Ru, R6 = 6.0 * f * Rz, y = fma(-10.0 * f * Rz, Ru, 2.0 * f);
    k.ei = MUL::mul(g.p, fma(-6.0 * f, hi, R10));
    k.ej = MUL::mul(g.p, fma(-6.0 * f, hj, R10));
    k.wi = fma(g.p, fma(R6, hi, y), k.b);
    k.wj = fma(g.p, fma(R6, hj, y), k.b);
    return k;
}
template <bool UF32 = false, class MUL = MulFp64>
__device__ __forceinline__ UFBlockD wt_block_d(const PairGeoD &g, double dz, double Rz, MUL = MUL())
{
    constexpr double f = UF32 ? 1.5 : 1.0;
    const double i3 = MUL::pos(g.i2, g.invr);
    double A = -0.5 * f * i3, Bc = 1.5 * f * MUL::pos(g.i2, i3);
    const bool near = MUL::lt4(g.r2);
    if (__any_sync(__activemask(), near)) {
        if (near) {
            const double r = g.r2 * g.invr;
            A = f * fma(fma(0.078125, g.r2, -0.84375), r, 1.0);
            Bc = f * fma(-0.046875, r, 0.28125 * g.invr);
        }
    }
    const double Ru = MUL::pos(Rz, g.u), Et = MUL::pos(MUL::pos(Rz, Ru), g.t);
    const double D = MUL::mul(Bc, dz), X = 1.5 * f * MUL::pos(g.p, Rz);
    UFBlockD m;
    m.Af = fma(-6.0 * f, Et, fma(3.5 * f, g.t, A));
    m.b2 = fma(-4.5 * f, g.p, Bc);
    m.t3 = D - X;
    m.t4 = D + X;
    m.zz = fma(D, dz, fma(-1.5 * f, Et, fma(0.5 * f, g.t, A)));
    return m;
}
template <class V>
__device__ __forceinline__ void ut_acc_d(const RotBlockD &k, double dx, double dy, double vx, double vy, double vz,
                                         double qx, double qy, double qz, double &ux, double &uy, double &uz,
                                         double &wx, double &wy, double &wz)
{
    const double Q = fma(dy, vx, -V::mul(dx, vy)), Qq = fma(dy, qx, -V::mul(dx, qy));
    const double bv = V::mul(k.b, vz), eQ = V::mul(k.ei, Q), bq = V::mul(k.b, qz), eq = V::mul(k.ej, Qq);
    ux = fma(k.a, vy, fma(bv, dy, fma(eQ, dx, ux)));
    uy = fma(-k.a, vx, fma(-bv, dx, fma(eQ, dy, uy)));
    uz = fma(-k.wi, Q, uz);
    wx = fma(k.ar, qy, fma(-bq, dy, fma(eq, dx, wx)));
    wy = fma(-k.ar, qx, fma(bq, dx, fma(eq, dy, wy)));
    wz = fma(k.wj, Qq, wz);
}
template <class V>
__device__ __forceinline__ void wf_acc_d(const RotBlockD &k, double dx, double dy, double vx, double vy, double vz,
                                         double qx, double qy, double qz, double &ux, double &uy, double &uz,
                                         double &wx, double &wy, double &wz)
{
    const double Q = fma(dy, vx, -V::mul(dx, vy)), Qq = fma(dy, qx, -V::mul(dx, qy));
    const double H = fma(k.ej, fma(dy, vy, V::mul(dx, vx)), V::mul(k.wj, vz));
    const double Hq = fma(k.ei, fma(dy, qy, V::mul(dx, qx)), -V::mul(k.wi, qz));
    ux = fma(-k.ar, vy, fma(H, dy, ux));
    uy = fma(k.ar, vx, fma(-H, dx, uy));
    uz = fma(-k.b, Q, uz);
    wx = fma(-k.a, qy, fma(Hq, dy, wx));
    wy = fma(k.a, qx, fma(-Hq, dx, wy));
    wz = fma(k.b, Qq, wz);
}

// ---------------------------------------------------------------------------
// Symmetric forms of the rotation blocks in FP32: M_ji is the M_ij formula
// with d -> -d and h_i <-> h_j, so one pair evaluation serves both targets.
// WT has no height dependence; UT and WF form the height-dependent
// coefficients for both heights.
template <typename T> __device__ __forceinline__ T fm(T a, T b, T c);
template <> __device__ __forceinline__ float fm<float>(float a, float b, float c) { return fmaf(a, b, c); }
template <> __device__ __forceinline__ double fm<double>(double a, double b, double c) { return fma(a, b, c); }

template <typename T> struct RotH {
    T f3s2, p, gs;  // f3 s^2, p = s^2 ez + f4, g s with g = s^2 + f2 + f3 ez
};
template <typename T>
__device__ __forceinline__ RotH<T> rot_h(T h, T s, T s2, T s3, T ez, T ezs4, T K)
{
    const T hs3 = h * s3;
    const T f2 = T(2) * fm<T>(T(6) * hs3, ez, K);
    const T f3 = T(-2) * fm<T>(T(3), hs3, T(-5) * ezs4);
    const T f4 = T(-2) * (hs3 - ezs4);
    const T p = fm<T>(s2, ez, f4);
    const T g = fm<T>(f3, ez, s2 + f2);
    return {f3 * s2, p, g * s};
}

template <typename T>
__device__ __forceinline__ void ut_apply(T c, const RotH<T> &H, T s3, T dx, T dy, T dz, T vx, T vy, T vz, T &ux,
                                         T &uy, T &uz)
{
    const T Q = fm<T>(dy, vx, -dx * vy);  // (v x d)_z
    const T X = fm<T>(vy, dz, -vz * dy), Y = fm<T>(vz, dx, -vx * dz);
    const T F3 = H.f3s2 * Q, F1 = s3 * vz;
    ux = fm<T>(c, X, fm<T>(F3, dx, fm<T>(F1, dy, fm<T>(H.p, vy, ux))));
    uy = fm<T>(c, Y, fm<T>(F3, dy, fm<T>(-F1, dx, fm<T>(-H.p, vx, uy))));
    uz = fm<T>(c - H.gs, Q, uz);
}

template <typename T>
__device__ __forceinline__ void wf_apply(T c, const RotH<T> &H, T s3, T dx, T dy, T dz, T vx, T vy, T vz, T &ux,
                                         T &uy, T &uz)
{
    const T Pxy = fm<T>(dy, vy, dx * vx);
    const T Q = fm<T>(dy, vx, -dx * vy);
    const T X = fm<T>(vy, dz, -vz * dy), Y = fm<T>(vz, dx, -vx * dz);
    const T Hh = fm<T>(H.f3s2, Pxy, H.gs * vz);
    ux = fm<T>(c, X, fm<T>(Hh, dy, fm<T>(-H.p, vy, ux)));
    uy = fm<T>(c, Y, fm<T>(H.p, vx, fm<T>(-Hh, dx, uy)));
    uz = fm<T>(c - s3, Q, uz);
}

template <typename T>
__device__ __forceinline__ void wt_apply(T Af, T Bc, T s5, T dx, T dy, T dz, T Rz, T vx, T vy, T vz, T &ux, T &uy,
                                         T &uz)
{
    const T Pxy = fm<T>(dy, vy, dx * vx);
    const T dv = fm<T>(dz, vz, Pxy);
    const T W = fm<T>(Rz, vz, Pxy);
    const T Q = fm<T>(dy, vx, -dx * vy);
    const T Gw = T(-1.5) * s5 * W;
    const T Tq = T(3) * s5 * Q;
    const T Gr = Bc * dv;
    const T G = Gr + Gw;
    ux = fm<T>(Af, vx, fm<T>(G, dx, fm<T>(Tq, dy, ux)));
    uy = fm<T>(Af, vy, fm<T>(G, dy, fm<T>(-Tq, dx, uy)));
    uz = fm<T>(Af, vz, fm<T>(Gr, dz, fm<T>(-Gw, Rz, uz)));
}

// UT, WF or WT for both orders of one pair: (ux, uy, uz) += M_ij v_j,
// (wx, wy, wz) += M_ji v_i.
template <typename T, int KIND>
__device__ __forceinline__ void pair_rot_sym(T dx, T dy, T dz, T Rz, T hi, T hj, T vx, T vy, T vz, T qx, T qy, T qz,
                                             T &ux, T &uy, T &uz, T &wx, T &wy, T &wz)
{
    const T rho2 = fm<T>(dx, dx, dy * dy);
    const T r2 = fm<T>(dz, dz, rho2);
    const T invr = rsq<T>(r2);
    const T Rz2 = Rz * Rz;
    const T s = rsq<T>(rho2 + Rz2);
    const T s2 = s * s, s3 = s2 * s, E = Rz2 * s2;
    const bool near = !(r2 >= T(4));  // r < 2
    if (KIND == RMW_WT) {
        const T invr2 = invr * invr, invr3 = invr2 * invr;
        T A = T(-0.5) * invr3;
        T Bc = T(1.5) * invr2 * invr3;
        if (__any_sync(__activemask(), near)) {
            if (near) {
                const T r = r2 * invr;
                A = T(1) - T(0.84375) * r + T(0.078125) * r * r2;
                Bc = T(0.28125) * invr - T(0.046875) * r;
            }
        }
        const T s5 = s3 * s2;
        const T Af = fm<T>(T(0.5) * s3, fm<T>(T(-6), E, T(1)), A);
        wt_apply<T>(Af, Bc, s5, dx, dy, dz, Rz, vx, vy, vz, ux, uy, uz);
        wt_apply<T>(Af, Bc, s5, -dx, -dy, -dz, Rz, qx, qy, qz, wx, wy, wz);
    } else {
        T c = invr * invr * invr;
        if (__any_sync(__activemask(), near)) {
            if (near) c = T(0.5) * (T(1) - T(0.375) * (r2 * invr));
        }
        const T s4 = s2 * s2, ez = Rz * s, ezs4 = ez * s4;
        const T K = fm<T>(T(-10), E, T(1)) * s4;
        const RotH<T> Hi = rot_h<T>(hi, s, s2, s3, ez, ezs4, K);
        const RotH<T> Hj = rot_h<T>(hj, s, s2, s3, ez, ezs4, K);
        if (KIND == RMW_UT) {
            ut_apply<T>(c, Hi, s3, dx, dy, dz, vx, vy, vz, ux, uy, uz);
            ut_apply<T>(c, Hj, s3, -dx, -dy, -dz, qx, qy, qz, wx, wy, wz);
        } else {
            wf_apply<T>(c, Hj, s3, dx, dy, dz, vx, vy, vz, ux, uy, uz);
            wf_apply<T>(c, Hi, s3, -dx, -dy, -dz, qx, qy, qz, wx, wy, wz);
        }
    }
}

// Free-space blocks for both orders of one pair (the symmetric no-wall
// kernels): M_ji = M_ij(-d), so UF and WT (even in d) apply the same block to
// the other vector and UT / WF (odd in d) its negative.  (ux, uy, uz) +=
// M_ij v, (wx, wy, wz) += M_ji q.
template <typename T, int KIND, class MUL>
__device__ __forceinline__ void pair_rpy_sym_body(T r2, T invr, T dx, T dy, T dz, T vx, T vy, T vz, T qx, T qy, T qz,
                                                  T &ux, T &uy, T &uz, T &wx, T &wy, T &wz)
{
    if (KIND == RMW_UT || KIND == RMW_WF) {
        T c = MUL::pos(MUL::pos(invr, invr), invr);
        const bool near = MUL::lt4(r2);  // r < 2
        if (__any_sync(__activemask(), near)) {
            if (near) c = T(0.5) * (T(1) - T(0.375) * (r2 * invr));
        }
        ux = fm<T>(c, fm<T>(vy, dz, -MUL::mul(vz, dy)), ux);
        uy = fm<T>(c, fm<T>(vz, dx, -MUL::mul(vx, dz)), uy);
        uz = fm<T>(c, fm<T>(dy, vx, -MUL::mul(dx, vy)), uz);
        wx = fm<T>(-c, fm<T>(qy, dz, -MUL::mul(qz, dy)), wx);
        wy = fm<T>(-c, fm<T>(qz, dx, -MUL::mul(qx, dz)), wy);
        wz = fm<T>(-c, fm<T>(dy, qx, -MUL::mul(dx, qy)), wz);
        return;
    }
    const T invr2 = MUL::pos(invr, invr);
    T A, Bc;
    if (KIND == RMW_UF) {
        A = MUL::pos(T(1) + T(2.0 / 3.0) * invr2, invr);
        Bc = MUL::pos(MUL::pos(T(1) - T(2) * invr2, invr2), invr);  // positive where it is used
        const bool near = MUL::le4(r2);  // r <= 2
        if (__any_sync(__activemask(), near)) {
            if (near) {
                const T r = r2 * invr;
                A = T(4.0 / 3.0) * (T(1) - T(0.28125) * r);
                Bc = T(0.125) * invr;
            }
        }
    } else {  // RMW_WT
        const T invr3 = MUL::pos(invr2, invr);
        A = T(-0.5) * invr3;
        Bc = MUL::pos(T(1.5) * invr2, invr3);
        const bool near = MUL::lt4(r2);
        if (__any_sync(__activemask(), near)) {
            if (near) {
                const T r = r2 * invr;
                A = T(1) - T(0.84375) * r + T(0.078125) * r * r2;
                Bc = T(0.28125) * invr - T(0.046875) * r;
            }
        }
    }
    const T G = MUL::mul(Bc, fm<T>(dx, vx, fm<T>(dy, vy, MUL::mul(dz, vz))));
    const T Gq = MUL::mul(Bc, fm<T>(dx, qx, fm<T>(dy, qy, MUL::mul(dz, qz))));
    ux = fm<T>(A, vx, fm<T>(G, dx, ux));
    uy = fm<T>(A, vy, fm<T>(G, dy, uy));
    uz = fm<T>(A, vz, fm<T>(G, dz, uz));
    wx = fm<T>(A, qx, fm<T>(Gq, dx, wx));
    wy = fm<T>(A, qy, fm<T>(Gq, dy, wy));
    wz = fm<T>(A, qz, fm<T>(Gq, dz, wz));
}
template <typename T, int KIND>
__device__ __forceinline__ void pair_rpy_sym(T dx, T dy, T dz, T vx, T vy, T vz, T qx, T qy, T qz, T &ux, T &uy,
                                             T &uz, T &wx, T &wy, T &wz, bool allow = false)
{
    if constexpr (std::is_same<T, double>::value) {
        if (allow) {  // as with_pair_geo_d, by whole warps too
            const double q2 = int_fma_pos(dx, dx, int_fma_pos(dy, dy, int_mul_signed(dz, dz)));
            if (__all_sync(0xffffffffu, int_range_sep(dx, dy, dz) && int_range(q2))) {
                pair_rpy_sym_body<T, KIND, MulInt>(q2, int_rsqrt(q2), dx, dy, dz, vx, vy, vz, qx, qy, qz, ux, uy, uz,
                                                   wx, wy, wz);
                return;
            }
        }
    }
    const T r2 = fm<T>(dx, dx, fm<T>(dy, dy, dz * dz));
    pair_rpy_sym_body<T, KIND, MulPipe<T>>(r2, rsq<T>(r2), dx, dy, dz, vx, vy, vz, qx, qy, qz, ux, uy, uz, wx, wy, wz);
}

// Free-space RPY blocks (no wall): the RPY parts of pair_contrib, for the
// no-wall products (mobility/mobility_numba.py:13-1190).  (dx, dy, dz) =
// (r_i - r_j)/a.  Accumulates M_ij v into (ux, uy, uz), unscaled.
template <int KIND, typename T>
__device__ __forceinline__ void pair_rpy(T dx, T dy, T dz, T vx, T vy, T vz, T &ux, T &uy, T &uz)
{
    const T r2 = dx * dx + dy * dy + dz * dz;
    const T invr = rsq<T>(r2);
    const T r = r2 * invr;
    const T dv = dx * vx + dy * vy + dz * vz;
    if (KIND == RMW_UF) {
        const T invr2 = invr * invr;
        T A = (T(1) + T(2.0 / 3.0) * invr2) * invr;
        T Bc = (T(1) - T(2) * invr2) * invr2 * invr;
        const bool near = !(r > T(2));
        if (__any_sync(__activemask(), near)) {
            if (near) {
                A = T(4.0 / 3.0) * (T(1) - T(0.28125) * r);
                Bc = T(0.125) * invr;
            }
        }
        const T G = Bc * dv;
        ux += A * vx + G * dx;
        uy += A * vy + G * dy;
        uz += A * vz + G * dz;
    } else if (KIND == RMW_UT || KIND == RMW_WF) {
        T c = invr * invr * invr;
        const bool near = !(r >= T(2));
        if (__any_sync(__activemask(), near)) {
            if (near) c = T(0.5) * (T(1) - T(0.375) * r);
        }
        ux += c * (vy * dz - vz * dy);
        uy += c * (vz * dx - vx * dz);
        uz += c * (dy * vx - dx * vy);
    } else {  // RMW_WT
        const T invr2 = invr * invr;
        const T invr3 = invr2 * invr;
        T A = T(-0.5) * invr3;
        T Bc = T(1.5) * invr2 * invr3;
        const bool near = !(r >= T(2));
        if (__any_sync(__activemask(), near)) {
            if (near) {
                A = T(1) - T(0.84375) * r + T(0.078125) * r * r2;
                Bc = T(0.28125) * invr - T(0.046875) * r;
            }
        }
        const T G = Bc * dv;
        ux += A * vx + G * dx;
        uy += A * vy + G * dy;
        uz += A * vz + G * dz;
    }
}

// Minimum-image projection of mobility/mobility_numba.py (int() truncates toward zero).
template <typename T> __device__ __forceinline__ T project(T d, T L)
{
    T s = (T)((d > T(0)) - (d < T(0)));
    return d - (T)(long long)(d / L + T(0.5) * s) * L;
}

}  // namespace rmw
