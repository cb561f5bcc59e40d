// The single-wall RPY pair formulas of pair_math.cuh in double-float
// arithmetic (df64 mode).  Same algebra (division-free, two reciprocal square
// roots per pair); exact float constants multiply with the cheaper df x float
// product, powers of two scale exactly.
#pragma once
#include "dfloat.cuh"
#include "f32x2.cuh"
#include "rmw_common.cuh"

namespace rmw {

struct dfc {
    // compile-time split of a double constant into hi + lo floats
    static constexpr df make(double d) { return {(float)d, (float)(d - (double)(float)d)}; }
};

// Writes the pair's contribution M_ij v_j (unscaled) to (ux, uy, uz).
template <int KIND>
__device__ __forceinline__ void pair_contrib_df(df dx, df dy, df dz, df Rz, df hi, df hj, df vx, df vy, df vz,
                                                df &ux, df &uy, df &uz)
{
    constexpr df TWO_THIRDS = dfc::make(2.0 / 3.0);
    constexpr df FOUR_THIRDS = dfc::make(4.0 / 3.0);
    constexpr df TEN_THIRDS = dfc::make(10.0 / 3.0);
    const df rho2 = mad(dx, dx, sqr(dy));
    const df r2 = mad(dz, dz, rho2);
    const df invr = rsqrt_df(r2);
    const df r = r2 * invr;
    const df Rz2 = sqr(Rz);
    const df s = rsqrt_df(rho2 + Rz2);
    const df s2 = sqr(s);
    const df s3 = s2 * s;
    const df E = Rz2 * s2;  // e_z^2
    const df Pxy = mad2(dx, vx, dy, vy);
    if (KIND == RMW_UF) {
        const df invr2 = sqr(invr);
        df A = mad(TWO_THIRDS, invr2, df_from(1.0f)) * invr;
        df Bc = (1.0f - scale2(invr2, 2.0f)) * invr2 * invr;
        const bool near = !(r > 2.0f);
        if (__any_sync(__activemask(), near)) {
            if (near) {
                A = FOUR_THIRDS * (1.0f - r * 0.28125f);
                Bc = scale2(invr, 0.125f);
            }
        }
        const df dv = mad(dz, vz, Pxy);
        const df W = mad(Rz, vz, Pxy);
        const df s5 = s3 * s2;
        const df hh = hi * hj * s2;
        const df ez = Rz * s;
        const df q5 = (1.0f - E * 5.0f) * s3;
        const df f1 = -mad(scale2(hh, 2.0f) + 1.0f, s, TWO_THIRDS * ((1.0f - E * 3.0f) * s3 - q5 * s2));
        const df f2 = -(mad((1.0f - hh * 6.0f), s, -scale2(q5, 2.0f)) + TEN_THIRDS * ((1.0f - E * 7.0f) * s5));
        const df f3 = TWO_THIRDS * (hj * s2 * 3.0f - (hh * ez * s) * 18.0f +
                                    ez * (((2.0f - E * 7.0f) * s5) * 10.0f - q5 * 6.0f));
        const df f4 = TWO_THIRDS * (hj * s2 * 3.0f - (ez * s5) * 10.0f);
        const df f5 = -FOUR_THIRDS * mad((sqr(hj) + E) * 3.0f, s3, (2.0f - E * 15.0f) * s5);
        const df Af = A + f1;
        const df Gr = Bc * dv;
        const df Gw = mad(f2 * W, s, f3 * vz) * s;
        const df G = Gr + Gw;
        ux = mad2(Af, vx, G, dx);
        uy = mad2(Af, vy, G, dy);
        uz = mad2(Af, vz, Gr, dz) + mad2(Gw, Rz, f4 * W, s) + f5 * vz;
    } else if (KIND == RMW_UT || KIND == RMW_WF) {
        df c = sqr(invr) * invr;
        const bool near = !(r >= 2.0f);
        if (__any_sync(__activemask(), near)) {
            if (near) c = scale2(1.0f - r * 0.375f, 0.5f);
        }
        const df Q = mad2(dy, vx, -dx, vy);  // (v x d)_z
        df ax = c * mad2(vy, dz, -vz, dy);
        df ay = c * mad2(vz, dx, -vx, dz);
        df az = c * Q;
        const df s4 = sqr(s2);
        const df ez = Rz * s;
        const df h = (KIND == RMW_UT) ? hi : hj;
        const df hs3 = h * s3;
        const df ezs4 = ez * s4;
        const df f2 = scale2(mad(hs3 * 6.0f, ez, (1.0f - E * 10.0f) * s4), 2.0f);
        const df f3 = scale2(hs3 * 3.0f - ezs4 * 5.0f, -2.0f);
        const df f4 = scale2(hs3 - ezs4, -2.0f);
        const df p = mad(s2, ez, f4);
        const df g = mad(f3, ez, s2 + f2);
        if (KIND == RMW_UT) {
            const df F3 = f3 * s2 * Q;
            const df F1 = s3 * vz;
            ax = ax + mad2(F3, dx, F1, dy) + p * vy;
            ay = ay + mad2(F3, dy, -F1, dx) - p * vx;
            az = az - g * s * Q;
        } else {
            const df H = mad2(f3 * s2, Pxy, g * s, vz);
            ax = ax + mad2(H, dy, -p, vy);
            ay = ay + mad2(p, vx, -H, dx);
            az = az - s3 * Q;
        }
        ux = ax;
        uy = ay;
        uz = az;
    } else {  // RMW_WT
        const df invr2 = sqr(invr);
        const df invr3 = invr2 * invr;
        df A = invr3 * -0.5f;
        df Bc = (invr2 * invr3) * 1.5f;
        const bool near = !(r >= 2.0f);
        if (__any_sync(__activemask(), near)) {
            if (near) {
                A = (1.0f - r * 0.84375f) + (r * r2) * 0.078125f;
                Bc = invr * 0.28125f - r * 0.046875f;
            }
        }
        const df dv = mad(dz, vz, Pxy);
        const df W = mad(Rz, vz, Pxy);
        const df Q = mad2(dy, vx, -dx, vy);
        const df s5 = s3 * s2;
        const df Af = A + scale2((1.0f - E * 6.0f) * s3, 0.5f);
        const df Gw = (s5 * W) * -1.5f;
        const df Tq = (s5 * Q) * 3.0f;
        const df Gr = Bc * dv;
        const df G = Gr + Gw;
        ux = mad2(Af, vx, G, dx) + Tq * dy;
        uy = mad2(Af, vy, G, dy) - Tq * dx;
        uz = mad2(Af, vz, Gr, dz) - Gw * Rz;
    }
}

// Free-space RPY block (no wall) in double-float: writes M_ij v (unscaled) to
// (ux, uy, uz); the double-float form of pair_rpy (pair_math.cuh).
template <int KIND>
__device__ __forceinline__ void pair_rpy_df(df dx, df dy, df dz, df vx, df vy, df vz, df &ux, df &uy, df &uz)
{
    constexpr df TWO_THIRDS = dfc::make(2.0 / 3.0);
    constexpr df FOUR_THIRDS = dfc::make(4.0 / 3.0);
    const df r2 = mad(dz, dz, mad(dx, dx, sqr(dy)));
    const df invr = rsqrt_df(r2);
    const df r = r2 * invr;
    const df dv = mad(dz, vz, mad2(dx, vx, dy, vy));
    if (KIND == RMW_UF) {
        const df invr2 = sqr(invr);
        df A = mad(TWO_THIRDS, invr2, df_from(1.0f)) * invr;
        df Bc = (1.0f - scale2(invr2, 2.0f)) * invr2 * invr;
        const bool near = !(r > 2.0f);
        if (__any_sync(__activemask(), near)) {
            if (near) {
                A = FOUR_THIRDS * (1.0f - r * 0.28125f);
                Bc = scale2(invr, 0.125f);
            }
        }
        const df G = Bc * dv;
        ux = mad2(A, vx, G, dx);
        uy = mad2(A, vy, G, dy);
        uz = mad2(A, vz, G, dz);
    } else if (KIND == RMW_UT || KIND == RMW_WF) {
        df c = sqr(invr) * invr;
        const bool near = !(r >= 2.0f);
        if (__any_sync(__activemask(), near)) {
            if (near) c = scale2(1.0f - r * 0.375f, 0.5f);
        }
        ux = c * mad2(vy, dz, -vz, dy);
        uy = c * mad2(vz, dx, -vx, dz);
        uz = c * mad2(dy, vx, -dx, vy);
    } else {
        const df invr2 = sqr(invr);
        const df invr3 = invr2 * invr;
        df A = invr3 * -0.5f;
        df Bc = (invr2 * invr3) * 1.5f;
        const bool near = !(r >= 2.0f);
        if (__any_sync(__activemask(), near)) {
            if (near) {
                A = (1.0f - r * 0.84375f) + (r * r2) * 0.078125f;
                Bc = invr * 0.28125f - r * 0.046875f;
            }
        }
        const df G = Bc * dv;
        ux = mad2(A, vx, G, dx);
        uy = mad2(A, vy, G, dy);
        uz = mad2(A, vz, G, dz);
    }
}

// UF as an explicit block, times 3/2 (which turns the RPY and Swan-Brady
// constants into exact floats; the finalize kernels multiply the pair sums by
// 2/3 in FP64).  With rho = (dx, dy), s = 1/R, u = s^2, t = s^3, p = s^5,
// E = (Rz s)^2, k = h_i h_j (so R^2 = r^2 + 4 k) and
//   F = Bc - (3/2) t,                  Bc = (3/2 - 3/r^2)/r^3
//   Y = 3 (1 + 3k) - 5 u (1 + 3 Rz^2 - 7 E)
//   X = Rz p (Y - 10 u)
// the block is, exactly,
//   M_xy part  = Af I + b2 rho rho^T,  b2 = F + p Y
//                Af = (3/2)(1/r - 1/R) + 1/r^3 - (1 + 3k) t + (1 + 3 Rz^2 - 5 E) p
//   M_xz = rho (dz F - X),   M_zx = rho (dz F + X)
//   M_zz = Af + dz^2 F - p (4 + Rz^2 (6 - 30 u + Y))
// and, for r <= 2, (3/2)/r + 1/r^3 -> 2 - 9r/16 and Bc -> 3/(16 r).  The
// transposed block (the reverse pair) exchanges the two z columns; it has no
// coefficient of its own.  Against the tensor form Af I + Bc d d^T + c2 e e^T
// + c3 e z^T + c4 z e^T + f5 z z^T this takes about 30 % fewer operations for a pair,
// both ways, with the same error (the 1/r - 1/R cancellation sets it in
// either): k replaces two height-dependent chains, X and D = dz F serve both
// off-diagonal columns, and an application is five dot products.
// D is df (one pair) or df2 (two pairs in packed lanes).  Products and sums
// stay unnormalised except where an error would grow (the squared distances,
// s^2 and 1/r^2): the low parts stay below 2^-22 of the terms they come from,
// so a product drops no more than the rounding of its operands (2^-46).  With
// the second-order step of rsqrt_df the error of a block, 2.3e-14 of its
// largest term, is below the 2.9e-14 of the fully normalised form with the
// first-order step (emulated in FP32 against extended precision over
// r = 2 .. 350 a).  Bounds used by the
// ordered sums: heights >= 1 (clamped by the wall regularisation), so k >= 1,
// Rz >= 2, u <= 1/4, E <= 1.
// p is held times kDfP and its partners (Y, Z, w5, ...) by 1 / kDfP, both
// exact: s^5 loses its low part 10^6 radii above the wall and vanishes at
// 10^8, while p Z and p w5 stay of the order of s and s^3.  2^100 keeps every
// term finite to 10^17 radii (2^64: to 10^14) and the low parts normal.
template <class D> struct UFBlockDF {
    D Af, b2, t3, t4, zz;
};

// lanes with r <= 2
__device__ __forceinline__ void uf_near_df(df r2, df invr, df &ia, df &a3, df &Bc)
{
    const bool near = !(r2 > 4.0f);
    if (__any_sync(__activemask(), near)) {
        if (near) {
            ia = df_from(0.f);
            a3 = scale2(1.0f - (r2 * invr) * 0.28125f, 2.0f);
            Bc = invr * 0.1875f;
        }
    }
}
__device__ __forceinline__ void uf_near_df(df2 r2, df2 invr, df2 &ia, df2 &a3, df2 &Bc)
{
    const df xa = {r2.hi.x, r2.lo.x}, xb = {r2.hi.y, r2.lo.y};
    const bool na = !(xa > 4.0f), nb = !(xb > 4.0f);
    if (__any_sync(__activemask(), na || nb)) {
        if (na) {
            const df v = {invr.hi.x, invr.lo.x};
            const df a = scale2(1.0f - (xa * v) * 0.28125f, 2.0f), b = v * 0.1875f;
            ia.hi.x = 0.f; ia.lo.x = 0.f;
            a3.hi.x = a.hi; a3.lo.x = a.lo;
            Bc.hi.x = b.hi; Bc.lo.x = b.lo;
        }
        if (nb) {
            const df v = {invr.hi.y, invr.lo.y};
            const df a = scale2(1.0f - (xb * v) * 0.28125f, 2.0f), b = v * 0.1875f;
            ia.hi.y = 0.f; ia.lo.y = 0.f;
            a3.hi.y = a.hi; a3.lo.y = a.lo;
            Bc.hi.y = b.hi; Bc.lo.y = b.lo;
        }
    }
}

// What the blocks of a pair share: r^2, 1/r, 1/r^2 and the powers of s = 1/R.
// h4 = 4 h_i, hj, Rz = h_i + h_j (may be unnormalised).  ZPER: dz is an
// image's and not h_i - h_j (= dw), so R^2 and the wall parts of G and zz are
// formed from the heights.
constexpr float kDfP = 0x1p100f;
template <class D> struct PairGeoDF {
    D r2, invr, i2, s, u, t, p;  // p = kDfP s^5
};
template <class D, bool ZPER = false>
__device__ __forceinline__ PairGeoDF<D> pair_geo_df(D dx, D dy, D dz, D Rz, D h4, D hj)
{
    PairGeoDF<D> g;
    const D rho2 = add_u(sqr_u(dx), sqr_u(dy));
    g.r2 = norm(add_u(sqr_u(dz), rho2));
    g.invr = rsqrt_df(g.r2);
    g.s = rsqrt_far_df(norm(ZPER ? add_u(rho2, sqr_u(Rz)) : add_u(g.r2, mul_u(h4, hj))));
    g.i2 = sqr(g.invr);
    g.u = sqr(g.s);
    g.t = mul_u(g.u, g.s);
    g.p = mul_u(g.t, scale2(g.u, kDfP));
    return g;
}

template <class D, bool ZPER = false>
__device__ __forceinline__ UFBlockDF<D> uf_block_df(const PairGeoDF<D> &g, D dz, D Rz, D h4, D hj, D dw = D{})
{
    const D k4 = mul_u(h4, hj), s = g.s, u = g.u, t = g.t, p = g.p;
    D ia = g.invr, a3 = mul_u(g.i2, g.invr);
    D Bc = mul_u(add_fast_u(1.5f, mul_u(g.i2, -3.0f)), a3);
    uf_near_df(g.r2, g.invr, ia, a3, Bc);
    const D z2 = sqr_u(Rz);
    const D E = mul_u(z2, u);
    constexpr float P = 1.0f / kDfP;
    const D w5 = add_fast_u(add_fast_u(mul_u(z2, 3.0f * P), P), mul_u(E, -5.0f * P));  // P (1 + 3 Rz^2 - 5 E)
    const D w7 = add_fast_u(w5, scale2(E, -2.0f * P));
    const D al = add_fast_u(mul_u(k4, 0.75f), 1.0f);  // 1 + 3 k
    UFBlockDF<D> m;
    m.Af = add_u(add_u(mul_u(sub_u(ia, s), 1.5f), a3), sub_u(mul_u(p, w5), mul_u(al, t)));
    const D F = add_u(Bc, mul_u(t, -1.5f));
    const D Y = add_fast_u(mul_u(al, 3.0f * P), mul_u(mul_u(u, w7), -5.0f));  // P times Y, and so on
    m.b2 = add_u(F, mul_u(p, Y));
    const D Y10 = add_fast_u(Y, mul_u(u, -10.0f * P));
    const D X = mul_u(mul_u(Rz, p), Y10);
    D G = mul_u(dz, F);  // dz F
    D dG = mul_u(dz, G);  // dz^2 F
    if constexpr (ZPER) {
        const D x = mul_u(dz, Bc), w = mul_u(mul_u(t, -1.5f), dw);
        G = add_u(x, w);
        dG = add_u(mul_u(dz, x), mul_u(dw, w));
    }
    m.t3 = sub_u(G, X);
    m.t4 = add_u(G, X);
    const D Z = add_fast_u(mul_u(z2, add_u(add_fast_u(6.0f * P, mul_u(u, -20.0f * P)), Y10)), 4.0f * P);
    m.zz = sub_u(add_u(m.Af, dG), mul_u(p, Z));
    return m;
}

// (ux, uy, uz) += (3/2) M v; with t3 and t4 exchanged, the transposed block
template <class D>
__device__ __forceinline__ void uf_block_acc_df(const UFBlockDF<D> &m, D t3, D t4, D dx, D dy, D vx, D vy, D vz,
                                                D &ux, D &uy, D &uz)
{
    const D P = mad2_u(dx, vx, dy, vy);
    const D G = mad2_u(m.b2, P, t3, vz);
    acc_dot2(ux, m.Af, vx, G, dx);
    acc_dot2(uy, m.Af, vy, G, dy);
    acc_dot2(uz, t4, P, m.zz, vz);
}

// ---------------------------------------------------------------------------
// The rotation blocks in tensor form, for the one-sided kernels: the UT
// coefficients take the target's height, the WF ones the source's, WT has
// none.

// The height-dependent coefficients of UT / WF for height h (unnormalised
// where only a sum consumes them).
struct RotHDF {
    df f3s2, p, gs;  // f3 s^2, p = s^2 ez + f4, g s with g = f3 ez + s^2 + f2
};
__device__ __forceinline__ RotHDF rot_h_df(df h, df s, df s2, df s3, df ez, df ezs4, df K)
{
    const df hs3 = h * s3;
    const df f2 = scale2(mad_u(hs3 * 6.0f, ez, K), 2.0f);
    const df f3 = scale2(mul_u(hs3, 3.0f) - mul_u(ezs4, 5.0f), -2.0f);
    const df f4 = scale2(sub_u(hs3, ezs4), -2.0f);
    const df p = mad(s2, ez, f4);
    const df g = mad(f3, ez, s2 + f2);
    return {f3 * s2, p, g * s};
}

// (ux, uy, uz) += M_UT v for the pair (d, coefficient set H)
__device__ __forceinline__ void ut_apply_df(df c, const RotHDF &H, df s3, df dx, df dy, df dz, df vx, df vy, df vz,
                                            df &ux, df &uy, df &uz)
{
    const df Q = mad2(dy, vx, -dx, vy);  // (v x d)_z
    const df X = mad2(vy, dz, -vz, dy), Y = mad2(vz, dx, -vx, dz);
    const df F3 = H.f3s2 * Q, F1 = s3 * vz;
    acc_dot4(ux, c, X, F3, dx, F1, dy, H.p, vy);
    acc_dot4(uy, c, Y, F3, dy, F1, -dx, H.p, -vx);
    acc_dot2(uz, c, Q, H.gs, -Q);
}

// (ux, uy, uz) += M_WF v for the pair (d, coefficient set H)
__device__ __forceinline__ void wf_apply_df(df c, const RotHDF &H, df s3, df dx, df dy, df dz, df vx, df vy, df vz,
                                            df &ux, df &uy, df &uz)
{
    const df Pxy = mad2(dx, vx, dy, vy);
    const df Q = mad2(dy, vx, -dx, vy);
    const df X = mad2(vy, dz, -vz, dy), Y = mad2(vz, dx, -vx, dz);
    const df Hh = mad2(H.f3s2, Pxy, H.gs, vz);
    acc_dot3(ux, c, X, Hh, dy, H.p, -vy);
    acc_dot3(uy, c, Y, H.p, vx, Hh, -dx);
    acc_dot2(uz, c, Q, s3, -Q);
}

// (ux, uy, uz) += M_WT v for the pair (d; Af = A + (1 - 6E) s^3 / 2, Bc, s^5)
__device__ __forceinline__ void wt_apply_df(df Af, df Bc, df s5, df dx, df dy, df dz, df Rz, df vx, df vy, df vz,
                                            df &ux, df &uy, df &uz)
{
    const df Pxy = mad2(dx, vx, dy, vy);
    const df dv = mad(dz, vz, Pxy);
    const df W = mad(Rz, vz, Pxy);
    const df Q = mad2(dy, vx, -dx, vy);
    const df Gw = (s5 * W) * -1.5f;
    const df Tq = (s5 * Q) * 3.0f;
    const df Gr = Bc * dv;
    const df G = Gr + Gw;
    acc_dot3(ux, Af, vx, G, dx, Tq, dy);
    acc_dot3(uy, Af, vy, G, dy, Tq, -dx);
    acc_dot3(uz, Af, vz, Gr, dz, Gw, -Rz);
}

// UT, WF and WT for both orders of a pair, two pairs in packed lanes.  With
// t = s^3, p = s^5, c the RPY factor (1/r^3, or (1 - 3r/8)/2 below 2),
// b = t - c, m = dz b, n = 2 Rz p and the two heights' coefficients
//   e_h = p (10 Rz u - 6 h),  W_h = b + p (2 - 10 E + 6 h Rz),
// the wall terms fold into a = n - m and a' = n + m (the heights' parts of
// s^2 ez + f4 are -dz t and +dz t, because Rz - 2 h_i = -dz), so that
//   UT_ij v = (a vy + b vz dy + e_i Q dx, -a vx - b vz dx + e_i Q dy, -W_i Q)
//   WF_ij v = (-a' vy + H dy, a' vx - H dx, -b Q),  H = e_j P + W_j vz
// with P = dx vx + dy vy, Q = dy vx - dx vy; the reverse blocks take the other
// height and a <-> a' with the signs of d.  WT, with the identity
// rho rho^T + rho' rho'^T = rho^2 I, has the five scalars of a UF block:
//   Af = A + 7t/2 - 6 E t,  b2 = Bc - 9p/2,  t3,4 = Bc dz -+ 3/2 p Rz,
//   zz = A + t/2 - 3/2 E t + Bc dz^2     (A = -1/(2 r^3), Bc = 3/(2 r^5)).
// About 500 FP32-pipe operations a pair against 720 (WT) and 840 (UT, WF) of
// the tensor forms above applied both ways.
struct RotBlockDF2 {
    df2 a, ar, b, ei, ej, wi, wj;
};

__device__ __forceinline__ void rot_near_c(df2 r2, df2 invr, df2 &c)
{
    const df xa = {r2.hi.x, r2.lo.x}, xb = {r2.hi.y, r2.lo.y};
    const bool na = !(xa >= 4.0f), nb = !(xb >= 4.0f);  // r < 2
    if (__any_sync(__activemask(), na || nb)) {
        if (na) {
            const df v = scale2(1.0f - (xa * df{invr.hi.x, invr.lo.x}) * 0.375f, 0.5f);
            c.hi.x = v.hi; c.lo.x = v.lo;
        }
        if (nb) {
            const df v = scale2(1.0f - (xb * df{invr.hi.y, invr.lo.y}) * 0.375f, 0.5f);
            c.hi.y = v.hi; c.lo.y = v.lo;
        }
    }
}
// r < 2: A = 1 - 27 r/32 + 5 r^3/64, Bc = 9/(32 r) - 3 r/64
__device__ __forceinline__ void wt_near(df2 r2, df2 invr, df2 &A, df2 &Bc)
{
    const df xa = {r2.hi.x, r2.lo.x}, xb = {r2.hi.y, r2.lo.y};
    const bool na = !(xa >= 4.0f), nb = !(xb >= 4.0f);
    if (__any_sync(__activemask(), na || nb)) {
        if (na) {
            const df v = {invr.hi.x, invr.lo.x}, r = xa * v;
            const df f = (1.0f - r * 0.84375f) + (r * xa) * 0.078125f, g = v * 0.28125f - r * 0.046875f;
            A.hi.x = f.hi; A.lo.x = f.lo;
            Bc.hi.x = g.hi; Bc.lo.x = g.lo;
        }
        if (nb) {
            const df v = {invr.hi.y, invr.lo.y}, r = xb * v;
            const df f = (1.0f - r * 0.84375f) + (r * xb) * 0.078125f, g = v * 0.28125f - r * 0.046875f;
            A.hi.y = f.hi; A.lo.y = f.lo;
            Bc.hi.y = g.hi; Bc.lo.y = g.lo;
        }
    }
}

// UF32: the block times 3/2, as the UF block (for sums of both); the factor
// only changes exact constants.
template <bool UF32 = false>
__device__ __forceinline__ RotBlockDF2 rot_block_df(const PairGeoDF<df2> &g, df2 dz, df2 Rz, df2 hi, df2 hj)
{
    constexpr float q = UF32 ? 1.5f : 1.0f, P = 1.0f / kDfP;  // y, R6, R10 times P
    df2 c = mul_u(g.i2, g.invr);
    rot_near_c(g.r2, g.invr, c);
    const df2 Ru = mul_u(Rz, g.u);
    const df2 y = add_u(mul_u(mul_u(Rz, Ru), -10.0f * q * P), df2_dup(df_from(2.0f * q * P)));
    RotBlockDF2 k;
    k.b = g.t - c;
    if constexpr (UF32) k.b = mul_u(k.b, 1.5f);
    const df2 m = mul_u(dz, k.b), Rp = mul_u(Rz, g.p), n = UF32 ? mul_u(Rp, 3.0f * P) : scale2(Rp, 2.0f * P);
    k.a = sub_u(n, m);
    k.ar = add_u(n, m);
    const df2 R10 = mul_u(Ru, 10.0f * q * P), R6 = mul_u(Rz, 6.0f * q * P);
    k.ei = mul_u(g.p, sub_u(R10, mul_u(hi, 6.0f * q * P)));
    k.ej = mul_u(g.p, sub_u(R10, mul_u(hj, 6.0f * q * P)));
    k.wi = add_u(k.b, mul_u(g.p, add_u(y, mul_u(R6, hi))));
    k.wj = add_u(k.b, mul_u(g.p, add_u(y, mul_u(R6, hj))));
    return k;
}

template <bool UF32 = false>
__device__ __forceinline__ UFBlockDF<df2> wt_block_df(const PairGeoDF<df2> &g, df2 dz, df2 Rz)
{
    constexpr float q = UF32 ? 1.5f : 1.0f, P = 1.0f / kDfP;
    const df2 i3 = mul_u(g.i2, g.invr);
    df2 A = scale2(i3, -0.5f), Bc = mul_u(mul_u(g.i2, i3), 1.5f);
    wt_near(g.r2, g.invr, A, Bc);
    if constexpr (UF32) {
        A = mul_u(A, q);
        Bc = mul_u(Bc, q);
    }
    const df2 Et = mul_u(mul_u(sqr_u(Rz), g.u), g.t);
    UFBlockDF<df2> m;
    m.Af = add_u(add_u(A, mul_u(g.t, 3.5f * q)), mul_u(Et, -6.0f * q));
    m.b2 = add_u(Bc, mul_u(g.p, -4.5f * q * P));
    const df2 D = mul_u(Bc, dz), X = mul_u(mul_u(g.p, Rz), 1.5f * q * P);
    m.t3 = sub_u(D, X);
    m.t4 = add_u(D, X);
    m.zz = add_u(add_u(A, mul_u(g.t, 0.5f * q)), add_u(mul_u(Et, -1.5f * q), mul_u(D, dz)));
    return m;
}

// u += UT v / WF v of the pair (i, j); w += the reverse block times q
__device__ __forceinline__ void ut_acc_df(const RotBlockDF2 &k, df2 dx, df2 dy, df2 vx, df2 vy, df2 vz, df2 qx, df2 qy,
                                          df2 qz, df2 &ux, df2 &uy, df2 &uz, df2 &wx, df2 &wy, df2 &wz)
{
    const df2 nx = -dx;
    {
        const df2 Q = mad2_u(dy, vx, nx, vy), bv = mul_u(k.b, vz), eQ = mul_u(k.ei, Q);
        acc_dot3(ux, k.a, vy, bv, dy, eQ, dx);
        acc_dot3(uy, -k.a, vx, bv, nx, eQ, dy);
        acc_dot1(uz, -k.wi, Q);
    }
    const df2 Q = mad2_u(dy, qx, nx, qy), bv = mul_u(k.b, qz), eQ = mul_u(k.ej, Q);
    acc_dot3(wx, k.ar, qy, -bv, dy, eQ, dx);
    acc_dot3(wy, -k.ar, qx, bv, dx, eQ, dy);
    acc_dot1(wz, k.wj, Q);
}
__device__ __forceinline__ void wf_acc_df(const RotBlockDF2 &k, df2 dx, df2 dy, df2 vx, df2 vy, df2 vz, df2 qx, df2 qy,
                                          df2 qz, df2 &ux, df2 &uy, df2 &uz, df2 &wx, df2 &wy, df2 &wz)
{
    const df2 nx = -dx;
    {
        const df2 P = mad2_u(dx, vx, dy, vy), Q = mad2_u(dy, vx, nx, vy), H = mad2_u(k.ej, P, k.wj, vz);
        acc_dot2(ux, -k.ar, vy, H, dy);
        acc_dot2(uy, k.ar, vx, H, nx);
        acc_dot1(uz, -k.b, Q);
    }
    const df2 P = mad2_u(dx, qx, dy, qy), Q = mad2_u(dy, qx, nx, qy), H = mad2_u(k.ei, P, -k.wi, qz);
    acc_dot2(wx, -k.a, qy, H, dy);
    acc_dot2(wy, k.a, qx, H, nx);
    acc_dot1(wz, k.b, Q);
}

// Free-space blocks for both orders of a pair: UF (times 3/2, as with the
// wall) and WT, even in d, A I + B d d^T; UT and WF, odd, c (v x d).
template <int KIND>
__device__ __forceinline__ void rpy_acc_df(df2 dx, df2 dy, df2 dz, df2 vx, df2 vy, df2 vz, df2 qx, df2 qy, df2 qz,
                                           df2 &ux, df2 &uy, df2 &uz, df2 &wx, df2 &wy, df2 &wz)
{
    const df2 r2 = norm(add_u(sqr_u(dz), add_u(sqr_u(dx), sqr_u(dy))));
    const df2 invr = rsqrt_df(r2);
    const df2 i2 = sqr(invr);
    if constexpr (KIND == RMW_UT || KIND == RMW_WF) {
        df2 c = mul_u(i2, invr);
        rot_near_c(r2, invr, c);
        const df2 nx = -dx, ny = -dy, nz = -dz;
        acc_dot1(ux, c, mad2_u(vy, dz, vz, ny));
        acc_dot1(uy, c, mad2_u(vz, dx, vx, nz));
        acc_dot1(uz, c, mad2_u(dy, vx, nx, vy));
        acc_dot1(wx, c, mad2_u(qz, dy, qy, nz));
        acc_dot1(wy, c, mad2_u(qx, dz, qz, nx));
        acc_dot1(wz, c, mad2_u(qy, dx, qx, ny));
        return;
    }
    df2 A, B;
    if constexpr (KIND == RMW_UF) {
        df2 ia = invr, a3 = mul_u(i2, invr);
        B = mul_u(add_fast_u(1.5f, mul_u(i2, -3.0f)), a3);
        uf_near_df(r2, invr, ia, a3, B);
        A = add_u(mul_u(ia, 1.5f), a3);
    } else {
        const df2 i3 = mul_u(i2, invr);
        A = scale2(i3, -0.5f);
        B = mul_u(mul_u(i2, i3), 1.5f);
        wt_near(r2, invr, A, B);
    }
    const df2 G = mul_u(B, add_u(mad2_u(dx, vx, dy, vy), mul_u(dz, vz)));
    const df2 Gq = mul_u(B, add_u(mad2_u(dx, qx, dy, qy), mul_u(dz, qz)));
    acc_dot2(ux, A, vx, G, dx);
    acc_dot2(uy, A, vy, G, dy);
    acc_dot2(uz, A, vz, G, dz);
    acc_dot2(wx, A, qx, Gq, dx);
    acc_dot2(wy, A, qy, Gq, dy);
    acc_dot2(wz, A, qz, Gq, dz);
}

// ---------------------------------------------------------------------------
// One-sided accumulating forms for the standard (all ordered pairs) kernels:
// (ux, uy, uz) += M_ij v_j, for UF times 3/2 (the finalize applies 2/3) with
// the coefficients and applies of the symmetric forms.
template <int KIND, bool ZPER = false>
__device__ __forceinline__ void pair_acc_df(df dx, df dy, df dz, df Rz, df hi, df hj, df vx, df vy, df vz, df &ux,
                                            df &uy, df &uz)
{
    if (KIND == RMW_UF) {
        const df h4 = scale2(hi, 4.0f);
        const UFBlockDF<df> m =
            uf_block_df<df, ZPER>(pair_geo_df<df, ZPER>(dx, dy, dz, Rz, h4, hj), dz, Rz, h4, hj, hi - hj);
        uf_block_acc_df(m, m.t3, m.t4, dx, dy, vx, vy, vz, ux, uy, uz);
        return;
    }
    const df rho2 = mad_u(dx, dx, sqr_u(dy));
    const df r2 = mad(dz, dz, rho2);
    const df invr = rsqrt_df(r2);
    const df Rz2 = sqr(Rz);
    const df s = rsqrt_df(rho2 + Rz2);
    const df s2 = sqr(s);
    const df s3 = s2 * s;
    const df E = Rz2 * s2;
    const bool near = !(r2 >= 4.0f);  // r < 2
    if (KIND == RMW_WT) {
        const df invr2 = sqr(invr);
        const df invr3 = invr2 * invr;
        df A = invr3 * -0.5f;
        df Bc = (invr2 * invr3) * 1.5f;
        if (__any_sync(__activemask(), near)) {
            if (near) {
                const df r = r2 * invr;
                A = (1.0f - r * 0.84375f) + (r * r2) * 0.078125f;
                Bc = invr * 0.28125f - r * 0.046875f;
            }
        }
        const df Af = A + scale2((1.0f - E * 6.0f) * s3, 0.5f);
        wt_apply_df(Af, Bc, s3 * s2, dx, dy, dz, Rz, vx, vy, vz, ux, uy, uz);
    } else {
        df c = sqr(invr) * invr;
        if (__any_sync(__activemask(), near)) {
            if (near) c = scale2(1.0f - (r2 * invr) * 0.375f, 0.5f);
        }
        const df s4 = sqr(s2);
        const df ez = Rz * s;
        const df ezs4 = ez * s4;
        const df K = mul_u(1.0f - mul_u(E, 10.0f), s4);
        if (KIND == RMW_UT) ut_apply_df(c, rot_h_df(hi, s, s2, s3, ez, ezs4, K), s3, dx, dy, dz, vx, vy, vz, ux, uy, uz);
        else wf_apply_df(c, rot_h_df(hj, s, s2, s3, ez, ezs4, K), s3, dx, dy, dz, vx, vy, vz, ux, uy, uz);
    }
}

}  // namespace rmw
