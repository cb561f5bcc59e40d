// Fused force-and-torque wall product:
//
//   U = M_UF F + M_UT T,    W = M_WF F + M_WT T     (W optional)
//
// in one pass over the pairs.  The reference's pycuda kernel
// velocity_from_force_and_torque (mobility/mobility_pycuda.py:1266-1392,
// wrapper mobility/mobility.py:384-411) returns U only; the 6N product
// [U; W] is what Lub_Solver.Wall_Mobility_Mult (Lubrication/Lub_Solver.py:
// 277-305) and the rollers' GMRES assemble from four separate products.  Here
// the four pair blocks are evaluated back to back on the same pair inputs:
// the pair functions are inlined, so the distances, the two reciprocal square
// roots and the powers of 1/R they share are formed once per pair.
//
// Scaling: with F' = b F and T' = b T / a (b the wall damping), and nf =
// 1/(8 pi eta a),
//   U_i = b_i nf       [ sum_j M_UF F'_j + M_UT T'_j + self(F'_i, T'_i) ]
//   W_i = b_i nf / a   [ sum_j M_WF F'_j + M_WT T'_j + self(F'_i, T'_i) ]
// because the four blocks carry 1/(8 pi eta a^p) with p = 1, 2, 2, 3.
//
// Same structure as the single products (wall_pair.cu): pack -> pair kernel
// over (target tiles) x (source chunks) -> finalize summing the chunks in
// fixed order (deterministic), adding the self terms and the scale.
// Precision modes as there: FP64; df64 (double-float on the FP32 pipe,
// <= 1e-12 against FP64); mixed (FP32 pairs from double-float position
// differences, compensated sums, <= 1e-6).
#include <algorithm>

#include "pair_math.cuh"
#include "pair_math_df.cuh"
#include "rmw_common.cuh"
#include "wall_pair.cuh"

namespace rmw {

namespace {

constexpr int kFtThreads = 128;  // targets per CTA
constexpr int kFtTile = 64;      // sources per shared-memory tile
constexpr int kFtDfGroup = 32;   // df64: sources per double-float group sum

struct FtImages {
    double Lx, Ly, Lz;  // periodic lengths over a (0 = not periodic)
};

// source records: positions over a (z clamped at a), F' and T'
struct __align__(16) FtSrcD {
    double x, y, z, pad0;
    double fx, fy, fz, pad1;
    double tx, ty, tz, pad2;
};
struct __align__(16) FtSrcF {
    float4 hi, lo;  // double-float positions over a
    float4 f, t;    // F', T' in FP32
};
struct __align__(16) FtSrcDF {
    float4 hi, lo;    // positions over a
    float4 fhi, flo;  // F'
    float4 thi, tlo;  // T'
};

__device__ __forceinline__ void ft_prep(const double *r, const double *F, const double *T, int i, double a,
                                        double &x, double &y, double &z, double f[3], double t[3])
{
    const double inva = 1.0 / a;
    const double zz = r[3 * i + 2];
    const double b = (zz < a) ? zz / a : 1.0;
    const double ze = (zz <= a) ? a : zz;
    x = r[3 * i] * inva;
    y = r[3 * i + 1] * inva;
    z = ze * inva;
    for (int c = 0; c < 3; ++c) {
        f[c] = b * F[3 * i + c];
        t[c] = b * T[3 * i + c] * inva;
    }
}

__global__ void ft_pack_fp64_kernel(const double *__restrict__ r, const double *__restrict__ F,
                                    const double *__restrict__ T, FtSrcD *__restrict__ src, int n, double a)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double x, y, z, f[3], t[3];
    ft_prep(r, F, T, i, a, x, y, z, f, t);
    FtSrcD s;
    s.x = x; s.y = y; s.z = z; s.pad0 = 0.0;
    s.fx = f[0]; s.fy = f[1]; s.fz = f[2]; s.pad1 = 0.0;
    s.tx = t[0]; s.ty = t[1]; s.tz = t[2]; s.pad2 = 0.0;
    src[i] = s;
}

__global__ void ft_pack_mixed_kernel(const double *__restrict__ r, const double *__restrict__ F,
                                     const double *__restrict__ T, FtSrcF *__restrict__ src, int n, double a)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double x, y, z, f[3], t[3];
    ft_prep(r, F, T, i, a, x, y, z, f, t);
    const float xh = (float)x, yh = (float)y, zh = (float)z;
    FtSrcF s;
    s.hi = make_float4(xh, yh, zh, 0.f);
    s.lo = make_float4((float)(x - (double)xh), (float)(y - (double)yh), (float)(z - (double)zh), 0.f);
    s.f = make_float4((float)f[0], (float)f[1], (float)f[2], 0.f);
    s.t = make_float4((float)t[0], (float)t[1], (float)t[2], 0.f);
    src[i] = s;
}

__global__ void ft_pack_df_kernel(const double *__restrict__ r, const double *__restrict__ F,
                                  const double *__restrict__ T, FtSrcDF *__restrict__ src, int n, double a)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double x, y, z, f[3], t[3];
    ft_prep(r, F, T, i, a, x, y, z, f, t);
    const df X = df_of_double(x), Y = df_of_double(y), Z = df_of_double(z);
    const df f0 = df_of_double(f[0]), f1 = df_of_double(f[1]), f2 = df_of_double(f[2]);
    const df t0 = df_of_double(t[0]), t1 = df_of_double(t[1]), t2 = df_of_double(t[2]);
    FtSrcDF s;
    s.hi = make_float4(X.hi, Y.hi, Z.hi, 0.f);
    s.lo = make_float4(X.lo, Y.lo, Z.lo, 0.f);
    s.fhi = make_float4(f0.hi, f1.hi, f2.hi, 0.f);
    s.flo = make_float4(f0.lo, f1.lo, f2.lo, 0.f);
    s.thi = make_float4(t0.hi, t1.hi, t2.hi, 0.f);
    s.tlo = make_float4(t0.lo, t1.lo, t2.lo, 0.f);
    src[i] = s;
}

// the periodic images the single products use: minimum image, then the
// neighbouring boxes along every periodic direction
template <typename T, typename F>
__device__ __forceinline__ void for_images(T rx, T ry, T rz, T Lx, T Ly, T Lz, bool self_pair, F &&f)
{
    if (Lx > T(0)) rx = project(rx, Lx);
    if (Ly > T(0)) ry = project(ry, Ly);
    if (Lz > T(0)) rz = project(rz, Lz);
    const int px = Lx > T(0), py = Ly > T(0), pz = Lz > T(0);
    for (int bx = -px; bx <= px; ++bx)
        for (int by = -py; by <= py; ++by)
            for (int bz = -pz; bz <= pz; ++bz) {
                const bool self = self_pair && bx == 0 && by == 0 && bz == 0;
                if (!self) f(rx + bx * Lx, ry + by * Ly, rz + bz * Lz);
            }
}

// ---------------------------------------------------------------------------
// FP64
template <bool WITH_W, bool PER>
__global__ void __launch_bounds__(kFtThreads) ft_pair_fp64_kernel(const FtSrcD *__restrict__ src, int n, int chunk,
                                                                   FtImages P, double *__restrict__ partial)
{
    __shared__ FtSrcD tile[kFtTile];
    const int i = blockIdx.x * kFtThreads + threadIdx.x;
    const bool valid = i < n;
    const int j0 = blockIdx.y * chunk, j1 = min(n, j0 + chunk);
    FtSrcD me;
    if (valid) me = src[i];
    else { me.x = 0.0; me.y = 0.0; me.z = 1.0e6; }
    double u[3] = {0.0, 0.0, 0.0}, w[3] = {0.0, 0.0, 0.0};
    for (int t0 = j0; t0 < j1; t0 += kFtTile) {
        const int cnt = min(kFtTile, j1 - t0);
        __syncthreads();
        for (int k = threadIdx.x; k < cnt; k += kFtThreads) tile[k] = src[t0 + k];
        __syncthreads();
        for (int k = 0; k < cnt; ++k) {
            const FtSrcD s = tile[k];
            const int j = t0 + k;
            const double Rz = me.z + s.z;
            auto add = [&](double dx, double dy, double dz) {
                double cu[3] = {0.0, 0.0, 0.0}, cw[3] = {0.0, 0.0, 0.0};
                pair_contrib<RMW_UF, double>(dx, dy, dz, Rz, me.z, s.z, s.fx, s.fy, s.fz, cu[0], cu[1], cu[2]);
                pair_contrib<RMW_UT, double>(dx, dy, dz, Rz, me.z, s.z, s.tx, s.ty, s.tz, cu[0], cu[1], cu[2]);
                if (WITH_W) {
                    pair_contrib<RMW_WF, double>(dx, dy, dz, Rz, me.z, s.z, s.fx, s.fy, s.fz, cw[0], cw[1], cw[2]);
                    pair_contrib<RMW_WT, double>(dx, dy, dz, Rz, me.z, s.z, s.tx, s.ty, s.tz, cw[0], cw[1], cw[2]);
                }
                for (int c = 0; c < 3; ++c) {
                    u[c] += cu[c];
                    w[c] += cw[c];
                }
            };
            const double dx = me.x - s.x, dy = me.y - s.y, dz = me.z - s.z;
            if (!PER) {
                // the self pair is evaluated (coincident points, finite near-field
                // branch) and discarded, so the warp stays convergent
                double cu[3] = {0.0, 0.0, 0.0}, cw[3] = {0.0, 0.0, 0.0};
                pair_contrib<RMW_UF, double>(dx, dy, dz, Rz, me.z, s.z, s.fx, s.fy, s.fz, cu[0], cu[1], cu[2]);
                pair_contrib<RMW_UT, double>(dx, dy, dz, Rz, me.z, s.z, s.tx, s.ty, s.tz, cu[0], cu[1], cu[2]);
                if (WITH_W) {
                    pair_contrib<RMW_WF, double>(dx, dy, dz, Rz, me.z, s.z, s.fx, s.fy, s.fz, cw[0], cw[1], cw[2]);
                    pair_contrib<RMW_WT, double>(dx, dy, dz, Rz, me.z, s.z, s.tx, s.ty, s.tz, cw[0], cw[1], cw[2]);
                }
                if (j != i)
                    for (int c = 0; c < 3; ++c) {
                        u[c] += cu[c];
                        w[c] += cw[c];
                    }
            } else {
                for_images(dx, dy, dz, P.Lx, P.Ly, P.Lz, j == i, add);
            }
        }
    }
    if (valid) {
        double *o = partial + (size_t)blockIdx.y * 6 * n;
        for (int c = 0; c < 3; ++c) {
            o[3 * (size_t)i + c] = u[c];
            o[3 * (size_t)n + 3 * (size_t)i + c] = w[c];
        }
    }
}

// ---------------------------------------------------------------------------
// mixed: FP32 pairs from double-float position differences; the FP32 sum over
// each tile is folded into TwoSum-compensated accumulators
template <bool WITH_W, bool PER>
__global__ void __launch_bounds__(kFtThreads) ft_pair_mixed_kernel(const FtSrcF *__restrict__ src, int n, int chunk,
                                                                    FtImages P, double *__restrict__ partial)
{
    __shared__ FtSrcF tile[kFtTile];
    const int i = blockIdx.x * kFtThreads + threadIdx.x;
    const bool valid = i < n;
    const int j0 = blockIdx.y * chunk, j1 = min(n, j0 + chunk);
    float4 mh = make_float4(0.f, 0.f, 1.0e6f, 0.f), ml = make_float4(0.f, 0.f, 0.f, 0.f);
    if (valid) { mh = src[i].hi; ml = src[i].lo; }
    const float hi = mh.z + ml.z;
    const float Lx = (float)P.Lx, Ly = (float)P.Ly, Lz = (float)P.Lz;
    float sh_[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f}, sl_[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    for (int t0 = j0; t0 < j1; t0 += kFtTile) {
        const int cnt = min(kFtTile, j1 - t0);
        __syncthreads();
        for (int k = threadIdx.x; k < cnt; k += kFtThreads) tile[k] = src[t0 + k];
        __syncthreads();
        float acc[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        for (int k = 0; k < cnt; ++k) {
            const float4 sh = tile[k].hi, sl = tile[k].lo, sf = tile[k].f, st = tile[k].t;
            const int j = t0 + k;
            const float dx = (mh.x - sh.x) + (ml.x - sl.x);
            const float dy = (mh.y - sh.y) + (ml.y - sl.y);
            const float dz = (mh.z - sh.z) + (ml.z - sl.z);
            const float hj = sh.z + sl.z;
            const float Rz = hi + hj;
            auto add = [&](float ex, float ey, float ez, float *o) {
                pair_contrib<RMW_UF, float>(ex, ey, ez, Rz, hi, hj, sf.x, sf.y, sf.z, o[0], o[1], o[2]);
                pair_contrib<RMW_UT, float>(ex, ey, ez, Rz, hi, hj, st.x, st.y, st.z, o[0], o[1], o[2]);
                if (WITH_W) {
                    pair_contrib<RMW_WF, float>(ex, ey, ez, Rz, hi, hj, sf.x, sf.y, sf.z, o[3], o[4], o[5]);
                    pair_contrib<RMW_WT, float>(ex, ey, ez, Rz, hi, hj, st.x, st.y, st.z, o[3], o[4], o[5]);
                }
            };
            if (!PER) {
                float c[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
                add(dx, dy, dz, c);
                if (j != i)
                    for (int q = 0; q < 6; ++q) acc[q] += c[q];
            } else {
                for_images(dx, dy, dz, Lx, Ly, Lz, j == i, [&](float ex, float ey, float ez) { add(ex, ey, ez, acc); });
            }
        }
        for (int q = 0; q < 6; ++q) comp_add(sh_[q], sl_[q], acc[q]);
    }
    if (valid) {
        double *o = partial + (size_t)blockIdx.y * 6 * n;
        for (int c = 0; c < 3; ++c) {
            o[3 * (size_t)i + c] = (double)sh_[c] + (double)sl_[c];
            o[3 * (size_t)n + 3 * (size_t)i + c] = (double)sh_[3 + c] + (double)sl_[3 + c];
        }
    }
}

// ---------------------------------------------------------------------------
// df64: double-float pairs on the FP32 pipe; each group of kFtDfGroup sources
// is summed in double-float and folded into FP64 accumulators
template <bool WITH_W, bool PER>
__global__ void __launch_bounds__(kFtThreads) ft_pair_df_kernel(const FtSrcDF *__restrict__ src, int n, int chunk,
                                                                 FtImages P, double *__restrict__ partial)
{
    __shared__ FtSrcDF tile[kFtTile];
    const int i = blockIdx.x * kFtThreads + threadIdx.x;
    const bool valid = i < n;
    const int j0 = blockIdx.y * chunk, j1 = min(n, j0 + chunk);
    float4 mh = make_float4(0.f, 0.f, 1.0e6f, 0.f), ml = make_float4(0.f, 0.f, 0.f, 0.f);
    if (valid) { mh = src[i].hi; ml = src[i].lo; }
    const df xi = {mh.x, ml.x}, yi = {mh.y, ml.y}, zi = {mh.z, ml.z};
    double acc[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
    for (int t0 = j0; t0 < j1; t0 += kFtTile) {
        const int cnt = min(kFtTile, j1 - t0);
        __syncthreads();
        for (int k = threadIdx.x; k < cnt; k += kFtThreads) tile[k] = src[t0 + k];
        __syncthreads();
        for (int g0 = 0; g0 < cnt; g0 += kFtDfGroup) {
            const int g1 = min(cnt, g0 + kFtDfGroup);
            df gs[6] = {df_from(0.f), df_from(0.f), df_from(0.f), df_from(0.f), df_from(0.f), df_from(0.f)};
            for (int k = g0; k < g1; ++k) {
                const FtSrcDF s = tile[k];
                const int j = t0 + k;
                const df xj = {s.hi.x, s.lo.x}, yj = {s.hi.y, s.lo.y}, zj = {s.hi.z, s.lo.z};
                const df fx = {s.fhi.x, s.flo.x}, fy = {s.fhi.y, s.flo.y}, fz = {s.fhi.z, s.flo.z};
                const df tx = {s.thi.x, s.tlo.x}, ty = {s.thi.y, s.tlo.y}, tz = {s.thi.z, s.tlo.z};
                const df Rz = zi + zj;
                auto add = [&](df ex, df ey, df ez) {
                    df a0, a1, a2, b0, b1, b2;
                    pair_contrib_df<RMW_UF>(ex, ey, ez, Rz, zi, zj, fx, fy, fz, a0, a1, a2);
                    pair_contrib_df<RMW_UT>(ex, ey, ez, Rz, zi, zj, tx, ty, tz, b0, b1, b2);
                    acc_add(gs[0], a0 + b0);
                    acc_add(gs[1], a1 + b1);
                    acc_add(gs[2], a2 + b2);
                    if (WITH_W) {
                        pair_contrib_df<RMW_WF>(ex, ey, ez, Rz, zi, zj, fx, fy, fz, a0, a1, a2);
                        pair_contrib_df<RMW_WT>(ex, ey, ez, Rz, zi, zj, tx, ty, tz, b0, b1, b2);
                        acc_add(gs[3], a0 + b0);
                        acc_add(gs[4], a1 + b1);
                        acc_add(gs[5], a2 + b2);
                    }
                };
                if (!PER) {
                    if (j != i) {
                        add(xi - xj, yi - yj, zi - zj);
                    } else {
                        // evaluate and discard the self pair so the warp stays convergent
                        df g2[6];
                        for (int q = 0; q < 6; ++q) g2[q] = gs[q];
                        add(xi - xj, yi - yj, zi - zj);
                        for (int q = 0; q < 6; ++q) gs[q] = g2[q];
                    }
                } else {
                    // minimum image in FP64 (rare path), then back to double-float
                    for_images(to_double(xi - xj), to_double(yi - yj), to_double(zi - zj), P.Lx, P.Ly, P.Lz, j == i,
                               [&](double ex, double ey, double ez) {
                                   add(df_of_double(ex), df_of_double(ey), df_of_double(ez));
                               });
                }
            }
            for (int q = 0; q < 6; ++q) acc[q] += to_double(gs[q]);
        }
    }
    if (valid) {
        double *o = partial + (size_t)blockIdx.y * 6 * n;
        for (int c = 0; c < 3; ++c) {
            o[3 * (size_t)i + c] = acc[c];
            o[3 * (size_t)n + 3 * (size_t)i + c] = acc[3 + c];
        }
    }
}

// ---------------------------------------------------------------------------
// finalize: fixed-order slot sum, FP64 self terms of the four blocks
// (mobility/mobility_numba.py self terms), b_i and the scales.  A CTA takes
// kFtFinBlobs blobs; thread (x, g) sums slots g, g + G, ... of component x
// (coalesced), one thread per blob adds the G sums in order.  pair_scale: 2/3
// where the slots hold 3/2 of the sums.
constexpr int kFtFinBlobs = 32, kFtFinGroups = 8;
__global__ void __launch_bounds__(3 * kFtFinBlobs * kFtFinGroups)
    ft_finalize_kernel(const double *__restrict__ r, const double *__restrict__ F, const double *__restrict__ T,
                       const double *__restrict__ partial, int nchunks, double *__restrict__ U,
                       double *__restrict__ W, int n, double a, double nf, double pair_scale)
{
    __shared__ double red[kFtFinGroups][2][3 * kFtFinBlobs];
    const int x = threadIdx.x, g = threadIdx.y;
    const long long e = 3LL * blockIdx.x * kFtFinBlobs + x;
    if (e < 3LL * n) {
        double su = 0.0, sw = 0.0;
#pragma unroll 4
        for (int s = g; s < nchunks; s += kFtFinGroups) {
            const double *p = partial + (size_t)s * 6 * n + e;
            su += p[0];
            if (W) sw += p[3 * (size_t)n];
        }
        red[g][0][x] = su;
        red[g][1][x] = sw;
    }
    __syncthreads();
    const int i = blockIdx.x * kFtFinBlobs + x;
    if (g != 0 || x >= kFtFinBlobs || i >= n) return;
    double u[3] = {0.0, 0.0, 0.0}, w[3] = {0.0, 0.0, 0.0};
    for (int k = 0; k < kFtFinGroups; ++k)
        for (int c = 0; c < 3; ++c) {
            u[c] += red[k][0][3 * x + c];
            w[c] += red[k][1][3 * x + c];
        }
    for (int c = 0; c < 3; ++c) {
        u[c] *= pair_scale;
        w[c] *= pair_scale;
    }
    const double z = r[3 * i + 2];
    const double b = (z < a) ? z / a : 1.0;
    const double ze = (z <= a) ? a : z;
    const double fx = b * F[3 * i], fy = b * F[3 * i + 1], fz = b * F[3 * i + 2];
    const double tx = b * T[3 * i] / a, ty = b * T[3 * i + 1] / a, tz = b * T[3 * i + 2] / a;
    const double iz = a / ze, iz3 = iz * iz * iz, iz5 = iz3 * iz * iz;
    const double mxx = 4.0 / 3.0 - (9.0 * iz - 2.0 * iz3 + iz5) / 12.0;
    const double mzz = 4.0 / 3.0 - (9.0 * iz - 4.0 * iz3 + iz5) / 6.0;
    const double sr = 0.125 * iz3 * iz;  // rotation-translation coupling 1/(8 h^4)
    u[0] += mxx * fx + sr * ty;
    u[1] += mxx * fy - sr * tx;
    u[2] += mzz * fz;
    U[3 * i] = b * nf * u[0];
    U[3 * i + 1] = b * nf * u[1];
    U[3 * i + 2] = b * nf * u[2];
    if (W) {
        w[0] += -sr * fy + (1.0 - 0.3125 * iz3) * tx;
        w[1] += sr * fx + (1.0 - 0.3125 * iz3) * ty;
        w[2] += (1.0 - 0.125 * iz3) * tz;
        const double sw = b * nf / a;
        W[3 * i] = sw * w[0];
        W[3 * i + 1] = sw * w[1];
        W[3 * i + 2] = sw * w[2];
    }
}

// ---------------------------------------------------------------------------
// Symmetric mixed-precision force-torque kernel: the grid and pairing of the
// symmetric single products (one CTA per tile pair T <= S of the upper
// triangle; lane l meets source (l + k) mod 128 at step k; per-warp source
// sums in shared memory), all four blocks per unordered pair, applied to both
// blobs: u_i += UF_ij f_j + UT_ij t_j, w_i += WF_ij f_j + WT_ij t_j and the
// same with i and j exchanged (M_ji = M_ij^T: UF through its transposed
// coefficients, the rotation blocks through pair_rot_sym).  The UF
// coefficients come times 3/2 and are scaled back per pair, so U and W keep
// the one-sided kernels' sums and finalize.  Partial slots: blob b of tile X
// gets one slot per tile, U at slot * 6n + 3b and W at slot * 6n + 3n + 3b.
constexpr int kFtSymWarps = 4;
constexpr int kFtSymTile = 32 * kFtSymWarps;

template <bool WITH_W>
__global__ void __launch_bounds__(kFtSymTile) ft_sym_mixed_kernel(const FtSrcF *__restrict__ src, int n, int nt,
                                                                  double *__restrict__ partial)
{
    __shared__ float4 thi[kFtSymTile], tlo[kFtSymTile], tf[kFtSymTile], tt[kFtSymTile];
    __shared__ float sacc[kFtSymWarps][6][kFtSymTile];
    int T, S;
    sym_tile_pair(blockIdx.x, nt, T, S);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const bool diag = (T == S);
    const int i = T * kFtSymTile + tid;
    const bool valid_i = i < n;
    // a target or source past the end is a dummy with zero vectors half a radius above the wall, where no blob is
    const FtSrcF dummy = {make_float4(0.f, 0.f, 0.5f, 0.f), make_float4(0.f, 0.f, 0.f, 0.f),
                          make_float4(0.f, 0.f, 0.f, 0.f), make_float4(0.f, 0.f, 0.f, 0.f)};
    const FtSrcF me = valid_i ? src[i] : dummy;
    const float hi = me.hi.z + me.lo.z;
    {
        const int j = S * kFtSymTile + tid;
        const FtSrcF sj = (j < n) ? src[j] : dummy;
        thi[tid] = sj.hi;
        tlo[tid] = sj.lo;
        tf[tid] = sj.f;
        tt[tid] = sj.t;
    }
    for (int c = 0; c < 6; ++c)
        for (int k = lane; k < kFtSymTile; k += 32) sacc[warp][c][k] = 0.f;
    __syncthreads();
    float u0 = 0.f, u1 = 0.f, u2 = 0.f, w0 = 0.f, w1 = 0.f, w2 = 0.f;
    constexpr float kThird2 = 2.0f / 3.0f;  // undoes the UF coefficients' 3/2
    auto step = [&](int k) {
        const int jl = (lane + k) & (kFtSymTile - 1);
        const float4 sh = thi[jl], sl = tlo[jl], sf = tf[jl], st = tt[jl];
        const float dx = (me.hi.x - sh.x) + (me.lo.x - sl.x);
        const float dy = (me.hi.y - sh.y) + (me.lo.y - sl.y);
        const float dz = (me.hi.z - sh.z) + (me.lo.z - sl.z);
        const float hj = sh.z + sl.z;
        const float Rz = hi + hj;
        float a0 = sacc[warp][0][jl], a1 = sacc[warp][1][jl], a2 = sacc[warp][2][jl];
        UFCoeffs c = uf_coeffs(dx, dy, dz, Rz, hi, hj);
        c.Af *= kThird2; c.Bc *= kThird2; c.c2 *= kThird2; c.c3 *= kThird2; c.c4 *= kThird2; c.Af5 *= kThird2;
        uf_apply(c, dx, dy, dz, Rz, sf.x, sf.y, sf.z, u0, u1, u2);
        const UFCoeffs ct = {c.Af, c.Bc, c.c2, c.c4, c.c3, c.Af5};  // M^T: f3 and f4 trade places
        uf_apply(ct, dx, dy, dz, Rz, me.f.x, me.f.y, me.f.z, a0, a1, a2);
        pair_rot_sym<float, RMW_UT>(dx, dy, dz, Rz, hi, hj, st.x, st.y, st.z, me.t.x, me.t.y, me.t.z, u0, u1, u2, a0,
                                    a1, a2);
        sacc[warp][0][jl] = a0;
        sacc[warp][1][jl] = a1;
        sacc[warp][2][jl] = a2;
        if (WITH_W) {
            float b0 = sacc[warp][3][jl], b1 = sacc[warp][4][jl], b2 = sacc[warp][5][jl];
            pair_rot_sym<float, RMW_WF>(dx, dy, dz, Rz, hi, hj, sf.x, sf.y, sf.z, me.f.x, me.f.y, me.f.z, w0, w1, w2,
                                        b0, b1, b2);
            pair_rot_sym<float, RMW_WT>(dx, dy, dz, Rz, hi, hj, st.x, st.y, st.z, me.t.x, me.t.y, me.t.z, w0, w1, w2,
                                        b0, b1, b2);
            sacc[warp][3][jl] = b0;
            sacc[warp][4][jl] = b1;
            sacc[warp][5][jl] = b2;
        }
    };
    if (diag) {
        for (int k = 0; k < kFtSymTile; ++k) {
            __syncwarp();
            const int off = (k - 32 * warp) & (kFtSymTile - 1);  // (source - target) mod 128, warp-uniform
            if (off == 0 || off > kFtSymTile / 2 || (off == kFtSymTile / 2 && warp >= kFtSymWarps / 2)) continue;
            step(k);
        }
    } else {
        for (int k = 0; k < kFtSymTile; ++k) {
            __syncwarp();
            step(k);
        }
    }
    __syncthreads();
    double q[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
    for (int w = 0; w < kFtSymWarps; ++w)
        for (int c = 0; c < (WITH_W ? 6 : 3); ++c) q[c] += (double)sacc[w][c][tid];
    const double tu[6] = {u0, u1, u2, w0, w1, w2};
    const size_t stride = 6 * (size_t)n;
    if (diag) {
        if (valid_i) {
            double *o = partial + (size_t)T * stride;
            for (int c = 0; c < 3; ++c) {
                o[3 * (size_t)i + c] = tu[c] + q[c];
                o[3 * (size_t)n + 3 * (size_t)i + c] = tu[3 + c] + q[3 + c];
            }
        }
    } else {
        if (valid_i) {
            double *o = partial + (size_t)S * stride;
            for (int c = 0; c < 3; ++c) {
                o[3 * (size_t)i + c] = tu[c];
                o[3 * (size_t)n + 3 * (size_t)i + c] = tu[3 + c];
            }
        }
        const int j = S * kFtSymTile + tid;
        if (j < n) {
            double *o = partial + (size_t)T * stride;
            for (int c = 0; c < 3; ++c) {
                o[3 * (size_t)j + c] = q[c];
                o[3 * (size_t)n + 3 * (size_t)j + c] = q[3 + c];
            }
        }
    }
}

void ft_finalize(const double *r, const double *F, const double *T, const double *partial, int slots, double *U,
                 double *W, int n, double eta, double a, double pair_scale, cudaStream_t st)
{
    ft_finalize_kernel<<<(n + kFtFinBlobs - 1) / kFtFinBlobs, dim3(3 * kFtFinBlobs, kFtFinGroups), 0, st>>>(
        r, F, T, partial, slots, U, W, n, a, 1.0 / (8.0 * kPi * eta * a), pair_scale);
}

// ---------------------------------------------------------------------------
// Symmetric FP64 and df64 force-torque kernels: the grid, pairing and split
// (gridDim.y CTAs share a tile pair's steps) of the symmetric single products,
// the four blocks of an unordered pair from one set of distances, reciprocal
// roots and powers (about 150 of 600 + 500 + 500 + 500 FP32-pipe operations
// in df64, 25 of 73 + 64 + 64 + 62 operations in FP64), applied both ways;
// every block times 3/2, undone by the finalize.  The sum of four symmetric
// single products, which this replaces, read the blobs and formed the geometry
// four times and needed a vector of scratch and two additions.  8,064 blobs,
// [U; W]: df64 2.20 -> 1.55 ms (3.51 before the blocks were written out), four
// CTAs of 255 registers per SM (six of 168 spill: 1.58 ms); FP64
// 23.0 -> 6.92 ms (10.6 with every operation on the FP64 pipe).
struct FtSteps {
    int k0, k1, nsplit, split;
    __device__ __forceinline__ size_t slot(int tile) const { return (size_t)tile * nsplit + split; }
};
__device__ __forceinline__ FtSteps ft_steps()
{
    const int m = gridDim.y, s = blockIdx.y;
    return {kFtSymTile * s / m, kFtSymTile * (s + 1) / m, m, s};
}

template <bool WITH_W>
__global__ void __launch_bounds__(kFtSymTile) ft_sym_fp64_kernel(const FtSrcD *__restrict__ src, int n, int nt,
                                                                 double *__restrict__ partial)
{
    constexpr int NC = WITH_W ? 6 : 3;
    __shared__ double sx[9][kFtSymTile];  // x y z f t
    __shared__ double sacc[kFtSymWarps][NC][kFtSymTile];
    int T, S;
    sym_tile_pair(blockIdx.x, nt, T, S);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const bool diag = (T == S);
    const int i = T * kFtSymTile + tid;
    const bool valid_i = i < n;
    // a target or source past the end is a dummy with zero vectors half a radius above the wall, where no blob is
    // (heights are at least 1; a dummy on a blob's place would make its products NaN)
    const FtSrcD dummy = {0.0, 0.0, 0.5, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
    const FtSrcD me = valid_i ? src[i] : dummy;
    bool in_range = int_range_blob(me.x, me.y, me.z, me.fx, me.fy, me.fz) && int_range_vec<150>(me.tx, me.ty, me.tz);
    {
        const int j = S * kFtSymTile + tid;
        const FtSrcD q = (j < n) ? src[j] : dummy;
        const double c[9] = {q.x, q.y, q.z, q.fx, q.fy, q.fz, q.tx, q.ty, q.tz};
        for (int k = 0; k < 9; ++k) sx[k][tid] = c[k];
        in_range = in_range && int_range_blob(q.x, q.y, q.z, q.fx, q.fy, q.fz) &&
                   int_range_vec<150>(q.tx, q.ty, q.tz);
    }
    for (int c = 0; c < NC; ++c)
        for (int k = lane; k < kFtSymTile; k += 32) sacc[warp][c][k] = 0.0;
    const bool allow = __syncthreads_and(in_range);  // the integer forms, for every blob of the tile pair
    double u[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
    auto step = [&](int k) {
        const int j = (lane + k) & (kFtSymTile - 1);
        const double zj = sx[2][j], dx = me.x - sx[0][j], dy = me.y - sx[1][j], dz = me.z - zj, Rz = me.z + zj;
        const double fx = sx[3][j], fy = sx[4][j], fz = sx[5][j], tx = sx[6][j], ty = sx[7][j], tz = sx[8][j];
        double w[NC];
        for (int c = 0; c < NC; ++c) w[c] = sacc[warp][c][j];
        with_pair_geo_d<false, false>(dx, dy, dz, 1.0, Rz, me.z, zj, allow,
                                      [&](const PairGeoD &g, double, double, double, auto mul) {
            using MUL = decltype(mul);
            {
                const UFBlockD m = uf_block_d<false, MUL>(g, dz, Rz, me.z, zj);
                uf_block_acc_d<MUL>(m, m.t3, m.t4, dx, dy, fx, fy, fz, u[0], u[1], u[2]);
                uf_block_acc_d<MUL>(m, m.t4, m.t3, dx, dy, me.fx, me.fy, me.fz, w[0], w[1], w[2]);
            }
            const RotBlockD k2 = rot_block_d<true, MUL>(g, dz, Rz, me.z, zj);
            ut_acc_d<MUL>(k2, dx, dy, tx, ty, tz, me.tx, me.ty, me.tz, u[0], u[1], u[2], w[0], w[1], w[2]);
            if constexpr (WITH_W) {
                wf_acc_d<MUL>(k2, dx, dy, fx, fy, fz, me.fx, me.fy, me.fz, u[3], u[4], u[5], w[3], w[4], w[5]);
                const UFBlockD m = wt_block_d<true, MUL>(g, dz, Rz);
                uf_block_acc_d<MUL>(m, m.t3, m.t4, dx, dy, tx, ty, tz, u[3], u[4], u[5]);
                uf_block_acc_d<MUL>(m, m.t4, m.t3, dx, dy, me.tx, me.ty, me.tz, w[3], w[4], w[5]);
            }
        });
        for (int c = 0; c < NC; ++c) sacc[warp][c][j] = w[c];
    };
    const FtSteps sp = ft_steps();
    for (int k = sp.k0; k < sp.k1; ++k) {
        __syncwarp();
        const int off = (k - 32 * warp) & (kFtSymTile - 1);  // (source - target) mod 128, warp-uniform
        if (diag && (off == 0 || off > kFtSymTile / 2 || (off == kFtSymTile / 2 && warp >= kFtSymWarps / 2))) continue;
        step(k);
    }
    __syncthreads();
    const int j = S * kFtSymTile + tid;
    for (int c = 0; c < NC; ++c) {
        double q = 0.0;
        for (int w = 0; w < kFtSymWarps; ++w) q += sacc[w][c][tid];
        const size_t comp = (c / 3) * 3 * (size_t)n + c % 3;
        if (valid_i) partial[sp.slot(diag ? T : S) * 6 * n + 3 * (size_t)i + comp] = diag ? u[c] + q : u[c];
        if (!diag && j < n) partial[sp.slot(T) * 6 * n + 3 * (size_t)j + comp] = q;
    }
}

// df64: two targets per thread in packed lanes, as wall_uf_df_sym_kernel.  An
// accumulator takes the terms of two blocks a step, so both sides' sums are
// renormalised every four steps: error at 8,064 blobs 9.46e-14, that of four
// single products 9.50e-14 (9.57e-14 with the targets' every eight, 0.5 % faster).
constexpr int kFtF2Threads = kFtSymTile / 2;

struct FtTarget {
    df2 x, y, z, h4, f[3], t[3];
};

template <bool DIAG, bool WITH_W>
__device__ __forceinline__ void ft_f2_step(const FtTarget &me, int ja, int jb, const float4 (*tile)[kFtSymTile],
                                           float4 (*sacc)[kFtSymTile], df2 (&u)[6], bool renorm)
{
    constexpr int NC = WITH_W ? 6 : 3;
    df2 v[3][3];  // position, F, T of the sources
#pragma unroll
    for (int q = 0; q < 3; ++q) {
        const float4 h = tile[2 * q][ja], l = tile[2 * q + 1][ja];
        float4 h1 = h, l1 = l;
        if (DIAG) {
            h1 = tile[2 * q][jb];
            l1 = tile[2 * q + 1][jb];
        }
        v[q][0] = {make_float2(h.x, h1.x), make_float2(l.x, l1.x)};
        v[q][1] = {make_float2(h.y, h1.y), make_float2(l.y, l1.y)};
        v[q][2] = {make_float2(h.z, h1.z), make_float2(l.z, l1.z)};
    }
    const df2 dx = me.x - v[0][0], dy = me.y - v[0][1], dz = me.z - v[0][2], zj = v[0][2], Rz = add_u(me.z, zj);
    const PairGeoDF<df2> g = pair_geo_df<df2>(dx, dy, dz, Rz, me.h4, zj);
    auto load = [&](int c) -> df2 {
        const float4 a = sacc[c][ja];
        if (!DIAG) return {make_float2(a.x, a.y), make_float2(a.z, a.w)};
        const float4 b = sacc[c][jb];
        return {make_float2(a.x, b.y), make_float2(a.z, b.w)};
    };
    auto store = [&](int c, const df2 &w) {
        if (!DIAG) {
            sacc[c][ja] = make_float4(w.hi.x, w.hi.y, w.lo.x, w.lo.y);
        } else {
            float *a = (float *)&sacc[c][ja], *b = (float *)&sacc[c][jb];
            a[0] = w.hi.x; a[2] = w.lo.x;
            b[1] = w.hi.y; b[3] = w.lo.y;
        }
    };
    df2 wx = load(0), wy = load(1), wz = load(2);
    {
        const UFBlockDF<df2> m = uf_block_df<df2>(g, dz, Rz, me.h4, zj);
        uf_block_acc_df(m, m.t3, m.t4, dx, dy, v[1][0], v[1][1], v[1][2], u[0], u[1], u[2]);
        uf_block_acc_df(m, m.t4, m.t3, dx, dy, me.f[0], me.f[1], me.f[2], wx, wy, wz);
    }
    const RotBlockDF2 k = rot_block_df<true>(g, dz, Rz, me.z, zj);
    ut_acc_df(k, dx, dy, v[2][0], v[2][1], v[2][2], me.t[0], me.t[1], me.t[2], u[0], u[1], u[2], wx, wy, wz);
    if (renorm) { wx = norm(wx); wy = norm(wy); wz = norm(wz); }
    store(0, wx); store(1, wy); store(2, wz);
    if constexpr (WITH_W) {
        wx = load(NC - 3); wy = load(NC - 2); wz = load(NC - 1);
        wf_acc_df(k, dx, dy, v[1][0], v[1][1], v[1][2], me.f[0], me.f[1], me.f[2], u[3], u[4], u[5], wx, wy, wz);
        const UFBlockDF<df2> m = wt_block_df<true>(g, dz, Rz);
        uf_block_acc_df(m, m.t3, m.t4, dx, dy, v[2][0], v[2][1], v[2][2], u[3], u[4], u[5]);
        uf_block_acc_df(m, m.t4, m.t3, dx, dy, me.t[0], me.t[1], me.t[2], wx, wy, wz);
        if (renorm) { wx = norm(wx); wy = norm(wy); wz = norm(wz); }
        store(NC - 3, wx); store(NC - 2, wy); store(NC - 1, wz);
    }
}

template <bool WITH_W>
__global__ void __launch_bounds__(kFtF2Threads, 4) ft_sym_df_kernel(const FtSrcDF *__restrict__ src, int n, int nt,
                                                                    double *__restrict__ partial)
{
    constexpr int NC = WITH_W ? 6 : 3;
    __shared__ float4 tile[6][kFtSymTile];  // hi, lo, fhi, flo, thi, tlo
    __shared__ float4 sacc[kFtF2Threads / 32][NC][kFtSymTile];
    __shared__ double tacc[2][NC][kFtF2Threads];  // the targets' FP64 sums
    int T, S;
    sym_tile_pair(blockIdx.x, nt, T, S);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const bool diag = (T == S);
    const int i0 = T * kFtSymTile + tid, i1 = i0 + kFtF2Threads;
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    const FtSrcDF dummy = {make_float4(0.f, 0.f, 0.5f, 0.f), zero, zero, zero, zero, zero};
    FtTarget me;
    {
        const FtSrcDF a = i0 < n ? src[i0] : dummy, b = i1 < n ? src[i1] : dummy;
        me.x = df2_pack({a.hi.x, a.lo.x}, {b.hi.x, b.lo.x});
        me.y = df2_pack({a.hi.y, a.lo.y}, {b.hi.y, b.lo.y});
        me.z = df2_pack({a.hi.z, a.lo.z}, {b.hi.z, b.lo.z});
        me.h4 = scale2(me.z, 4.0f);
        me.f[0] = df2_pack({a.fhi.x, a.flo.x}, {b.fhi.x, b.flo.x});
        me.f[1] = df2_pack({a.fhi.y, a.flo.y}, {b.fhi.y, b.flo.y});
        me.f[2] = df2_pack({a.fhi.z, a.flo.z}, {b.fhi.z, b.flo.z});
        me.t[0] = df2_pack({a.thi.x, a.tlo.x}, {b.thi.x, b.tlo.x});
        me.t[1] = df2_pack({a.thi.y, a.tlo.y}, {b.thi.y, b.tlo.y});
        me.t[2] = df2_pack({a.thi.z, a.tlo.z}, {b.thi.z, b.tlo.z});
    }
    for (int k = tid; k < kFtSymTile; k += kFtF2Threads) {
        const int j = S * kFtSymTile + k;
        const FtSrcDF q = (j < n) ? src[j] : dummy;
        tile[0][k] = q.hi; tile[1][k] = q.lo;
        tile[2][k] = q.fhi; tile[3][k] = q.flo;
        tile[4][k] = q.thi; tile[5][k] = q.tlo;
    }
    for (int c = 0; c < NC; ++c)
        for (int k = lane; k < kFtSymTile; k += 32) sacc[warp][c][k] = zero;
    for (int c = 0; c < NC; ++c) tacc[0][c][tid] = tacc[1][c][tid] = 0.0;
    __syncthreads();
    df2 u[6];
    for (int c = 0; c < 6; ++c) u[c] = df2_zero();
    const FtSteps sp = ft_steps();
    auto renorm = [&](int k) {
        if (k & 3) return;
        for (int c = 0; c < NC; ++c) u[c] = norm(u[c]);
    };
    auto fold = [&]() {
        for (int c = 0; c < NC; ++c) {
            tacc[0][c][tid] += to_double(df{u[c].hi.x, u[c].lo.x});
            tacc[1][c][tid] += to_double(df{u[c].hi.y, u[c].lo.y});
            u[c] = df2_zero();
        }
    };
    if (diag) {
        // offsets (source - target) 1..63, and 64 for lane x alone (lane y's pairs are lane x's)
        for (int o = 1 + sp.k0 / 2; o < 1 + sp.k1 / 2; ++o) {
            __syncwarp();
            const int ja = (tid + o) & (kFtSymTile - 1), jb = (tid + kFtF2Threads + o) & (kFtSymTile - 1);
            if (o < kFtSymTile / 2) {
                ft_f2_step<true, WITH_W>(me, ja, jb, tile, sacc[warp], u, !(o & 3));
            } else {
                FtTarget half = me;
                for (int c = 0; c < 3; ++c)
                    half.f[c].hi.y = half.f[c].lo.y = half.t[c].hi.y = half.t[c].lo.y = 0.f;
                df2 v[6];
                for (int c = 0; c < 6; ++c) v[c] = u[c];
                ft_f2_step<true, WITH_W>(half, ja, jb, tile, sacc[warp], v, true);
                for (int c = 0; c < NC; ++c) {
                    u[c].hi.x = v[c].hi.x;
                    u[c].lo.x = v[c].lo.x;
                }
            }
            renorm(o);
            if (!(o & (kFtDfGroup - 1))) fold();
        }
    } else {
#pragma unroll 1
        for (int k = sp.k0; k < sp.k1; ++k) {
            __syncwarp();
            const int j = (lane + k) & (kFtSymTile - 1);
            ft_f2_step<false, WITH_W>(me, j, j, tile, sacc[warp], u, !((k + 1) & 3));
            renorm(k + 1);
            if (!((k + 1) & (kFtDfGroup - 1))) fold();
        }
    }
    fold();
    __syncthreads();
    for (int half = 0; half < 2; ++half) {
        const int l = tid + half * kFtF2Threads, i = T * kFtSymTile + l, j = S * kFtSymTile + l;
        for (int c = 0; c < NC; ++c) {
            const double t = tacc[half][c][tid];
            static_assert(kFtF2Threads == 64, "two warps' sums, two lanes each");
            const float4 f = sacc[0][c][l], g = sacc[1][c][l];
            const double q = sum4_to_double({f.x, f.z}, {f.y, f.w}, {g.x, g.z}, {g.y, g.w});
            const size_t comp = (c / 3) * 3 * (size_t)n + c % 3;
            if (i < n) partial[sp.slot(diag ? T : S) * 6 * n + 3 * (size_t)i + comp] = diag ? t + q : t;
            if (!diag && j < n) partial[sp.slot(T) * 6 * n + 3 * (size_t)j + comp] = q;
        }
    }
}

__global__ void ft_add_kernel(const double *__restrict__ x, double *__restrict__ y, long long m)
{
    const long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (k < m) y[k] += x[k];
}

// U (and W) as sums of single products, each through the symmetric kernel
// (every unordered pair once per block): faster than the fused one-sided pass
// (10,752 blobs df64 3.7 against 7.6 ms), with half the partial sums of the
// fused symmetric kernel.
int ft_by_symmetric_products(const double *r, const double *F, const double *T, double *U, double *W, int n,
                             double eta, double a, int mode, cudaStream_t st)
{
    void *tmp = nullptr;
    if (int rc = scratch(SCRATCH_FT_TERM, sizeof(double) * 3 * (size_t)n, &tmp, st)) return rc;
    double *t = (double *)tmp;
    const unsigned g = (unsigned)((3LL * n + 255) / 256);
    if (int rc = wall_product(RMW_UF, r, F, U, n, eta, a, nullptr, mode, st)) return rc;
    if (int rc = wall_product(RMW_UT, r, T, t, n, eta, a, nullptr, mode, st)) return rc;
    ft_add_kernel<<<g, 256, 0, st>>>(t, U, 3LL * n);
    if (W) {
        if (int rc = wall_product(RMW_WF, r, F, W, n, eta, a, nullptr, mode, st)) return rc;
        if (int rc = wall_product(RMW_WT, r, T, t, n, eta, a, nullptr, mode, st)) return rc;
        ft_add_kernel<<<g, 256, 0, st>>>(t, W, 3LL * n);
    }
    RMW_CHECK_LAUNCH("force-torque through symmetric products");
    return RMW_OK;
}

// FP64 and df64, not periodic: the fused symmetric product.  RMW_ERR_ALLOC:
// its partial sums do not fit (the caller takes the one-sided pass).
int ft_symmetric(const double *r, const double *F, const double *T, double *U, double *W, int n, double eta, double a,
                 int mode, cudaStream_t st)
{
    const int nt = (n + kFtSymTile - 1) / kFtSymTile;
    const size_t rec = mode == RMW_MODE_DF64 ? sizeof(FtSrcDF) : sizeof(FtSrcD);
    const size_t packed = ((rec * (size_t)n + 255) / 256) * 256, slot = sizeof(double) * 6 * (size_t)n * nt;
    int nsplit = wall_sym_split(mode, n, packed, false, 6);
    void *ws = nullptr;
    if (slot > wall_sym_partial_budget()) return RMW_ERR_ALLOC;
    int rc = scratch(SCRATCH_PAIR, packed + slot * nsplit, &ws, st, wall_reserve_bytes(mode, n, packed, true, 6));
    if (rc && nsplit > 1) {  // memory pressure: whole tile pairs need the least
        cudaGetLastError();
        nsplit = 1;
        rc = scratch(SCRATCH_PAIR, packed + slot, &ws, st);
    }
    if (rc) {
        cudaGetLastError();
        return RMW_ERR_ALLOC;
    }
    double *partial = (double *)((char *)ws + packed);
    const int pb = 64, pg = (n + pb - 1) / pb;
    if (mode == RMW_MODE_FP64) ft_pack_fp64_kernel<<<pg, pb, 0, st>>>(r, F, T, (FtSrcD *)ws, n, a);
    else ft_pack_df_kernel<<<pg, pb, 0, st>>>(r, F, T, (FtSrcDF *)ws, n, a);
    const dim3 grid((unsigned)((long long)nt * (nt + 1) / 2), nsplit);
    void *tok = nullptr;
    if (int rc = trace_begin(TRACE_PAIR, st, &tok)) return rc;
    if (mode == RMW_MODE_FP64) {
        if (W) ft_sym_fp64_kernel<true><<<grid, kFtSymTile, 0, st>>>((const FtSrcD *)ws, n, nt, partial);
        else ft_sym_fp64_kernel<false><<<grid, kFtSymTile, 0, st>>>((const FtSrcD *)ws, n, nt, partial);
    } else {
        if (W) ft_sym_df_kernel<true><<<grid, kFtF2Threads, 0, st>>>((const FtSrcDF *)ws, n, nt, partial);
        else ft_sym_df_kernel<false><<<grid, kFtF2Threads, 0, st>>>((const FtSrcDF *)ws, n, nt, partial);
    }
    if (int rc = trace_end(tok, st)) return rc;
    ft_finalize(r, F, T, partial, nt * nsplit, U, W, n, eta, a, kUFCoeffScale, st);
    RMW_CHECK_LAUNCH("symmetric force-torque wall product");
    return RMW_OK;
}

}  // namespace

size_t wall_ft_scratch_bytes(int n, int mode, int nchunks)
{
    const size_t rec = (mode == RMW_MODE_MIXED) ? sizeof(FtSrcF) : (mode == RMW_MODE_DF64 ? sizeof(FtSrcDF)
                                                                                          : sizeof(FtSrcD));
    const size_t packed = ((rec * (size_t)n + 255) / 256) * 256;
    return packed + sizeof(double) * 6 * (size_t)n * (size_t)nchunks;
}

template <bool WITH_W, bool PER>
static void ft_launch(int mode, dim3 grid, cudaStream_t st, void *src, int n, int chunk, FtImages P,
                      double *partial)
{
    if (mode == RMW_MODE_FP64)
        ft_pair_fp64_kernel<WITH_W, PER><<<grid, kFtThreads, 0, st>>>((const FtSrcD *)src, n, chunk, P, partial);
    else if (mode == RMW_MODE_DF64)
        ft_pair_df_kernel<WITH_W, PER><<<grid, kFtThreads, 0, st>>>((const FtSrcDF *)src, n, chunk, P, partial);
    else
        ft_pair_mixed_kernel<WITH_W, PER><<<grid, kFtThreads, 0, st>>>((const FtSrcF *)src, n, chunk, P, partial);
}

int wall_force_torque(const double *r, const double *F, const double *T, double *U, double *W, int64_t n,
                      double eta, double a, const double *L, int mode, cudaStream_t st)
{
    if (int rc = validate_product_args(RMW_UF, r, F, U, n, eta, a, mode)) return rc;
    if (n > 0 && !T) return fail(RMW_ERR_ARG, "null torque array");
    if (n == 0) return RMW_OK;
    const int N = (int)n;
    const bool per = L && (L[0] > 0 || L[1] > 0 || L[2] > 0);
    // mixed: the symmetric fused kernel from 8,192 blobs
    if (!per && mode == RMW_MODE_MIXED && N >= 8192) {
        const int nt = (N + kFtSymTile - 1) / kFtSymTile;
        const size_t packed = ((sizeof(FtSrcF) * (size_t)N + 255) / 256) * 256;
        const size_t part = sizeof(double) * 6 * (size_t)N * (size_t)nt;
        void *ws = nullptr;
        // the partial sums may not fit next to the caller's allocations (or
        // above rmw_set_scratch_limit): then the one-sided pass below, whose
        // scratch is far smaller, does the product
        if (part <= wall_sym_partial_budget() && scratch(SCRATCH_PAIR, packed + part, &ws, st) != RMW_OK) {
            cudaGetLastError();
            ws = nullptr;
        }
        if (ws) {
            double *partial = (double *)((char *)ws + packed);
            const int pb = 256, pg = (N + pb - 1) / pb;
            ft_pack_mixed_kernel<<<pg, pb, 0, st>>>(r, F, T, (FtSrcF *)ws, N, a);
            const unsigned ncta = (unsigned)((long long)nt * (nt + 1) / 2);
            void *tok = nullptr;
            if (int rc = trace_begin(TRACE_PAIR, st, &tok)) return rc;
            if (W) ft_sym_mixed_kernel<true><<<ncta, kFtSymTile, 0, st>>>((const FtSrcF *)ws, N, nt, partial);
            else ft_sym_mixed_kernel<false><<<ncta, kFtSymTile, 0, st>>>((const FtSrcF *)ws, N, nt, partial);
            if (int rc = trace_end(tok, st)) return rc;
            ft_finalize(r, F, T, partial, nt, U, W, N, eta, a, 1.0, st);
            RMW_CHECK_LAUNCH("symmetric force-torque wall product");
            return RMW_OK;
        }
    }
    // FP64 and df64 where all four products prefer the symmetric kernel (untuned: from 256 blobs; a tuned or pinned
    // source split keeps the one-sided pass and its small scratch): the fused symmetric kernel, where its partial sums
    // fit; where they do not, four symmetric single products, whose sums are half as large; else the one-sided pass
    if (!per && (mode == RMW_MODE_FP64 || mode == RMW_MODE_DF64) && N >= 2 * kFtSymTile) {
        bool prefer = true, applies = true;
        for (int kind : {RMW_UF, RMW_UT, RMW_WF, RMW_WT}) {
            prefer = prefer && wall_prefers_sym(kind, mode, N);
            applies = applies && wall_sym_applicable(kind, mode, N, nullptr);
        }
        if (prefer) {
            const int rc = ft_symmetric(r, F, T, U, W, N, eta, a, mode, st);
            if (rc != RMW_ERR_ALLOC) return rc;
            if (applies) return ft_by_symmetric_products(r, F, T, U, W, N, eta, a, mode, st);
        }
    }
    const int nchunks = wall_default_chunks(N);
    void *ws = nullptr;
    if (int rc = scratch(SCRATCH_PAIR, wall_ft_scratch_bytes(N, mode, nchunks), &ws, st)) return rc;
    const size_t rec = (mode == RMW_MODE_MIXED) ? sizeof(FtSrcF) : (mode == RMW_MODE_DF64 ? sizeof(FtSrcDF)
                                                                                          : sizeof(FtSrcD));
    const size_t packed = ((rec * (size_t)N + 255) / 256) * 256;
    double *partial = (double *)((char *)ws + packed);
    const int pb = 256, pg = (N + pb - 1) / pb;
    if (mode == RMW_MODE_FP64) ft_pack_fp64_kernel<<<pg, pb, 0, st>>>(r, F, T, (FtSrcD *)ws, N, a);
    else if (mode == RMW_MODE_DF64) ft_pack_df_kernel<<<pg, pb, 0, st>>>(r, F, T, (FtSrcDF *)ws, N, a);
    else ft_pack_mixed_kernel<<<pg, pb, 0, st>>>(r, F, T, (FtSrcF *)ws, N, a);
    const FtImages P{L ? L[0] / a : 0.0, L ? L[1] / a : 0.0, L ? L[2] / a : 0.0};
    const int chunk = (N + nchunks - 1) / nchunks;
    const dim3 grid((N + kFtThreads - 1) / kFtThreads, nchunks);
    void *tok = nullptr;
    if (int rc = trace_begin(TRACE_PAIR, st, &tok)) return rc;
    if (W) {
        if (per) ft_launch<true, true>(mode, grid, st, ws, N, chunk, P, partial);
        else ft_launch<true, false>(mode, grid, st, ws, N, chunk, P, partial);
    } else {
        if (per) ft_launch<false, true>(mode, grid, st, ws, N, chunk, P, partial);
        else ft_launch<false, false>(mode, grid, st, ws, N, chunk, P, partial);
    }
    if (int rc = trace_end(tok, st)) return rc;
    ft_finalize(r, F, T, partial, nchunks, U, W, N, eta, a, 1.0, st);
    RMW_CHECK_LAUNCH("force-torque wall product");
    return RMW_OK;
}

}  // namespace rmw

extern "C" {

// U = M_UF F + M_UT T and, if W is not NULL, W = M_WF F + M_WT T, in one pass
// over the pairs (device arrays of 3n doubles; see rmw_gb300.h).
int rmw_wall_force_torque(const double *r, const double *F, const double *T, double *U, double *W, int64_t n,
                          double eta, double a, const double *L_host, int mode, void *stream)
{
    return rmw::wall_force_torque(r, F, T, U, W, n, eta, a, L_host, mode, rmw::as_stream(stream));
}

}  // extern "C"
