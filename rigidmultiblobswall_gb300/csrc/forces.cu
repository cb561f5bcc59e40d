// Blob forces on the GPU: the right-hand side of the mobility problem.
//
// * blob-blob repulsion (multi_bodies/forces_pycuda.py:40-118, Python form
//   multi_bodies/multi_bodies_functions.py:297-345): from the potential
//   U(r) = U0 exp(-(r - 2a)/b) for r > 2a (linear below), the force on blob i
//   is  f_i = -sum_{j != i} (eps/b) g(r_ij) (r_j - r_i) / r_ij  with
//   g = exp(-(r - 2a)/b) beyond 2a and 1 inside, minimum periodic image.
//   Pairs that can matter are evaluated in FP64, as the reference does; FP32
//   distances decide which.  A pair adds exactly 0 once (r - 2a)/b > 746, and
//   less than 2^-65 / n of the blob's largest term once
//     r > max(2a, r_min) + b (65 ln 2 + ln n),
//   r_min the distance to the nearest blob: all such pairs together change no
//   bit of the sum (the largest term's own rounding is 2^-53).  A component in
//   which the blob's largest terms vanish (stacked blobs, equal heights) may
//   live off those pairs: where its own largest term is below 2^-12 of the
//   blob's, it is summed again over every pair (far_kernel).  An optional
//   cutoff restricts the sum to pairs within it (the reference's
//   neighbour-list variant uses 2a + 30 b, multi_bodies/forces_numba.py:228-270).
//   Any blob's distance may stand for r_min, which only moves the line
//   outwards: the nearest of the 1,024 blobs around i in memory does.  One
//   FP32 pass over all pairs (candidates; two sources in packed lanes, 60 us
//   at 12,288 blobs) and the FP64 work of about 25 candidates per blob (lanes
//   of a warp have lists of different lengths), several source chunks per
//   target tile so that the GPU is full.
//   1,024 shells of 12 blobs with the wall and body reduction, Debye length
//   0.1a: 19.2 -> 0.22 ms (before: FP64 for a fifth of all pairs, lanes waiting
//   for each other's, on 96 CTAs); 0.5a 25.4 -> 0.91 ms; 1a 24.6 -> 2.4 ms;
//   172,032 blobs, 0.1a 195 -> 20 ms.  Of these 10 us are the test of the
//   components; with what far_kernel does, 20,000 free blobs 494 -> 551 us, a
//   layer of 12,321 blobs at one height 0.27 -> 0.66 ms, two of them 8.2 ms.
// * external blob forces (multi_bodies_functions.py:153-189): gravity
//   -g m e_z and the wall repulsion (e/b) exp(-(h - a)/b) (e/b for h <= a).
// The body reduction [F_b, T_b] = K^T f is rmw_rigid_KT_mult.
#include <algorithm>
#include <cmath>
#include <type_traits>

#include "pair_math.cuh"
#include "rmw_common.cuh"

namespace rmw {

namespace {

// Pair lists of the FP64 work: kPend candidates per thread in shared memory,
// evaluated together when some lane's list is full, so the lanes of a warp
// work on different pairs instead of waiting for each other's.  32 rather
// than 16: the blobs of three shells share a warp and meet their neighbours
// at different times (12,288 blobs, Debye length 0.5a: 1.22 -> 0.90 ms).
constexpr int kPend = 32;

// FP32 coordinates relative to the CTA's first target (absolute if that is not
// finite) in units of 2a + b, and the error bound of a distance to them: with
// m = |x_i| + |x_j| + L, rounding coordinates, differences and image shifts
// loses at most 6 2^-24 m per component, 6.2e-7 m in the distance, its sum and
// root 1.6e-7 m, and an image chosen differently next to L/2 6.2e-7 m.
constexpr float kErr = 2e-6f;

struct Box {
    double x, y, z;  // periodic lengths, 0 = none
    float fx, fy, fz, ix, iy, iz, big;  // in units of 2a + b: the same, their inverses, the largest
    float unit;      // 1 / (2a + b)
};

struct Screen {
    double x0[3];
    float x, y, z;  // this thread's target
    float ext;      // largest |coordinate| of the CTA's targets
};

template <int NT>
__device__ __forceinline__ Screen screen_setup(const double *__restrict__ r, int n, const Box &L, unsigned *bits)
{
    Screen s;
    const int i0 = blockIdx.x * NT, i = min(i0 + (int)threadIdx.x, n - 1);
    if (threadIdx.x == 0) *bits = 0u;
    for (int c = 0; c < 3; ++c) {
        s.x0[c] = r[3 * i0 + c];
        if (!isfinite(s.x0[c])) s.x0[c] = 0.0;
    }
    __syncthreads();
    s.x = (float)(r[3 * i] - s.x0[0]) * L.unit;
    s.y = (float)(r[3 * i + 1] - s.x0[1]) * L.unit;
    s.z = (float)(r[3 * i + 2] - s.x0[2]) * L.unit;
    atomicMax(bits, __float_as_uint(fmaxf(fabsf(s.x), fmaxf(fabsf(s.y), fabsf(s.z)))));
    __syncthreads();
    s.ext = __uint_as_float(*bits);
    return s;
}

// source tile: FP32 coordinates and the error bound w of distances to them,
// two sources side by side (x x' y y', z z' w w'), so that a scan works on
// packed pairs; a source past the end is out of every reach
__device__ __forceinline__ void screen_tile(const double *__restrict__ r, const Screen &s, const Box &L, int j, int j1,
                                            float4 *tile)
{
    float *o = (float *)(tile + 2 * (threadIdx.x >> 1)) + (threadIdx.x & 1);
    if (j >= j1) {
        o[0] = o[2] = o[4] = 3.0e18f;
        o[6] = 0.f;
    } else {
        const float x = (float)(r[3 * (size_t)j] - s.x0[0]) * L.unit,
                    y = (float)(r[3 * (size_t)j + 1] - s.x0[1]) * L.unit,
                    z = (float)(r[3 * (size_t)j + 2] - s.x0[2]) * L.unit;
        o[0] = x;
        o[2] = y;
        o[4] = z;
        o[6] = kErr * (fmaxf(fabsf(x), fmaxf(fabsf(y), fabsf(z))) + s.ext + L.big);
    }
}

__device__ __forceinline__ f2 image_f2(f2 d, float L, float inv)
{
    if (!(L > 0.f)) return d;
    const f2 t = f2_mul(d, f2_dup(inv));
    return f2_fma(f2_dup(-L), make_float2(rintf(t.x), rintf(t.y)), d);
}

template <bool PER>
__device__ __forceinline__ f2 screen_r2(const Screen &s, const Box &L, float4 a, float4 b)
{
    f2 ex = f2_sub(make_float2(a.x, a.y), f2_dup(s.x)), ey = f2_sub(make_float2(a.z, a.w), f2_dup(s.y)),
       ez = f2_sub(make_float2(b.x, b.y), f2_dup(s.z));
    if (PER) {
        ex = image_f2(ex, L.fx, L.ix);
        ey = image_f2(ey, L.fy, L.iy);
        ez = image_f2(ez, L.fz, L.iz);
    }
    return f2_fma(ex, ex, f2_fma(ey, ey, f2_mul(ez, ez)));
}

// The blobs with a component that lives off the pairs beyond the cut.
struct FarList {
    unsigned *count;  // number of them
    int *blob;        // in no particular order
    unsigned *mask;   // by blob: its components (bits 0 to 2) and, above, its finished chunks
};

// nearest[i] = min over the kNearWindow sources around blob i's tile of an upper
// bound on the distance to blob i (bit pattern of a positive float: atomicMin
// keeps it independent of the order); blobs that may coincide with i, which
// exert no force, do not count.  Any blob's distance bounds the largest term
// from below, so a window is as valid as all sources.  A shell's blobs are
// neighbours in memory, so theirs is the nearest blob; n free blobs in random
// order have about n / kNearWindow candidates more each, whose FP64 work is
// below that of the FP32 scan of the sources left out.
constexpr int kNearWindow = 1024, kNearSplit = 4;
template <int NT, bool PER>
__global__ void __launch_bounds__(NT) nearest_kernel(const double *__restrict__ r, int n, Box L,
                                                             unsigned *__restrict__ nearest, FarList far)
{
    __shared__ float4 tile[NT];
    __shared__ unsigned bits;
    const Screen s = screen_setup<NT>(r, n, L, &bits);
    const int i = blockIdx.x * NT + threadIdx.x;
    if (blockIdx.y == 0) {  // force_sum_kernel fills the list
        if (i < n) far.mask[i] = 0u;
        if (i == 0) *far.count = 0u;
    }
    const int w0 = max(0, min((int)blockIdx.x * NT - kNearWindow / 2, n - kNearWindow));
    const int j0 = w0 + blockIdx.y * (kNearWindow / kNearSplit), j1 = min(n, j0 + kNearWindow / kNearSplit);
    float best = 3.0e38f, err = 0.f;
    for (int t0 = j0; t0 < j1; t0 += NT) {
        __syncthreads();
        screen_tile(r, s, L, t0 + threadIdx.x, j1, tile);
        __syncthreads();
        const int cnt = min(NT, j1 - t0);
#pragma unroll 4
        for (int k = 0; k < cnt; k += 2) {
            const float4 a = tile[k], b = tile[k + 1];
            const f2 r2 = screen_r2<PER>(s, L, a, b), w2 = f2_mul(make_float2(b.z, b.w), make_float2(b.z, b.w));
            if (r2.x < best && r2.x > w2.x) {
                best = r2.x;
                err = b.z;
            }
            if (r2.y < best && r2.y > w2.y) {
                best = r2.y;
                err = b.w;
            }
        }
    }
    if (i < n && best < 3.0e38f) atomicMin(&nearest[i], __float_as_uint(fmaf(sqrtf(best), 1.0f + 1e-6f, err)));
}

// m of the force -m (dx, dy, dz) of one pair; 0: coincident blobs (no
// direction), or beyond rc (exactly zero).  1/r on the integer pipes, r = r^2 / r with one Newton
// correction (four FP64 instructions instead of the library's square root and division, about 35).
struct Pair {
    double dx, dy, dz, m;
};
template <bool PER>
__device__ __forceinline__ Pair pair_force(double dx, double dy, double dz, const Box &L, double eps_over_b,
                                           double inv_b, double two_a, double rc)
{
    if (PER) {
        if (L.x > 0) dx = project(dx, L.x);
        if (L.y > 0) dy = project(dy, L.y);
        if (L.z > 0) dz = project(dz, L.z);
    }
    const double r2 = dx * dx + dy * dy + dz * dz, invr = int_range(r2) ? int_rsqrt(r2) : rsqrt64(r2);
    const double r0 = r2 * invr;
    const double rn = fma(fma(-r0, r0, r2), 0.5 * invr, r0);
    if (!(rn > 0.0) || rn > rc) return {0.0, 0.0, 0.0, 0.0};
    const double g = (rn > two_a) ? exp(-(rn - two_a) * inv_b) : 1.0;
    return {dx, dy, dz, eps_over_b * g * invr};
}

// Size of a term m d from the exponents alone: |m d| >= 2^(term_size - 2046); 0: a factor is subnormal or zero
__device__ __forceinline__ int term_size(double m, double d)
{
    const int em = (__double2hiint(m) >> 20) & 0x7ff, ed = (__double2hiint(d) >> 20) & 0x7ff;
    return em && ed ? em + ed : 0;
}

// the cut (in units of 2a + b) that `nearest` allows: pairs beyond it are below 2^-65 / n of the blob's largest term
__device__ __forceinline__ float near_cut(float near, double two_a, const Box &L, float reach)
{
    return (fmaxf((float)two_a * L.unit, near) + reach) * (1.0f + 1e-6f);
}

// f_i over this CTA's sources: FP32 distances pick the candidates (nearest !=
// NULL: within max(2a, r_min) + reach; always within rc = rcut units), FP64
// evaluates them.
// Partial sums and term sizes to part[blockIdx.y][3n] and size[blockIdx.y][3n], or (part = NULL, one chunk, every
// pair) straight to f.
template <int NT, bool PER>
__global__ void __launch_bounds__(NT) blob_blob_kernel(const double *__restrict__ r, double *__restrict__ f,
                                                               double *__restrict__ part,
                                                               unsigned short *__restrict__ size, int n, int chunk,
                                                               double eps_over_b, double inv_b, double two_a,
                                                               double rc, float rcut,
                                                               const unsigned *__restrict__ nearest, float reach,
                                                               Box L, int accumulate)
{
    __shared__ float4 tile[NT];
    __shared__ int pend[kPend][NT];
    __shared__ unsigned bits;
    const Screen s = screen_setup<NT>(r, n, L, &bits);
    const int tid = threadIdx.x, i = blockIdx.x * NT + tid;
    const bool valid = i < n;
    const int ii = valid ? i : n - 1;
    const double xi = r[3 * (size_t)ii], yi = r[3 * (size_t)ii + 1], zi = r[3 * (size_t)ii + 2];
    // (a bound FP32 cannot hold: no screen, every pair is a candidate)
    float cut = rcut < 1e15f ? rcut : __int_as_float(0x7fffffff);
    if (nearest) {
        const float near = __uint_as_float(nearest[ii]);
        if (near < 1e15f) cut = fminf(cut, near_cut(near, two_a, L, reach));
    }
    if (!valid) cut = -1e30f;  // no candidate
    double fx = 0.0, fy = 0.0, fz = 0.0;
    int ex = 0, ey = 0, ez = 0;  // the largest term_size of each component
    int np = 0;
    auto drain = [&]() {  // every lane works off its list
        for (int k = 0; __any_sync(0xffffffffu, k < np); ++k) {
            if (k >= np) continue;
            const size_t j = pend[k][tid];
            const Pair p = pair_force<PER>(r[3 * j] - xi, r[3 * j + 1] - yi, r[3 * j + 2] - zi, L, eps_over_b, inv_b,
                                           two_a, rc);
            fx -= p.m * p.dx;
            fy -= p.m * p.dy;
            fz -= p.m * p.dz;
            ex = max(ex, term_size(p.m, p.dx));
            ey = max(ey, term_size(p.m, p.dy));
            ez = max(ez, term_size(p.m, p.dz));
        }
        np = 0;
    };
    const int j0 = blockIdx.y * chunk, j1 = min(n, j0 + chunk);
    for (int t0 = j0; t0 < j1; t0 += NT) {
        __syncthreads();
        screen_tile(r, s, L, t0 + tid, j1, tile);
        __syncthreads();
        const int cnt = min(NT, j1 - t0);
        for (int k0 = 0; k0 < cnt; k0 += kPend / 2) {
            const int k1 = min(cnt, k0 + kPend / 2);
            for (int k = k0; k < k1; k += 2) {
                const float4 a = tile[k], b = tile[k + 1];
                const f2 r2 = screen_r2<PER>(s, L, a, b), t = f2_add(f2_dup(cut), make_float2(b.z, b.w));
                const f2 t2 = f2_mul(t, make_float2(fabsf(t.x), fabsf(t.y)));
                if (!(r2.x >= t2.x) && t0 + k != i) pend[np++][tid] = t0 + k;
                if (!(r2.y >= t2.y) && t0 + k + 1 != i && k + 1 < cnt) pend[np++][tid] = t0 + k + 1;
            }
            if (__any_sync(0xffffffffu, np > kPend / 2)) drain();
        }
    }
    drain();
    if (!valid) return;
    if (part) {
        double *o = part + ((size_t)blockIdx.y * n + i) * 3;
        o[0] = fx; o[1] = fy; o[2] = fz;
        unsigned short *q = size + ((size_t)blockIdx.y * n + i) * 3;
        q[0] = ex; q[1] = ey; q[2] = ez;
    } else if (accumulate) {
        f[3 * (size_t)i] += fx;
        f[3 * (size_t)i + 1] += fy;
        f[3 * (size_t)i + 2] += fz;
    } else {
        f[3 * (size_t)i] = fx;
        f[3 * (size_t)i + 1] = fy;
        f[3 * (size_t)i + 2] = fz;
    }
}

// Sum of the chunks, component by component, and the test of the cut: with
// T = 2^log_t a bound on the blob's largest term from below (its nearest
// blob's, at most), all pairs beyond the cut are below 2^-65 T, that is
// below 2^-53 of the component's own largest term if that is 2^-12 T or more.
__global__ void force_sum_kernel(const double *__restrict__ part, const unsigned short *__restrict__ size,
                                 double *__restrict__ f, int m, int nchunks, int accumulate,
                                 const unsigned *__restrict__ nearest, float reach, float rcut, double two_a,
                                 float log_eps, float log_slope, Box L, FarList far)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= m) return;
    double v = 0.0;
    int e = 0;
#pragma unroll 8
    for (int c = 0; c < nchunks; ++c) {
        v += part[(size_t)c * m + k];
        e = max(e, (int)size[(size_t)c * m + k]);
    }
    const int i = k / 3;
    const float near = __uint_as_float(nearest[i]);
    if (near < 1e15f && !(near_cut(near, two_a, L, reach) >= rcut)) {
        const float log_t = log_eps - fmaxf(near - (float)two_a * L.unit, 0.f) * log_slope;
        if ((float)(e - 2046) < log_t - 11.0f) {  // 2^-12 and the rounding of log_t
            if (atomicOr(&far.mask[i], 1u << (k - 3 * i)) == 0) far.blob[atomicAdd(far.count, 1u)] = i;
            return;
        }
    }
    f[k] = accumulate ? f[k] + v : v;
}

// The listed components over every pair within rc, chunk by chunk of the
// sources into the blob's own slots of part; the CTA that finishes a blob's
// last chunk adds them in order.  A CTA takes eight blobs, a warp each, or
// while few are listed one blob, so that a handful does not wait for one
// warp's scan (15 of 20,000 free blobs: a warp each 1,000 us).  Pairs whose
// coordinates agree in every listed component contribute nothing to it: the
// coordinates' bits, an integer compare, leave a layer of blobs of equal
// height without FP64 work.
constexpr int kFarThreads = 256, kFarWarps = kFarThreads / 32;
template <bool PER>
__global__ void __launch_bounds__(kFarThreads) far_kernel(const double *__restrict__ r, double *__restrict__ f,
                                                          double *part, int n, int chunk, int nchunks,
                                                          double eps_over_b, double inv_b, double two_a, double rc,
                                                          Box L, int accumulate, FarList far)
{
    __shared__ double tile[3][kFarThreads];
    __shared__ double red[kFarWarps][3];
    const unsigned count = *far.count;
    if (count == 0) return;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const bool one = count < 152 * 8;
    const unsigned items = (one ? count : (count + kFarWarps - 1) / kFarWarps) * nchunks;
    for (unsigned item = blockIdx.x; item < items; item += gridDim.x) {
        const unsigned g = item / nchunks, c = item % nchunks, q = one ? g : g * kFarWarps + warp;
        const bool on = q < count;
        const int i = on ? far.blob[q] : 0;
        const unsigned mask = on ? *(volatile unsigned *)&far.mask[i] & 7u : 0u;
        const double xi = r[3 * (size_t)i], yi = r[3 * (size_t)i + 1], zi = r[3 * (size_t)i + 2];
        double v[3] = {0.0, 0.0, 0.0};
        const int j1 = min(n, (int)(c + 1) * chunk);
        for (int t0 = c * chunk; t0 < j1; t0 += kFarThreads) {
            const int cnt = min(kFarThreads, j1 - t0);
            __syncthreads();
            for (int k = threadIdx.x; k < 3 * cnt; k += kFarThreads) tile[k % 3][k / 3] = r[3 * (size_t)t0 + k];
            __syncthreads();
            for (int k = one ? threadIdx.x : lane; k < cnt; k += one ? kFarThreads : 32) {
                const double x = tile[0][k], y = tile[1][k], z = tile[2][k];
                const bool any = ((mask & 1u) && __double_as_longlong(x) != __double_as_longlong(xi)) ||
                                 ((mask & 2u) && __double_as_longlong(y) != __double_as_longlong(yi)) ||
                                 ((mask & 4u) && __double_as_longlong(z) != __double_as_longlong(zi));
                if (!any) continue;
                const Pair p = pair_force<PER>(x - xi, y - yi, z - zi, L, eps_over_b, inv_b, two_a, rc);
                v[0] -= p.m * p.dx;
                v[1] -= p.m * p.dy;
                v[2] -= p.m * p.dz;
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
            for (int d = 0; d < 3; ++d) v[d] += __shfl_down_sync(0xffffffffu, v[d], o);
        if (one) {
            if (lane == 0)
                for (int d = 0; d < 3; ++d) red[warp][d] = v[d];
            __syncthreads();
            for (int d = 0; d < 3; ++d) {
                v[d] = 0.0;
                for (int w = 0; w < kFarWarps; ++w) v[d] += red[w][d];
            }
        }
        if (lane != 0 || !on || (one && warp != 0)) continue;
        for (int d = 0; d < 3; ++d) __stcg(&part[((size_t)c * n + i) * 3 + d], v[d]);
        __threadfence();
        if ((atomicAdd(&far.mask[i], 8u) >> 3) != nchunks - 1u) continue;
        __threadfence();
        for (int d = 0; d < 3; ++d) {
            if (!(mask & (1u << d))) continue;
            double sum = 0.0;
            for (int k = 0; k < nchunks; ++k) sum += __ldcg(&part[((size_t)k * n + i) * 3 + d]);
            f[3 * (size_t)i + d] = accumulate ? f[3 * (size_t)i + d] + sum : sum;
        }
    }
}

__global__ void external_force_kernel(const double *__restrict__ r, double *__restrict__ f, int n, double weight,
                                      double blob_radius, double e_over_b, double inv_b, int accumulate)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double h = r[3 * i + 2];
    const double fz = -weight + ((h > blob_radius) ? e_over_b * exp(-(h - blob_radius) * inv_b) : e_over_b);
    if (accumulate) {
        f[3 * i + 2] += fz;
    } else {
        f[3 * i] = 0.0;
        f[3 * i + 1] = 0.0;
        f[3 * i + 2] = fz;
    }
}

template <int NT, bool PER>
int blob_blob_launch(const double *r, double *f, int n, double eps_over_b, double b, double two_a, double rc,
                     const Box &L, int accumulate, cudaStream_t st)
{
    const int tiles = (n + NT - 1) / NT;
    // enough CTAs for eight per SM, no chunk below two tiles of sources
    const int want = std::min((152 * 8 + tiles - 1) / tiles, std::max(1, n / (2 * NT)));
    const int chunk = (((n + want - 1) / want + NT - 1) / NT) * NT;
    const int nchunks = (n + chunk - 1) / chunk;
    auto up = [](size_t b) { return (b + 255) / 256 * 256; };
    const size_t word = up(sizeof(unsigned) * (size_t)n), sums = up(sizeof(double) * 3 * (size_t)n * nchunks);
    const size_t bytes = 3 * word + 256 + sums + sizeof(unsigned short) * 3 * (size_t)n * nchunks;
    // Without scratch (a capture must not allocate; a scratch limit; memory
    // pressure) one chunk and the fixed radius: same pairs to rounding, slower.
    const float rcut = (float)(rc / (two_a + b) * 1.000001);
    void *ws = nullptr;
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(st, &cap) != cudaSuccess || cap != cudaStreamCaptureStatusNone ||
        scratch(SCRATCH_FORCES, bytes, &ws, st) != RMW_OK) {
        cudaGetLastError();
        blob_blob_kernel<NT, PER><<<tiles, NT, 0, st>>>(r, f, nullptr, nullptr, n, n, eps_over_b, 1.0 / b, two_a, rc,
                                                        rcut, nullptr, 0.f, L, accumulate);
        RMW_CHECK_LAUNCH("blob-blob forces");
        return RMW_OK;
    }
    char *p = (char *)ws;
    unsigned *nearest = (unsigned *)p;
    const FarList far = {(unsigned *)(p + word), (int *)(p + word + 256), (unsigned *)(p + 2 * word + 256)};
    double *part = (double *)(p + 3 * word + 256);
    unsigned short *size = (unsigned short *)(p + 3 * word + 256 + sums);
    const dim3 grid(tiles, nchunks);
    RMW_CUDA(cudaMemsetAsync(nearest, 0x7f, sizeof(unsigned) * (size_t)n, st));  // 3.4e38
    nearest_kernel<NT, PER><<<dim3(tiles, kNearSplit), NT, 0, st>>>(r, n, L, nearest, far);
    const float reach = (float)(b / (two_a + b) * (65.0 * 0.69314718055994531 + std::log((double)n)) * 1.000001);
    blob_blob_kernel<NT, PER><<<grid, NT, 0, st>>>(r, f, part, size, n, chunk, eps_over_b, 1.0 / b, two_a, rc, rcut,
                                                   nearest, reach, L, accumulate);
    force_sum_kernel<<<(3 * n + 255) / 256, 256, 0, st>>>(
        part, size, f, 3 * n, nchunks, accumulate, nearest, reach, rcut, two_a,
        (float)std::log2(std::fabs(eps_over_b)), (float)((two_a + b) / b * 1.4426950408889634), L, far);
    far_kernel<PER><<<152 * 4, kFarThreads, 0, st>>>(r, f, part, n, chunk, nchunks, eps_over_b, 1.0 / b, two_a, rc, L,
                                                     accumulate, far);
    RMW_CHECK_LAUNCH("blob-blob forces");
    return RMW_OK;
}

}  // namespace

static int blob_blob(const double *r, double *f, int n, double eps_over_b, double b, double two_a, double rc, double Lx,
                     double Ly, double Lz, int accumulate, cudaStream_t st)
{
    const double unit = 1.0 / (two_a + b);
    auto inv = [unit](double L) { return L > 0 ? (float)(1.0 / (L * unit)) : 0.f; };
    const Box L = {Lx, Ly, Lz, (float)(Lx * unit), (float)(Ly * unit), (float)(Lz * unit), inv(Lx), inv(Ly), inv(Lz),
                   (float)(unit * std::max(0.0, std::max(Lx, std::max(Ly, Lz)))), (float)unit};
    const bool per = Lx > 0 || Ly > 0 || Lz > 0;
    auto launch = [&](auto nt) {
        constexpr int NT = decltype(nt)::value;
        return per ? blob_blob_launch<NT, true>(r, f, n, eps_over_b, b, two_a, rc, L, accumulate, st)
                   : blob_blob_launch<NT, false>(r, f, n, eps_over_b, b, two_a, rc, L, accumulate, st);
    };
    // Targets per CTA.  A tile's FP64 work falls to the one CTA whose sources
    // are its neighbours, so small suspensions take tiles small enough to
    // reach every SM; large ones the tile that reads sources least often.
    // 32 / 64 / 128 targets, Debye length 0.4a: 600 blobs 123 / 201 / 344 us,
    // 4,200 387 / 401 / 542, 9,600 541 / 529 / 552, 12,288 720 / 689 / 652;
    // 0.1a: 4,200 175 / 205 / 248, 12,288 244 / 219 / 215.
    if (n <= 6000) return launch(std::integral_constant<int, 32>());
    if (n <= 11000) return launch(std::integral_constant<int, 64>());
    return launch(std::integral_constant<int, 128>());
}

}  // namespace rmw

extern "C" {

// f (+)= blob-blob repulsion forces of n blobs (device arrays, 3n doubles);
// cutoff <= 0: every pair (exact), else pairs within the cutoff only.
int rmw_blob_blob_forces(const double *r, double *f, int64_t n, double repulsion_strength, double debye_length,
                         double blob_radius, double cutoff, const double *L_host, int accumulate, void *stream)
{
    if (n < 0 || n > (int64_t(1) << 28)) return rmw::fail(RMW_ERR_ARG, "number of blobs out of range [0, 2^28]");
    if (n > 0 && (!r || !f)) return rmw::fail(RMW_ERR_ARG, "null array pointer");
    if (!(debye_length > 0) || !(blob_radius >= 0))
        return rmw::fail(RMW_ERR_ARG, "debye length must be positive and the blob radius non-negative");
    if (n == 0) return RMW_OK;
    const double Lx = L_host ? L_host[0] : 0.0, Ly = L_host ? L_host[1] : 0.0, Lz = L_host ? L_host[2] : 0.0;
    // beyond 2a + 746 b the FP64 exponential is exactly zero: such pairs
    // contribute nothing; a positive cutoff truncates earlier (pairs farther
    // than it are left out, as the reference's neighbour-list variant does)
    const double rexact = 2.0 * blob_radius + 746.0 * debye_length;
    const double rc = (cutoff > 0.0) ? fmin(cutoff, rexact) : rexact;
    const int N = (int)n;
    return rmw::blob_blob(r, f, N, repulsion_strength / debye_length, debye_length, 2.0 * blob_radius, rc, Lx, Ly, Lz,
                          accumulate, rmw::as_stream(stream));
}

// f (+)= gravity and wall repulsion of n blobs (device arrays, 3n doubles).
int rmw_blob_external_forces(const double *r, double *f, int64_t n, double blob_mass, double blob_radius, double g,
                             double repulsion_strength_wall, double debye_length_wall, int accumulate, void *stream)
{
    if (n < 0 || n > (int64_t(1) << 28)) return rmw::fail(RMW_ERR_ARG, "number of blobs out of range [0, 2^28]");
    if (n > 0 && (!r || !f)) return rmw::fail(RMW_ERR_ARG, "null array pointer");
    if (!(debye_length_wall > 0)) return rmw::fail(RMW_ERR_ARG, "wall debye length must be positive");
    if (n == 0) return RMW_OK;
    const int N = (int)n;
    rmw::external_force_kernel<<<(N + 255) / 256, 256, 0, rmw::as_stream(stream)>>>(
        r, f, N, g * blob_mass, blob_radius, repulsion_strength_wall / debye_length_wall, 1.0 / debye_length_wall,
        accumulate);
    RMW_CHECK_LAUNCH("external blob forces");
    return RMW_OK;
}

}  // extern "C"
