// Host build of csrc/fp64_int.cuh: the device intrinsics it uses, written out, and an exhaustive-edge driver that
// prints the largest errors in ulp (products and 1/sqrt against long double).
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <random>

static double seed_error;  // relative error given to the FP32 estimate of 1/sqrt
static uint64_t bits(double x) { uint64_t u; std::memcpy(&u, &x, 8); return u; }
static uint32_t __funnelshift_l(uint32_t lo, uint32_t hi, uint32_t s) { return s &= 31, s ? (hi << s) | (lo >> (32 - s)) : hi; }
static int __double2hiint(double x) { return (int)(bits(x) >> 32); }
static int __double2loint(double x) { return (int)(uint32_t)bits(x); }
static long long __double_as_longlong(double x) { return (long long)bits(x); }
static double __hiloint2double(int h, int l)
{
    const uint64_t u = ((uint64_t)(uint32_t)h << 32) | (uint32_t)l;
    double x;
    std::memcpy(&x, &u, 8);
    return x;
}
static uint32_t __umulhi(uint32_t a, uint32_t b) { return (uint32_t)(((uint64_t)a * b) >> 32); }
static int __mulhi(int a, int b) { return (int)(((int64_t)a * b) >> 32); }
static uint32_t __float2uint_rn(float x) { return x >= 4294967296.f ? 0xffffffffu : (uint32_t)std::nearbyint((double)x); }
using std::max;
using std::min;
static int __clzll(long long x) { return x ? __builtin_clzll((unsigned long long)x) : 64; }
static int __clz(int x) { return x ? __builtin_clz((unsigned)x) : 32; }
namespace rmw {
static float rsqrt_approx(float x) { return (float)((1.0 / std::sqrt((double)x)) * (1.0 + seed_error)); }
}
#include FP64_INT_HEADER

int main()
{
    using namespace rmw;
    std::mt19937_64 g(7);
    std::uniform_real_distribution<double> u(0.0, 1.0);
    auto ulp = [](double v) { int e; std::frexp(v, &e); return std::ldexp(1.0, e - 53); };
    auto number = [&](int span) {  // a positive number, every fourth one beside a power of two
        const double p = std::ldexp(1.0, (int)(g() % (2 * span)) - span);
        switch (g() % 12) {
        case 0: return p;
        case 1: return std::nextafter(p, 0.0);
        case 2: return std::nextafter(p, 1e300);
        default: return p * (1.0 + u(g));
        }
    };
    double ea = 0, ef = 0, em = 0, es = 0, er = 0;
    int bad = 0;
    for (int it = 0; it < 3000000; ++it) {
        const double a = number(200), b = number(200);
        const long double p = (long double)a * b;
        em = std::max(em, (double)(std::fabs(p - (long double)int_mul(a, b)) / ulp((double)p)));
        double sa = (g() & 1) ? -a : a, sb = (g() & 1) ? -b : b;
        es = std::max(es, (double)std::fabs(int_mul_signed(sa, sb) - (long double)sa * sb) / ulp(sa * sb));
        sa = (it & 1) ? -0.0 : ((it & 2) ? 0.0 : 3e-310);
        bad += int_mul_signed(sa, sb) != 0.0 || int_mul_signed(sb, sa) != 0.0;
        {
            const double fb = number(60), fa = it % 7 == 0 ? 0.0 : (it % 5 == 0 ? fb : number(60));
            double fc = it % 3 == 0 ? fa * fb * std::ldexp(1.0, (int)(g() % 9) - 4) : number(100);
            if (it % 11 == 0 && fa != 0.0) fc = 0.0;
            if (fa != 0.0 || fc != 0.0) {
                const long double w = (long double)fa * fb + fc;
                ef = std::max(ef, (double)(std::fabs(w - (long double)int_fma_pos((g() & 1) ? -fa : fa, fb, fc)) /
                                           ulp((double)w)));
            }
            bad += !(std::fabs(int_fma_pos(0.0, 0.0, -0.0)) < 1e-300);
        }
        {
            double fa = number(60), fb = number(60), fc = number(100);
            if (it % 3 == 0) fc = fa * fb * std::ldexp(1.0 + 1e-3 * u(g), (int)(g() % 9) - 4);
            if (it % 7 == 0) fa = 0.0;
            else if (it % 11 == 0) fc = 0.0;
            if (g() & 1) fa = -fa;
            if (g() & 1) fb = -fb;
            if (g() & 1) fc = -fc;
            const long double p = (long double)fa * fb, w = p + fc;
            const long double larger = std::max(std::fabs(p), (long double)std::fabs(fc));
            // half an ulp of the result, 2^-59 of the larger term
            const long double tol = 0.5L * ulp((double)(w == 0 ? larger : w)) + std::ldexp(larger, -59);
            ea = std::max(ea, (double)(std::fabs(w - (long double)int_fma(fa, fb, fc)) / tol));
            bad += int_fma(0.0, fb, 0.0) != 0.0 || int_fma(fa, -1.5, 1.5 * fa) > 1e-15 * std::fabs(fa);
        }
        seed_error = (u(g) - 0.5) * std::ldexp(1.0, -21);
        const double x = number(64);
        const long double y = 1.0L / std::sqrt((long double)x);
        er = std::max(er, (double)(std::fabs(y - (long double)int_rsqrt(x)) / ulp((double)y)));
        const double c = (it & 1) ? 4.0 : std::nextafter(4.0, (it & 2) ? 0.0 : 9.0);
        bad += MulInt::le4(c) != MulFp64::le4(c) || MulInt::lt4(c) != MulFp64::lt4(c);
        bad += MulInt::le4(x) != MulFp64::le4(x) || MulInt::lt4(x) != MulFp64::lt4(x);
    }
    const double lo = std::ldexp(1.0, -64), hi = std::ldexp(1.0, 64), inf = INFINITY;
    bad += !int_range(lo) || int_range(std::nextafter(lo, 0.0)) || int_range(hi) || !int_range(std::nextafter(hi, 0.0));
    bad += int_range(0.0) || int_range(inf) || int_range(NAN) || int_range(-1.0) || int_range(-NAN) || int_range(1e-310);
    for (double v : {0.0, -0.0, std::ldexp(1.0, -300), -std::nextafter(std::ldexp(1.0, 300), 0.0)}) bad += !int_range_vec(v);
    for (double v : {3e-310, std::ldexp(1.0, -301), std::ldexp(1.0, 300), -inf, (double)NAN}) bad += int_range_vec(v);
    bad += !int_range_sep(-4e9, 0.0, 1e-310) || int_range_sep(0.0, 4.3e9, 0.0) || int_range_sep(0.0, 0.0, NAN);
    std::printf("%.6f %.6f %.6f %.6f %.6f %d\n", ea, ef, em, es, er, bad);
    return 0;
}
