"""The warp's tridiagonal eigen-solver (csrc/krylov_device.cu) with its lanes out of step: a host build runs 32 lanes
one after the other between two synchronisations, the furthest apart that the hardware may let them get, in both
orders."""
import os
import subprocess



from conftest import ROOT

MAIN = r"""
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>
#include <ucontext.h>
#include <vector>
static int __double2hiint(double x) { uint64_t u; std::memcpy(&u, &x, 8); return (int)(u >> 32); }
static double rsqrt64(double x) { return 1.0 / std::sqrt(x); }
static int __ffs(unsigned x) { return x ? __builtin_ctz(x) + 1 : 0; }
static ucontext_t driver, lane_ctx[32];
static bool done[32];
static unsigned votes;
static int me;
static void __syncwarp() { swapcontext(&lane_ctx[me], &driver); }  // the other lanes' turn
static unsigned __ballot_sync(unsigned, bool p)
{
    votes = p ? votes | 1u << me : votes & ~(1u << me);
    __syncwarp();
    const unsigned v = votes;
    __syncwarp();
    return v;
}
using std::copysign; using std::fabs; using std::hypot; using std::sqrt;
#include SOLVER

static std::vector<double> d, e, z;
static int k;
static bool ok[32];
static char stacks[32][1 << 16];
static void lane_main()
{
    const int l = me;
    ok[l] = tridiag_eigen_warp(d.data(), e.data(), z.data(), k, l);
    done[l] = true;
}

int main()
{
    std::mt19937_64 g(3);
    std::uniform_real_distribution<double> u(-1.0, 1.0);
    double worst = 0.0;
    for (int rows : {1, 2, 5, 31, 32, 33, 40, 70})
        for (int kind = 0; kind < 2; ++kind)
            for (int s : {1, -1}) {
                k = rows;
                d.assign(k, 0.0); e = d; z.assign(k * k, 0.0);
                for (int q = 0; q < k; ++q) {
                    d[q] = kind ? u(g) : 2.0;
                    e[q] = q + 1 < k ? (kind ? u(g) * (q % 7 ? 1.0 : 0.0) : -1.0) : 0.0;
                }
                const std::vector<double> d0 = d, e0 = e;
                for (int l = 0; l < 32; ++l) {
                    getcontext(&lane_ctx[l]);
                    lane_ctx[l].uc_stack.ss_sp = stacks[l];
                    lane_ctx[l].uc_stack.ss_size = sizeof stacks[l];
                    lane_ctx[l].uc_link = &driver;
                    makecontext(&lane_ctx[l], lane_main, 0);
                    done[l] = ok[l] = false;
                }
                bool more = true;
                for (int round = 0; more && round < 1000000; ++round) {  // every lane up to its next synchronisation
                    more = false;
                    for (int q = 0; q < 32; ++q) {
                        me = s > 0 ? q : 31 - q;
                        if (!done[me]) swapcontext(&driver, &lane_ctx[me]);
                        more = more || !done[me];
                    }
                }
                for (bool b : ok) if (!b) worst = INFINITY;
                for (int i = 0; i < k; ++i)
                    for (int j = 0; j < k; ++j) {  // Z diag(d) Z^T against the matrix
                        double a = 0.0;
                        for (int q = 0; q < k; ++q) a += z[i + k * q] * d[q] * z[j + k * q];
                        const double t = i == j ? d0[i] : (i == j + 1 ? e0[j] : (j == i + 1 ? e0[i] : 0.0));
                        if (!(std::fabs(a - t) <= worst)) worst = std::fabs(a - t);
                    }
            }
    std::printf("%g\n", worst);
    return 0;
}
"""


def test_lanes_out_of_step(tmp_path):
    src = open(os.path.join(ROOT, "rigidmultiblobswall_gb300", "csrc", "krylov_device.cu")).read()
    cut = lambda a, b: src[src.index(a):src.index(b)]  # noqa: E731
    code = (cut("struct RootInv", "// The first jobs of a CTA") +
            cut("__device__ bool tridiag_eigen_warp", "struct LzArgs"))
    for a, b in (("__device__ ", ""), ("__forceinline__", "inline")):
        code = code.replace(a, b)
    (tmp_path / "solver.hpp").write_text(code)
    (tmp_path / "main.cpp").write_text(MAIN)
    exe = tmp_path / "lanes"
    subprocess.run(["g++", "-O2", "-std=c++17", f'-DSOLVER="{tmp_path}/solver.hpp"',
                    str(tmp_path / "main.cpp"), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0
    # 40 rows, entries of order 1, some 60 rotations a column: a few hundred roundings
    assert float(out.stdout) <= 1e-13
