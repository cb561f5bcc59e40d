"""The error bounds that csrc/fp64_int.cuh states, on the host against long double, and the FP64 reciprocal root of the
pair kernels on the GPU."""
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT

MAIN = r"""
int main()
{
    using namespace rmw;
    std::mt19937_64 g(11);
    std::uniform_real_distribution<double> u(0.0, 1.0);
    auto ulp = [](double v) { int e; std::frexp(v, &e); return std::ldexp(1.0, e - 53); };
    auto number = [&](int span) { return std::ldexp(1.0 + u(g), (int)(g() % (2 * span)) - span); };
    double ei = 0, es = 0, ef = 0;
    int bad = 0;
    for (int it = 0; it < 4000000; ++it) {
        double x = number(64);
        if (it % 5 == 0) x = std::nextafter(std::ldexp(1.0, (int)(g() % 120) - 60), it % 2 ? 0.0 : 1e300);
        const long double y = 1.0L / std::sqrt((long double)x);
        seed_error = (u(g) - 0.5) * std::ldexp(1.0, -21);
        ei = std::max(ei, (double)(std::fabs(y - (long double)int_rsqrt(x)) / ulp((double)y)));
        const double est = (double)(y * (1.0L + (it % 3 ? u(g) - 0.5 : (it & 1 ? 0.5 : -0.5)) * std::ldexp(2.0, -20)));
        es = std::max(es, (double)(std::fabs(y - (long double)rsqrt64_step(x, est)) / ulp((double)y)));
        const double a = (g() & 1 ? -1 : 1) * number(50), b = number(50);
        double c = -a * b * (1.0 + (it % 2 ? std::ldexp(u(g), -(int)(g() % 50)) : u(g)));
        if (it % 3 == 0) c = (g() & 1 ? -1 : 1) * number(100);
        const long double p = (long double)a * b, w = p + c;  // exact to 2^-64 of the larger term
        const long double larger = std::max(std::fabs(p), (long double)std::fabs(c));
        ef = std::max(ef, (double)((std::fabs(w - (long double)int_fma(a, b, c)) - std::ldexp(larger, -59)) /
                                   ulp((double)w)));
        bad += int_fma_pos(0.0, 0.0, 0.0) != 0.0 || int_fma_pos(-0.0, 0.0, -0.0) != 0.0;
    }
    std::printf("%.6f %.6f %.6f %d\n", ei, es, ef, bad);
    return 0;
}
"""


def test_stated_bounds_on_the_host(tmp_path):
    src = open(os.path.join(ROOT, "rigidmultiblobswall_gb300", "csrc", "fp64_int.cuh")).read()
    for a, b in (("#include <cuda_runtime.h>", ""), ('#include "rmw_common.cuh"', ""), ("__device__ ", ""),
                 ("__forceinline__", "inline")):
        src = src.replace(a, b)
    (tmp_path / "fp64_int.hpp").write_text(src)
    host = open(os.path.join(ROOT, "tests", "fp64_int_host.cpp")).read()  # the intrinsics
    (tmp_path / "main.cpp").write_text(host[:host.index("int main()")] + MAIN)
    exe = tmp_path / "host"
    subprocess.run(["g++", "-O2", "-std=c++17", "-fwrapv", f'-DFP64_INT_HEADER="{tmp_path}/fp64_int.hpp"',
                    str(tmp_path / "main.cpp"), "-o", str(exe)], check=True)
    rsqrt, step, fma, bad = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split()
    assert float(rsqrt) <= 0.51
    assert float(step) <= 1.0
    assert float(fma) <= 0.5 + 2.0 ** -8
    assert int(bad) == 0


@pytest.mark.gpu
def test_reciprocal_root_on_the_gpu(cuda_device):
    """Two blobs far apart in free space, the force across: the velocity is 1/r times factors that are one to the
    last bit or rounded once each (1 ulp for the root, half for each of six roundings)."""
    from rigidmultiblobswall_gb300 import mobility as mob
    rng = np.random.default_rng(2)
    dist = np.concatenate([2.0 ** rng.uniform(28, 100, 200), 2.0 ** np.arange(28, 60), 3.0 * 4.0 ** np.arange(14, 40)])
    nf = np.longdouble(1.0) / (8 * np.longdouble(np.pi))
    for x in dist:
        got = mob.no_wall_product("uf", np.array([[0, 0, 0], [x, 0, 0]]), np.array([0, 1.0, 0, 0, 0, 0]), 1.0, 1.0,
                                  mode="fp64")[4]
        ref = nf / np.longdouble(x)
        assert abs(np.longdouble(got) - ref) <= 4 * np.spacing(float(ref))
