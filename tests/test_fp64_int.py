"""The FP64 products and reciprocal square roots on the integer pipes (csrc/fp64_int.cuh): the arithmetic on the host
against long double, and the FP64 kernels that use it against the oracle where their two forms meet."""
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT, rel_err

A = 0.5


def test_integer_forms_on_the_host(tmp_path):
    src = open(os.path.join(ROOT, "rigidmultiblobswall_gb300", "csrc", "fp64_int.cuh")).read()
    for a, b in (("#include <cuda_runtime.h>", ""), ('#include "rmw_common.cuh"', ""), ("__device__ ", ""),
                 ("__forceinline__", "inline")):
        src = src.replace(a, b)
    header = tmp_path / "fp64_int.hpp"
    header.write_text(src)
    exe = tmp_path / "host"
    subprocess.run(["g++", "-O2", "-std=c++17", "-fwrapv", f'-DFP64_INT_HEADER="{header}"',
                    os.path.join(ROOT, "tests", "fp64_int_host.cpp"), "-o", str(exe)], check=True)
    any_sign, fma, mul, signed, rsqrt, bad = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split()
    # half an ulp, and what is left out: 3 units of the 64-bit product, 2^-10 .. 2^-9 ulp each, and one of the smaller
    # term of a sum, 2^-8; six of 2^-7 ulp
    assert float(fma) <= 0.5 + 3 * 2.0 ** -9 + 2.0 ** -8
    assert float(mul) <= 0.5 + 3 * 2.0 ** -9 and float(signed) <= 0.5 + 3 * 2.0 ** -9
    assert float(rsqrt) <= 0.5 + 6 * 2.0 ** -7
    assert float(any_sign) <= 1.0
    assert int(bad) == 0


def _blobs(n, seed):
    """Overlapping and far blobs, stacks (dx = dy = 0), equal heights (dz = 0), touching pairs (r = 2a to the bit)
    and one blob beyond the integer forms' range."""
    rng = np.random.default_rng(seed)
    r = rng.uniform(0.0, 4.0 * A * np.sqrt(n), (n, 3))
    r[:, 2] = rng.uniform(0.4 * A, 12 * A, n)
    r[1] = r[0] + [0.0, 0.0, 3 * A]
    r[2] = r[0] + [1.25 * A, 0.0, 0.0]
    r[3] = [100.0, 100.0, 1.0]
    r[4] = r[3] + [2 * A, 0.0, 0.0]
    r[n - 1] = [1e12, -1e12, 2.0]
    v = rng.standard_normal((n, 3))
    v[5] = 0.0
    v[6] = [0.0, 0.0, -1e-30]
    v[7] = [1e-200, 0.0, 0.0]
    return r, v


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["uf", "ut", "wf", "wt"])
@pytest.mark.parametrize("n", [9, 255, 256, 257, 640])
def test_fp64_products_match_oracle(cuda_device, kind, n):
    from oracle import wall as owall
    from rigidmultiblobswall_gb300 import mobility as mob
    r, v = _blobs(n, n)
    got = mob.wall_product(kind, r, v, 1.0, A, mode="fp64")
    assert rel_err(got, owall.wall_product(kind, r, v, 1.0, A)) <= 1e-14
    assert not np.any(mob.wall_product(kind, r, np.zeros_like(v), 1.0, A, mode="fp64"))


@pytest.mark.gpu
@pytest.mark.parametrize("n", [256, 300])
@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_non_finite_vectors_and_positions_reach_the_result(cuda_device, n, bad):
    from rigidmultiblobswall_gb300 import mobility as mob
    r, v = _blobs(n, n)
    r[n - 1] = [3.0, 3.0, 3.0]
    w = v.copy()
    w[8, 1] = bad
    out = np.asarray(mob.wall_product("uf", r, w, 1.0, A, mode="fp64")).reshape(-1, 3)
    assert not np.isfinite(np.delete(out, 8, axis=0)).any() and not np.isfinite(out[8, 1])
    s = r.copy()
    s[8, 0] = bad
    out = np.asarray(mob.wall_product("uf", s, v, 1.0, A, mode="fp64")).reshape(-1, 3)
    assert not np.isfinite(out[8]).all()


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["uf", "wf"])
@pytest.mark.parametrize("exponent", [-600, -290, 250, 700])
def test_scale_of_the_vector(cuda_device, kind, exponent):
    """Vectors within and beyond the integer forms' range: products are linear in a power of two."""
    from rigidmultiblobswall_gb300 import mobility as mob
    r, v = _blobs(300, 3)
    v[7] = 0.0
    ref = mob.wall_product(kind, r, v, 1.0, A, mode="fp64")
    got = mob.wall_product(kind, r, v * 2.0 ** exponent, 1.0, A, mode="fp64")
    assert rel_err(np.asarray(got) * 2.0 ** -exponent, ref) <= 1e-14
