"""A product's scratch buffer serves every smaller product of its route (csrc/product_plan.h): the rules on the host,
and on the GPU the device memory that smaller products take after a larger one."""
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT

MAIN = r"""
#include <cstdio>
#include "product_plan.h"
int main()
{
    using namespace rmw;
    long long bad = 0;
    for (int comps : {3, 6})
        for (int form = 0; form < 3; ++form) {
            double most = 0.0;
            for (int n = 256; n < 40000; ++n) {
                const double packed = (comps == 6 ? 96.0 : 64.0) * n;
                const int s = sym_split(form > 0, form == 2, n, comps, packed, 1e11, 0.0);
                most = std::max(most, packed + sym_slot_bytes(n, comps) * s);
                bad += most > packed + sym_reserve_bytes(n, comps);
            }
        }
    for (bool fp64 : {false, true}) {
        double most = 0.0;
        for (int n = 1; n < 60000; ++n) {
            const double packed = 64.0 * n;
            most = std::max(most, packed + 24.0 * n * fine_chunks(fp64, n, packed, 0.0));
            bad += most > packed + fine_reserve_bytes(n);
            const double cap = packed + 24.0 * n * (coarse_chunks(n) + 2.5);
            bad += packed + 24.0 * n * fine_chunks(fp64, n, packed, cap) > cap;
        }
    }
    std::printf("%lld\n", bad);
    return 0;
}
"""


def test_reserve_covers_smaller_products(tmp_path):
    (tmp_path / "main.cpp").write_text(MAIN)
    exe = tmp_path / "plan"
    csrc = os.path.join(ROOT, "rigidmultiblobswall_gb300", "csrc")
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", csrc, str(tmp_path / "main.cpp"), "-o", str(exe)], check=True)
    assert subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.strip() == "0"


@pytest.mark.gpu
@pytest.mark.parametrize("mode", ["fp64", "df64"])
@pytest.mark.parametrize("entry", ["wall", "free", "periodic", "force_torque"])
def test_smaller_products_take_no_more_memory(cuda_device, entry, mode):
    import torch
    from rigidmultiblobswall_gb300 import _native
    from rigidmultiblobswall_gb300 import mobility as mob
    # largest sizes whose own split is coarse: 22 MB of partial sums (df64; 10,000 blobs 38 MB), 38 MB (9,000: 61 MB)
    a, sizes = 0.41, (10752 if mode == "df64" else 14000, 10000, 9000, 5003, 1500, 300)
    rng = np.random.default_rng(2)
    n = sizes[0]
    r = rng.uniform(0, 60, (n, 3))
    r[:, 2] = 0.5 + 0.2 * r[:, 2]
    dev = [torch.tensor(x, device="cuda") for x in (r, rng.standard_normal((n, 3)), rng.standard_normal((n, 3)))]
    L = np.array([60.0, 60.0, 0.0])

    def run(m):
        x, v, t = (q[:m].contiguous() for q in dev)
        if entry == "force_torque":
            mob.wall_force_torque(x, v.reshape(-1), t.reshape(-1), 1.0, a, mode=mode)
        elif entry == "free":
            mob.no_wall_product("uf", x, v.reshape(-1), 1.0, a, mode=mode)
        else:
            mob.wall_product("uf", x, v.reshape(-1), 1.0, a, mode=mode, periodic_length=L if entry == "periodic" else None)
        torch.cuda.synchronize()
        return torch.cuda.mem_get_info()[0]

    mob.autotune_clear()
    for m in sizes:  # the caching allocator's and the library's own first allocations
        run(m)
    _native.release_scratch()
    try:
        free = run(sizes[0])
        assert all(run(m) == free for m in sizes[1:])
    finally:
        _native.release_scratch()
