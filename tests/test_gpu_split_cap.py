"""GPU: a scratch cap between the unsplit and the finest split's scratch keeps the symmetric kernels, with the split
that fits beside the packed records: the products bit for bit those of the largest cap that allows that split alone."""
import numpy as np
import pytest

from conftest import rel_err
from oracle import wall as owall
from rigidmultiblobswall_gb300 import _native
from rigidmultiblobswall_gb300 import mobility as mob

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["fp64", "df64"])
@pytest.mark.parametrize("entry,comps", [("wall", 3), ("free", 3), ("periodic", 3), ("force_torque", 6)])
def test_cap_that_holds_whole_tile_pairs(cuda_device, entry, comps, mode):
    if entry == "periodic" and mode == "df64":
        pytest.skip("periodic df64 products are one-sided")
    n, a = 2100, 0.41
    rng = np.random.default_rng(8)
    r = np.empty((n, 3))
    r[:, :2] = rng.uniform(0, 2.5 * a * np.sqrt(n), (n, 2))
    r[:, 2] = rng.uniform(0.5 * a, 10 * a, n)
    v, t = rng.standard_normal(3 * n), rng.standard_normal(3 * n)
    L = np.array([50.0, 51.0, 0.0])
    run = {"wall": lambda: mob.wall_product("ut", r, v, 1.0, a, mode=mode),
           "free": lambda: mob.no_wall_product("uf", r, v, 1.0, a, mode=mode),
           "periodic": lambda: mob.wall_product("uf", r, v, 1.0, a, mode=mode, periodic_length=L),
           "force_torque": lambda: np.concatenate(mob.wall_force_torque(r, v, t, 1.0, a, mode=mode))}[entry]
    ref = {"wall": lambda: owall.wall_product("ut", r, v, 1.0, a),
           "free": lambda: owall.no_wall_product("uf", r, v, 1.0, a),
           "periodic": lambda: owall.wall_product("uf", r, v, 1.0, a, periodic_length=L),
           "force_torque": lambda: np.concatenate(owall.force_torque(r, v, t, 1.0, a))}[entry]()
    packed = (64 if comps == 3 else 96) * n
    packed = (packed + 255) // 256 * 256
    slot = 8 * comps * n * ((n + 127) // 128)
    mob.autotune_clear()
    try:
        for s in (1, 2):
            _native.set_scratch_limit(packed + s * slot)
            whole = run()
            assert rel_err(whole, ref) <= 1e-12
            _native.set_scratch_limit((s + 1) * slot + packed // 2)  # the next split's slots fit, its records do not
            assert np.array_equal(run(), whole)
    finally:
        _native.set_scratch_limit(0)
