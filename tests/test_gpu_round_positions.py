"""GPU: products that do not fill their last tile of 128 blobs, with a blob at a round position far from the others:
nothing that stands in for the missing blobs may meet it."""
import numpy as np
import pytest

from conftest import rel_err
from oracle import wall as owall
from rigidmultiblobswall_gb300 import mobility as mob

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["fp64", "df64"])
@pytest.mark.parametrize("at", [(1e6, 1e6, 1e6), (0.0, 0.0, 0.5), (0.0, 0.0, 1.0)])
def test_blob_at_a_round_position(cuda_device, mode, at):
    n, a = 300, 1.0
    rng = np.random.default_rng(6)
    r = np.column_stack([rng.uniform(5, 60, n), rng.uniform(5, 60, n), rng.uniform(1.0, 9.0, n)])
    r[17] = at
    v, t = rng.standard_normal(3 * n), rng.standard_normal(3 * n)
    for kind in ("uf", "ut", "wf", "wt"):
        ref = owall.wall_product(kind, r, v, 1.0, a)
        assert rel_err(mob.wall_product(kind, r, v, 1.0, a, mode=mode), ref) <= 1e-12
        ref = owall.no_wall_product(kind, r, v, 1.0, a)
        assert rel_err(mob.no_wall_product(kind, r, v, 1.0, a, mode=mode), ref) <= 1e-12
    for got, ref in zip(mob.wall_force_torque(r, v, t, 1.0, a, mode=mode), owall.force_torque(r, v, t, 1.0, a)):
        assert rel_err(got, ref) <= 1e-12


# mixed: the wall's symmetric kernels pinned, those of the free-space and force-torque products from 8,192 blobs
@pytest.mark.parametrize("at", [(1e6, 1e6, 1e6), (0.0, 0.0, 0.5), (0.0, 0.0, 1.0)])
def test_blob_at_a_round_position_mixed(cuda_device, at):
    n, a = 8300, 1.0
    rng = np.random.default_rng(7)
    r = np.column_stack([rng.uniform(5, 300, n), rng.uniform(5, 300, n), rng.uniform(1.0, 9.0, n)])
    r[17] = at
    v, t = rng.standard_normal(3 * n), rng.standard_normal(3 * n)
    few = r[:300]
    try:
        for kind in ("uf", "ut", "wf", "wt"):
            mob.autotune_set(kind, 300, "mixed", -1)
            ref = owall.wall_product(kind, few, v[:900], 1.0, a)
            assert rel_err(mob.wall_product(kind, few, v[:900], 1.0, a, mode="mixed"), ref) <= 1e-6
    finally:
        mob.autotune_clear()
    for kind in ("uf", "ut", "wf", "wt"):
        ref = owall.no_wall_product(kind, r, v, 1.0, a)
        assert rel_err(mob.no_wall_product(kind, r, v, 1.0, a, mode="mixed"), ref) <= 1e-6
    for got, ref in zip(mob.wall_force_torque(r, v, t, 1.0, a, mode="mixed"), owall.force_torque(r, v, t, 1.0, a)):
        assert rel_err(got, ref) <= 1e-6
