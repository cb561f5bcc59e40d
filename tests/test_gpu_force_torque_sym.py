"""GPU: the fused symmetric force-torque kernels in FP64 and df64 against the oracle: sizes around the tiles and
the size they start at, overlapping blobs and blobs on the wall, U alone, and under scratch limits that leave
room for four single products or for neither."""
import numpy as np
import pytest

from conftest import rel_err
from oracle import wall as owall
from rigidmultiblobswall_gb300 import _native
from rigidmultiblobswall_gb300 import mobility as mob

pytestmark = pytest.mark.gpu
TOL = {"fp64": 2e-14, "df64": 1e-12}  # sums of at most 2,100 pairs; the modes' bar is 1e-12
A = 0.39


def _case(n, seed):
    rng = np.random.default_rng(seed)
    r = np.empty((n, 3))
    r[:, :2] = rng.uniform(0, 2.2 * A * np.sqrt(n), (n, 2))
    r[:, 2] = rng.uniform(0.2 * A, 9 * A, n)
    k = np.arange(1, n, 5)  # overlapping neighbours
    r[k] = r[k - 1] + rng.uniform(0.2, 0.9, (k.size, 3)) * A
    return r, rng.standard_normal(3 * n), rng.standard_normal(3 * n)


@pytest.mark.parametrize("mode", ["fp64", "df64"])
@pytest.mark.parametrize("n", [255, 256, 257, 319, 321, 383, 385, 1025, 2049])
def test_fused_products_match_oracle(cuda_device, n, mode):
    r, F, T = _case(n, n)
    U0, W0 = owall.force_torque(r, F, T, 1.0, A)
    U, W = mob.wall_force_torque(r, F, T, 1.0, A, mode=mode)
    assert rel_err(U, U0) <= TOL[mode]
    assert rel_err(W, W0) <= TOL[mode]
    assert rel_err(mob.wall_force_torque(r, F, T, 1.0, A, with_rotation=False, mode=mode), U0) <= TOL[mode]
    U1, W1 = mob.wall_force_torque(r, F, T, 1.0, A, mode=mode)
    assert np.array_equal(U, U1) and np.array_equal(W, W1)


@pytest.mark.parametrize("mode", ["fp64", "df64"])
def test_fused_products_under_scratch_limits(cuda_device, mode):
    n = 4200
    r, F, T = _case(n, 7)
    rows = np.random.default_rng(1).choice(n, 40, replace=False)
    U0, W0 = owall.force_torque(r, F, T, 1.0, A, rows=rows)
    pick = lambda x: np.asarray(x).reshape(-1, 3)[rows].reshape(-1)  # noqa: E731
    try:
        # 6.7 MB of slots for the fused kernel unsplit, 3.3 MB for a single product; the one-sided pass asks for
        # 3.6 MB, and a limit below that is refused
        for mib in (64, 8, 4, 2):
            _native.set_scratch_limit(mib << 20)
            if mib == 2:
                with pytest.raises(_native.RMWError) as e:
                    mob.wall_force_torque(r, F, T, 1.0, A, mode=mode)
                assert e.value.code == _native.RMW_ERR_ALLOC
                continue
            U, W = mob.wall_force_torque(r, F, T, 1.0, A, mode=mode)
            assert rel_err(pick(U), U0) <= 2 * TOL[mode]
            assert rel_err(pick(W), W0) <= 2 * TOL[mode]
    finally:
        _native.set_scratch_limit(0)
