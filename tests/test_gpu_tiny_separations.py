"""GPU: FP64 products of two blobs stacked but for a separation far below the range of the integer products: the
components that it alone makes, against the oracle."""
import numpy as np
import pytest

from oracle import wall as owall
from rigidmultiblobswall_gb300 import mobility as mob

pytestmark = pytest.mark.gpu
A = 0.41


@pytest.mark.parametrize("entry", ["wall", "free", "force_torque"])
@pytest.mark.parametrize("tiny", [1e-20, 1e-60, 1e-130, 1e-250])
@pytest.mark.parametrize("push", [(0.0, 0.0, 1.0), (1.0, 0.0, 0.0), (0.0, 1e-60, 1e-60)])
def test_almost_stacked_blobs(cuda_device, entry, tiny, push):
    n = 300
    rng = np.random.default_rng(3)
    r = np.column_stack([rng.uniform(20, 60, n), rng.uniform(20, 60, n), rng.uniform(1, 9, n)])
    r[0], r[1] = [0.0, 0.0, 2.0], [tiny, 0.0, 3.5]
    v = np.zeros((n, 3))
    v[0] = push
    if entry == "force_torque":
        got = mob.wall_force_torque(r, v.reshape(-1), v.reshape(-1), 1.0, A, mode="fp64")
        ref = owall.force_torque(r, v.reshape(-1), v.reshape(-1), 1.0, A)
        pairs = list(zip(got, ref))
    else:
        f, g = (mob.wall_product, owall.wall_product) if entry == "wall" else (mob.no_wall_product, owall.no_wall_product)
        pairs = [(f(k, r, v.reshape(-1), 1.0, A, mode="fp64"), g(k, r, v.reshape(-1), 1.0, A))
                 for k in ("uf", "ut", "wf", "wt")]
    for got, ref in pairs:
        got, ref = np.asarray(got).reshape(-1, 3)[1], np.asarray(ref).reshape(-1, 3)[1]
        # one pair: a few dozen roundings, up to a few digits of cancellation in a wall coefficient
        assert (np.abs(got - ref) <= 1e-13 * np.abs(ref) + 1e-300).all(), (got, ref)
