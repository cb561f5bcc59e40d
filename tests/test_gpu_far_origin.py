"""GPU: FP64 wall products of blobs near each other and far from the origin - separations are formed before they are
scaled by a radius that is not a power of two - against the oracle, through the symmetric kernel (from 256 blobs,
periodic in x and y too) and the one-sided one."""
import numpy as np
import pytest

from conftest import rel_err
from oracle import wall as owall
from rigidmultiblobswall_gb300 import mobility as mob

pytestmark = pytest.mark.gpu
A = 0.41


def _blobs(n, offset):
    rng = np.random.default_rng(n)
    r = np.empty((n, 3))
    r[:, :2] = rng.uniform(0, 2.5 * A * np.sqrt(n), (n, 2))
    r[:, 2] = rng.uniform(0.5 * A, 10 * A, n)
    return r + np.array(offset), rng.standard_normal(3 * n)


# sums of at most 1,000 pairs whose inputs are exact: the bar of the FP64 products at the origin
@pytest.mark.parametrize("kind", ["uf", "ut", "wf", "wt"])
@pytest.mark.parametrize("n", [200, 256, 257, 1000])
@pytest.mark.parametrize("offset", [(4.3e3, -4.1e3, 0.0), (4.3e5, 3.9e5, 0.0), (0.0, 0.0, 4.1e5)])
def test_products_far_from_the_origin(cuda_device, kind, n, offset):
    r, v = _blobs(n, offset)
    mob.autotune_clear()
    assert rel_err(mob.wall_product(kind, r, v, 1.0, A, mode="fp64"), owall.wall_product(kind, r, v, 1.0, A)) <= 2e-14


@pytest.mark.parametrize("offset", [(4.3e5, 3.9e5, 0.0), (0.0, 0.0, 4.1e5)])
def test_periodic_products_far_from_the_origin(cuda_device, offset):
    r, v = _blobs(300, offset)
    L = np.array([19.0, 20.0, 0.0])
    ref = owall.wall_product("uf", r, v, 1.0, A, periodic_length=L)
    assert rel_err(mob.wall_product("uf", r, v, 1.0, A, mode="fp64", periodic_length=L), ref) <= 2e-14
