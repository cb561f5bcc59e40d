"""GPU: the explicit M_UF blocks of the double-float pair kernels against the oracle where they can go wrong:
tails of the two-targets-per-thread tiles, overlapping blobs in one packed lane and not in the other, blobs on
and below the wall, far coordinates, and images in z (whose separation is not the difference of the heights)."""
import numpy as np
import pytest

from conftest import rel_err
from oracle import wall as owall
from rigidmultiblobswall_gb300 import mobility as mob

pytestmark = pytest.mark.gpu
# pairs are good to 2^-45 of 1/r; the sum of up to 1,000 of them over a result no smaller than the self term
TOL = 2e-13


def _blobs(n, seed, a, spread, zlo=0.2, overlap=True):
    rng = np.random.default_rng(seed)
    r = np.empty((n, 3))
    r[:, :2] = rng.uniform(0, spread, (n, 2))
    r[:, 2] = rng.uniform(zlo * a, 12 * a, n)
    if overlap:  # every third blob touches or overlaps its predecessor
        k = np.arange(1, n, 3)
        d = rng.standard_normal((k.size, 3))
        r[k] = r[k - 1] + d / np.linalg.norm(d, axis=1)[:, None] * rng.uniform(0.3, 2.2, k.size)[:, None] * a
        r[:, 2] = np.maximum(r[:, 2], zlo * a)
    return r, rng.standard_normal(3 * n)


def _run(r, v, a, mode, pin=None, L=None):
    mob.autotune_clear()
    if pin is not None:
        mob.autotune_set("uf", len(r), mode, pin)
    try:
        return mob.wall_product("uf", r, v, 1.0, a, mode=mode, periodic_length=np.zeros(3) if L is None else L)
    finally:
        mob.autotune_clear()


@pytest.mark.parametrize("pin", [-1, 8])
@pytest.mark.parametrize("n", [256, 319, 320, 321, 447, 448, 449, 1000])
def test_df64_block_tiles_and_overlaps(cuda_device, n, pin):
    a = 0.37
    r, v = _blobs(n, n, a, 1.5 * a * np.sqrt(n))
    assert rel_err(_run(r, v, a, "df64", pin), owall.wall_product("uf", r, v, 1.0, a)) <= TOL


@pytest.mark.parametrize("pin", [-1, 8])
def test_df64_block_low_and_far(cuda_device, pin):
    a = 1.3
    r, v = _blobs(300, 5, a, 400 * a, zlo=0.0, overlap=False)
    assert rel_err(_run(r, v, a, "df64", pin), owall.wall_product("uf", r, v, 1.0, a)) <= TOL


@pytest.mark.parametrize("L", [(9.0, 8.0, 0.0), (0.0, 9.0, 7.0), (9.0, 9.0, 8.0), (0.0, 0.0, 6.0)])
def test_df64_block_images(cuda_device, L):
    a = 0.4
    r, v = _blobs(131, 7, a, 9.0, zlo=0.5)
    L = np.array(L)
    ref = owall.wall_product("uf", r, v, 1.0, a, periodic_length=L)
    assert rel_err(_run(r, v, a, "df64", L=L), ref) <= 1e-12  # the mode's bar; up to 27 images of every pair
