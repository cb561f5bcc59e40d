"""GPU: products of few blobs in FP64 and df64 - tile pairs shared by several CTAs (from 256 blobs), finer
source splits of the one-sided kernels (below, and periodic) - against the oracle at tile edges and at the
sizes where the split changes, under a scratch limit, and bit-identical from call to call."""
import numpy as np
import pytest

from conftest import rel_err
from oracle import wall as owall
from rigidmultiblobswall_gb300 import _native
from rigidmultiblobswall_gb300 import mobility as mob

pytestmark = pytest.mark.gpu
# the modes' documented bar is 1e-12; FP64 sums of at most 2,100 pairs stay far below it
TOL = {"fp64": 2e-14, "df64": 1e-12}
KINDS = ["uf", "ut", "wf", "wt"]


def _blobs(n, seed, a):
    rng = np.random.default_rng(seed)
    r = np.empty((n, 3))
    r[:, :2] = rng.uniform(0, 2.5 * a * np.sqrt(n), (n, 2))
    r[:, 2] = rng.uniform(0.3 * a, 10 * a, n)
    return r, rng.standard_normal(3 * n)


@pytest.mark.parametrize("mode", ["fp64", "df64"])
@pytest.mark.parametrize("n", [1, 2, 31, 127, 129, 255, 256, 257, 512, 513, 1025, 2049])
def test_small_products_match_oracle(cuda_device, n, mode):
    a = 0.41
    r, v = _blobs(n, n, a)
    mob.autotune_clear()
    for kind in KINDS:
        ref, got = owall.wall_product(kind, r, v, 1.0, a), mob.wall_product(kind, r, v, 1.0, a, mode=mode)
        assert rel_err(got, ref) <= TOL[mode]
        assert np.array_equal(got, mob.wall_product(kind, r, v, 1.0, a, mode=mode))
        if n > 1:  # the self block of UT and WF is zero in free space
            ref, got = owall.no_wall_product(kind, r, v, 1.0, a), mob.no_wall_product(kind, r, v, 1.0, a, mode=mode)
            assert rel_err(got, ref) <= TOL[mode]


@pytest.mark.parametrize("mode", ["fp64", "df64"])
@pytest.mark.parametrize("n,L", [(77, (6.0, 6.0, 0.0)), (300, (12.0, 0.0, 0.0)), (640, (20.0, 21.0, 0.0)),
                                 (200, (0.0, 7.0, 6.0))])
def test_small_periodic_products_match_oracle(cuda_device, n, L, mode):
    a = 0.41
    r, v = _blobs(n, n + 1, a)
    L = np.array(L)
    for kind in KINDS:
        ref = owall.wall_product(kind, r, v, 1.0, a, periodic_length=L)
        assert rel_err(mob.wall_product(kind, r, v, 1.0, a, mode=mode, periodic_length=L), ref) <= TOL[mode]


@pytest.mark.parametrize("mode", ["fp64", "df64"])
def test_split_products_under_a_scratch_limit(cuda_device, mode):
    """Scratch limits from what the finest split asks for down to what one chunk does: the same products."""
    n, a = 1000, 0.41
    r, v = _blobs(n, 3, a)
    ref = owall.wall_product("uf", r, v, 1.0, a)
    refL = owall.wall_product("uf", r, v, 1.0, a, periodic_length=np.array([30.0, 30.0, 0.0]))
    try:
        for kib in (4096, 1024, 512, 192):  # 3 chunks of 24 kB and 64 kB of records: 136 kB
            _native.set_scratch_limit(kib << 10)
            assert rel_err(mob.wall_product("uf", r, v, 1.0, a, mode=mode), ref) <= TOL[mode]
            assert rel_err(mob.no_wall_product("uf", r, v, 1.0, a, mode=mode),
                           owall.no_wall_product("uf", r, v, 1.0, a)) <= TOL[mode]
            got = mob.wall_product("uf", r, v, 1.0, a, mode=mode, periodic_length=np.array([30.0, 30.0, 0.0]))
            assert rel_err(got, refL) <= TOL[mode]
    finally:
        _native.set_scratch_limit(0)
