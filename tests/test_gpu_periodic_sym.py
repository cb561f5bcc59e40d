"""GPU: FP64 products periodic in x and / or y through the symmetric kernel, against the oracle and the one-sided
kernel: tile tails, splits, blobs several boxes away, pairs exactly half a box apart (where the minimum image
flips), and lattices with z periodic, which keep the one-sided kernel."""
import ctypes

import numpy as np
import pytest

from conftest import rel_err
from oracle import wall as owall
from rigidmultiblobswall_gb300 import _native
from rigidmultiblobswall_gb300 import mobility as mob

pytestmark = pytest.mark.gpu
TOL = 2e-14  # FP64 sums of 9 x n pairs
A = 0.41


def _blobs(n, seed, side, boxes):
    rng = np.random.default_rng(seed)
    r = np.empty((n, 3))
    r[:, :2] = rng.uniform(-boxes * side, boxes * side, (n, 2))
    r[:, 2] = rng.uniform(0.3 * A, 10 * A, n)
    return r, rng.standard_normal(3 * n)


def _route(mode, n, L):
    out = ctypes.c_int(-1)
    L = np.array(L)
    _native.call("rmw_wall_product_route", 0, {"fp64": 0, "mixed": 1, "df64": 2}[mode], n,
                 L.ctypes.data_as(ctypes.c_void_p), ctypes.byref(out))
    return out.value


@pytest.mark.parametrize("kind", ["uf", "ut", "wf", "wt"])
@pytest.mark.parametrize("n,L,boxes", [(256, (15.0, 17.0, 0.0), 0.5), (257, (15.0, 0.0, 0.0), 3.0),
                                       (513, (0.0, 21.0, 0.0), 0.5), (900, (25.0, 25.0, 0.0), 40.0)])
def test_symmetric_periodic_matches_oracle_and_one_sided(cuda_device, kind, n, L, boxes):
    r, v = _blobs(n, n, max(L), boxes)
    Lv = np.array(L)
    mob.autotune_clear()
    assert _route("fp64", n, L) == 1
    got = mob.wall_product(kind, r, v, 1.0, A, mode="fp64", periodic_length=Lv)
    assert np.array_equal(got, mob.wall_product(kind, r, v, 1.0, A, mode="fp64", periodic_length=Lv))
    mob.autotune_set(kind, n, "fp64", 8)
    try:
        assert rel_err(got, mob.wall_product(kind, r, v, 1.0, A, mode="fp64", periodic_length=Lv)) <= TOL
    finally:
        mob.autotune_clear()
    assert rel_err(got, owall.wall_product(kind, r, v, 1.0, A, periodic_length=Lv)) <= TOL


def test_pairs_half_a_box_apart(cuda_device):
    L = np.array([16.0, 8.0, 0.0])
    g = np.arange(16) * 1.0
    x, y = np.meshgrid(g, g)
    r = np.column_stack([x.ravel(), y.ravel(), 1.0 + 0.01 * np.arange(256)])
    v = np.random.default_rng(0).standard_normal(3 * 256)
    got = mob.wall_product("uf", r, v, 1.0, A, mode="fp64", periodic_length=L)
    assert rel_err(got, owall.wall_product("uf", r, v, 1.0, A, periodic_length=L)) <= TOL


def test_routes(cuda_device):
    mob.autotune_clear()
    assert _route("fp64", 1000, (9.0, 9.0, 9.0)) == 0
    assert _route("df64", 1000, (9.0, 9.0, 0.0)) == 0
    assert _route("fp64", 255, (9.0, 9.0, 0.0)) == 0
