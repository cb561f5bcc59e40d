"""GPU: df64 wall products of suspensions as wide and as high above the wall as 10^7 to 10^10 radii, where s^5 of the
distance to an image leaves the range of FP32, against the oracle: symmetric kernels, the one-sided one (200 blobs)
and the force-torque product.  Forces act on every other blob and the velocities of the others are compared: their own
terms, eight to ten orders larger, do not enter."""
import numpy as np
import pytest

from oracle import wall as owall
from rigidmultiblobswall_gb300 import mobility as mob

pytestmark = pytest.mark.gpu
A = 1.0


def _blobs(n, scale):
    rng = np.random.default_rng(n)
    v = rng.standard_normal((n, 3))
    v[1::2] = 0.0
    return rng.uniform(0.4, 1.6, (n, 3)) * scale, v.reshape(-1)


def _check(got, ref):
    got, ref = (np.asarray(x).reshape(-1, 3)[1::2] for x in (got, ref))
    assert np.linalg.norm(got - ref) <= 1e-12 * np.linalg.norm(ref)  # the documented bar of the mode


@pytest.mark.parametrize("n", [200, 300, 1000])
@pytest.mark.parametrize("scale", [1e7, 1e9, 1e10])
def test_forces_far_from_the_wall(cuda_device, n, scale):
    r, v = _blobs(n, scale)
    _check(mob.wall_product("uf", r, v, 1.0, A, mode="df64"), owall.wall_product("uf", r, v, 1.0, A))


@pytest.mark.parametrize("kind", ["ut", "wf"])
@pytest.mark.parametrize("n", [300, 1000])
def test_rotations_far_from_the_wall(cuda_device, kind, n):
    r, v = _blobs(n, 1e7)
    _check(mob.wall_product(kind, r, v, 1.0, A, mode="df64"), owall.wall_product(kind, r, v, 1.0, A))


def test_force_torque_far_from_the_wall(cuda_device):
    r, F = _blobs(300, 1e9)
    _check(mob.wall_force_torque(r, F, 0.0 * F, 1.0, A, mode="df64")[0], owall.force_torque(r, F, 0.0 * F, 1.0, A)[0])


@pytest.mark.parametrize("n", [200, 300])
@pytest.mark.parametrize("kind", ["uf", "ut", "wf", "wt"])
def test_parked_blobs(cuda_device, kind, n):
    """Blobs moved out of the way, 10^16 radii up and aside, leave the others' product as it is."""
    rng = np.random.default_rng(n)
    r = np.column_stack([rng.uniform(0, 60, n), rng.uniform(0, 60, n), rng.uniform(1.0, 9.0, n)])
    r[::7] = rng.uniform(0.5, 1.5, (r[::7].shape[0], 3)) * 1e16
    v = rng.standard_normal(3 * n)
    got = np.asarray(mob.wall_product(kind, r, v, 1.0, A, mode="df64"))
    ref = owall.wall_product(kind, r, v, 1.0, A)
    assert np.linalg.norm(got - ref) <= 1e-12 * np.linalg.norm(ref)
