"""GPU: blob-blob forces component by component where a blob's largest terms vanish in one component - stacked blobs,
a layer of equal heights, rows - and only blobs many Debye lengths further away push there."""
import numpy as np
import pytest

from rigidmultiblobswall_gb300 import forces as F

pytestmark = pytest.mark.gpu
EPS, B, A = 0.7, 0.05, 0.4


def _check(r, L=(0.0, 0.0, 0.0), **kw):
    L = np.array(L)
    got = F.calc_blob_blob_forces_pycuda(r, periodic_length=L, repulsion_strength=EPS, debye_length=B, blob_radius=A,
                                         **kw).reshape(-1, 3)
    d = r[None, :, :] - r[:, None, :]
    for k in range(3):
        if L[k] > 0:
            d[..., k] -= L[k] * np.trunc(d[..., k] / L[k] + 0.5 * np.sign(d[..., k]))
    rn = np.linalg.norm(d, axis=2)
    g = np.where(rn > 2 * A, np.exp(-np.maximum(rn - 2 * A, 0) / B), 1.0) * EPS / B
    t = (np.where(rn > 0, g, 0.0) / np.where(rn > 0, rn, 1.0))[..., None] * d
    mag = np.abs(t).sum(axis=1)
    # every component against the sum of its own terms: each carries the rounding of its exponent (2^-53 r / b, at
    # most 750 of them) and the sum n more; subnormal terms carry their own
    assert (np.abs(got + t.sum(axis=1)) <= 2e-13 * mag + 1e-300).all()
    return mag


def _columns(gap):
    """Two stacks of four blobs, `gap` apart: all x and y forces come from the other stack."""
    z = 1.0 + 0.9 * np.arange(4)
    c = np.column_stack([np.zeros(4), np.zeros(4), z])
    return np.vstack([c, c + [gap, 0.3 * gap, 0.2]])


@pytest.mark.parametrize("gap", [2.0, 5.0, 12.0, 25.0])
def test_stacked_blobs(cuda_device, gap):
    mag = _check(_columns(gap))
    assert mag[0, 0] > 0 or gap > 20
    _check(_columns(gap)[np.random.default_rng(1).permutation(8)])


def test_stacks_among_others(cuda_device):
    """Stacks in a suspension of several thousand blobs, next to blobs with ordinary neighbours."""
    rng = np.random.default_rng(4)
    r = np.column_stack([rng.uniform(0, 60, 2000), rng.uniform(0, 60, 2000), rng.uniform(0.5, 6, 2000)])
    for k in range(6):
        r[8 * k:8 * k + 8] = _columns(6.0) + [100.0 + 20 * k, -40.0, 0.0]
    _check(r)
    _check(r[rng.permutation(2000)], L=(300.0, 290.0, 0.0))


@pytest.mark.parametrize("heights", [1, 2])
def test_layers(cuda_device, heights):
    """A square layer at one height (no z force at all), or two layers many Debye lengths apart."""
    x, y = np.meshgrid(0.85 * np.arange(20), 0.9 * np.arange(20))
    layer = np.column_stack([x.ravel(), y.ravel(), np.full(x.size, 1.5)])
    r = layer if heights == 1 else np.vstack([layer, layer + [0.1, 0.2, 4.0]])
    _check(r)
    got = F.calc_blob_blob_forces_pycuda(layer, repulsion_strength=EPS, debye_length=B, blob_radius=A).reshape(-1, 3)
    assert not got[:, 2].any()
