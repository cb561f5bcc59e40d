"""GPU: the blob-blob forces' FP32 candidate screen and source chunks against the oracle, blob by blob: Debye
lengths for which most terms vanish beside the nearest blob's, isolated blobs whose only terms are 1e-300 of
contact, coincident blobs, boxes much larger and units much smaller than a blob, images, and a captured call."""
import numpy as np
import pytest

from oracle import forces as of
from rigidmultiblobswall_gb300 import forces as F

pytestmark = pytest.mark.gpu
# per blob, relative to the sum of its terms' magnitudes: each term carries the rounding of its exponent
# (2^-53 r/b, at most 750 of them) and the sum n more
TOL = 2e-13


def _check(r, eps, b, a, L=None, got=None):
    L = np.zeros(3) if L is None else np.asarray(L, dtype=float)
    ref = of.blob_blob_forces(r, eps, b, a, periodic_length=L)
    if got is None:
        got = F.calc_blob_blob_forces_pycuda(r, periodic_length=L, repulsion_strength=eps, debye_length=b, blob_radius=a)
    assert np.isfinite(got).all()
    d = r[None, :, :] - r[:, None, :]
    for k in range(3):
        if L[k] > 0:
            d[..., k] -= L[k] * np.trunc(d[..., k] / L[k] + 0.5 * np.sign(d[..., k]))
    rn = np.linalg.norm(d, axis=2)
    g = np.where(rn > 0, np.where(rn > 2 * a, np.exp(-np.maximum(rn - 2 * a, 0) / b), 1.0), 0.0) * eps / b
    mag = g.sum(axis=1)
    err = np.linalg.norm(got - ref, axis=1)
    assert (err <= TOL * mag + 1e-300 * eps / b).all(), (err / np.maximum(mag, 1e-320)).max()


def _slab(n, seed, side, h):
    rng = np.random.default_rng(seed)
    return np.column_stack([rng.uniform(0, side, n), rng.uniform(0, side, n), rng.uniform(0.5, h, n)])


@pytest.mark.parametrize("n", [1, 2, 127, 129, 257, 700, 1100])
@pytest.mark.parametrize("b", [0.004, 0.04, 0.4, 4.0])
def test_screened_forces_match_oracle(cuda_device, n, b):
    _check(_slab(n, n, 1.2 * np.sqrt(n), 4.0), 0.7, b, 0.4)


@pytest.mark.parametrize("L", [(11.0, 0.0, 0.0), (9.0, 13.0, 0.0), (8.0, 9.0, 7.0)])
@pytest.mark.parametrize("b", [0.03, 0.5])
def test_screened_periodic_forces_match_oracle(cuda_device, L, b):
    r = _slab(515, 3, 60.0, 6.0)  # coordinates several boxes wide
    _check(r, 0.7, b, 0.4, L)


def test_isolated_and_coincident_blobs(cuda_device):
    """A pair 600 Debye lengths apart, coincident blobs (no force between them, but from the others), a blob
    beyond every exponent."""
    r = _slab(300, 5, 15.0, 4.0)
    r[10] = r[20]
    r[30] = [500.0, 500.0, 3.0]
    r[31] = [506.8, 500.0, 3.0]
    r[40] = r[41] = [900.0, 0.0, 3.0]
    r[42] = [903.0, 0.0, 3.0]
    _check(r, 0.7, 0.01, 0.4)


@pytest.mark.parametrize("unit", [2.0 ** -80, 2.0 ** -30, 2.0 ** 40])
def test_units_of_length(cuda_device, unit):
    """Lengths in other units (a power of two: exact) with eps / b unchanged give the same forces."""
    r = _slab(400, 8, 20.0, 4.0)
    got = F.calc_blob_blob_forces_pycuda(r * unit, repulsion_strength=0.7 * unit, debye_length=0.05 * unit,
                                         blob_radius=0.4 * unit)
    _check(r, 0.7, 0.05, 0.4, got=got)


def test_far_box_and_accumulate(cuda_device):
    """Blobs 3e6 radii from the origin and from each other: the screen's error bound exceeds every distance."""
    rng = np.random.default_rng(9)
    r = _slab(600, 9, 30.0, 4.0)
    r[::3, 0] += 1.2e6
    r[1::3, 1] -= 9e5
    _check(r[rng.permutation(600)], 0.7, 0.1, 0.4)


def test_captured_forces_match_oracle(cuda_device):
    """Inside a capture nothing may be allocated: one chunk, the fixed radius."""
    import torch
    r = _slab(600, 11, 30.0, 4.0)
    rt = torch.tensor(r, device=cuda_device)
    kw = dict(repulsion_strength=0.7, debye_length=0.05, blob_radius=0.4)
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        F.calc_blob_blob_forces_pycuda(rt, **kw)
    side.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=side):
        out = F.calc_blob_blob_forces_pycuda(rt, **kw)
    graph.replay()
    torch.cuda.synchronize()
    _check(r, 0.7, 0.05, 0.4, got=out.cpu().numpy())


@pytest.mark.parametrize("n", [6000, 6001, 11000, 11003])
@pytest.mark.parametrize("b,L", [(0.02, 0.0), (0.2, 70.0)])
def test_tile_widths_and_distant_nearest_blobs(cuda_device, n, b, L):
    """Every tile width against an FP64 sum over all pairs; blobs in random order, so that the nearest blob is
    seldom among the sources next to it in memory."""
    import torch
    r = torch.tensor(_slab(n, n, 1.2 * np.sqrt(n), 4.0), device=cuda_device)
    a, eps = 0.4, 0.7
    got = F.calc_blob_blob_forces_pycuda(r, periodic_length=np.array([L, L, 0.0]), repulsion_strength=eps,
                                         debye_length=b, blob_radius=a).reshape(-1, 3)
    ref, mag = torch.zeros_like(r), torch.zeros(n, dtype=torch.float64, device=cuda_device)
    for i in torch.arange(n, device=cuda_device).split(1000):
        d = r[None] - r[i, None]
        if L > 0:
            d[..., :2] -= L * torch.trunc(d[..., :2] / L + 0.5 * torch.sign(d[..., :2]))
        rn = d.norm(dim=2)
        g = torch.where(rn > 0, torch.exp(-(rn - 2 * a).clamp(min=0) / b), torch.zeros_like(rn)) * eps / b
        mag[i] = g.sum(1)
        ref[i] = -(g / rn.clamp(min=1e-300))[..., None].mul(d).sum(1)
    assert (((got - ref).norm(dim=1)) <= TOL * mag + 1e-300).all()
