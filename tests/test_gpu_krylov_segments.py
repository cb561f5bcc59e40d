"""GPU: the fused Krylov step kernels over segment layouts with many jobs per CTA and with a single one.

A CTA of the step kernels keeps the segment ranges of its first eight jobs in shared memory and reads the
others' from global memory; norms, Givens rotations and the tridiagonal eigen-problem use a reciprocal
square root inside the mid exponent range and the library's functions outside it (a zero segment's norm).
The host-driven loops do the same algorithms with one host round trip per step."""
import numpy as np
import pytest

from conftest import rel_err
from rigidmultiblobswall_gb300 import _native
from rigidmultiblobswall_gb300.rigid import RigidSystem

pytestmark = pytest.mark.gpu

TETRA = np.array([[1.0, 1.0, 1.0], [1.0, -1.0, -1.0], [-1.0, 1.0, -1.0], [-1.0, -1.0, 1.0]]) / np.sqrt(3.0)


# bodies per suspension; 18 unknowns a body, 256 or more per CTA: up to 14 jobs of a CTA in the first layout
@pytest.mark.parametrize("counts", [[1] * 40 + [2] * 5, [1, 1, 30, 1, 2, 1, 1, 1, 1, 1, 1, 3, 1, 1], [2]])
def test_many_segments_per_cta_match_host_loop(cuda_device, counts):
    nb = sum(counts)
    rng = np.random.default_rng(100 + nb)
    x = np.stack([3.0 * (np.arange(nb) % 7), 3.0 * (np.arange(nb) // 7), rng.uniform(1.5, 4.0, nb)], axis=1)
    r = (x[:, None, :] + TETRA[None]).reshape(-1, 3)
    s = RigidSystem([4] * nb, 1.0, 0.3)
    s.set_configuration(r, x)
    s.set_suspensions(counts)
    s.build_pc(stochastic=True)
    rhs = rng.standard_normal(s.size)
    Z = rng.standard_normal((3, 3 * s.n_blobs))
    Z[1, :12 * counts[0]] = 0.0  # a zero segment
    out = {}
    try:
        for dev in (True, False):
            _native.use_device_krylov(dev)
            sol, it, rr, stt = s.solve_batched(rhs, tol=1e-10, mode="fp64")
            noise, itl = s.lanczos_batched(Z, factor=1.0, tol=1e-4, mode="fp64")
            assert (np.asarray(stt) == 0).all() and (np.asarray(rr) <= 1e-10).all()
            out[dev] = (sol.cpu().numpy(), np.asarray(it), noise.cpu().numpy(), np.asarray(itl))
    finally:
        _native.use_device_krylov(True)
    d, h = out[True], out[False]
    # both residuals are below 1e-10 and the preconditioned operator's condition number below 50
    assert rel_err(d[0], h[0]) <= 1e-8
    # the same few iterations of a reorthogonalised recurrence: rounding errors only
    assert (d[3] == h[3]).all()
    assert rel_err(d[2], h[2]) <= 1e-10
    assert not d[2][1, :12 * counts[0]].any()
