"""GPU: a pinned source split keeps the FP64 and df64 force-torque product on its one-sided pass, whose scratch is
small - the remedy for a caller who holds most of the device."""
import numpy as np
import pytest

from conftest import rel_err
from oracle import wall as owall
from rigidmultiblobswall_gb300 import _native
from rigidmultiblobswall_gb300 import mobility as mob

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["fp64", "df64"])
def test_pinned_split_keeps_the_scratch_small(cuda_device, mode):
    import torch
    n, a = 12000, 0.4  # slots of the symmetric kernel: 94 x 6n doubles, 54 MB; the one-sided pass: 13 x 6n, 7.5 MB
    rng = np.random.default_rng(5)
    r = np.empty((n, 3))
    r[:, :2] = rng.uniform(0, 2.5 * a * np.sqrt(n), (n, 2))
    r[:, 2] = rng.uniform(0.4 * a, 9 * a, n)
    F, T = rng.standard_normal(3 * n), rng.standard_normal(3 * n)
    rows = rng.choice(n, 30, replace=False)
    U0, W0 = owall.force_torque(r, F, T, 1.0, a, rows=rows)
    pick = lambda x: x.cpu().numpy().reshape(-1, 3)[rows].reshape(-1)  # noqa: E731
    dev = [torch.tensor(x, device="cuda") for x in (r, F, T)]

    def product():
        """The product and the device memory that it took."""
        mob.wall_force_torque(*dev, 1.0, a, mode="mixed")  # the outputs' and the library's own first allocations
        torch.cuda.synchronize()
        _native.release_scratch()
        free = torch.cuda.mem_get_info()[0]
        U, W = mob.wall_force_torque(*dev, 1.0, a, mode=mode)
        torch.cuda.synchronize()
        assert rel_err(pick(U), U0) <= 1e-12 and rel_err(pick(W), W0) <= 1e-12
        return free - torch.cuda.mem_get_info()[0]

    mob.autotune_clear()
    try:
        assert product() > 40 << 20
        for pinned in (["uf", "ut", "wf", "wt"], ["wf"]):
            mob.autotune_clear()
            for kind in pinned:
                mob.autotune_set(kind, n, mode, 8)
            assert product() < 24 << 20
    finally:
        mob.autotune_clear()
        _native.release_scratch()
