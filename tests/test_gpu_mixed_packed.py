"""GPU: the mixed symmetric M_UF kernel with two targets per thread against the oracle at the edges of its tiles:
sizes around multiples of 64 and 128, overlapping blobs in one packed lane and not in the other, blobs on the
wall, and several suspensions of such sizes at once."""
import numpy as np
import pytest

from conftest import rel_err
from oracle import wall as owall
from rigidmultiblobswall_gb300 import mobility as mob

pytestmark = pytest.mark.gpu
TOL = 1e-6  # the mode's bar


def _blobs(n, seed, a):
    rng = np.random.default_rng(seed)
    r = np.empty((n, 3))
    r[:, :2] = rng.uniform(0, 2.0 * a * np.sqrt(n), (n, 2))
    r[:, 2] = rng.uniform(0.0, 10 * a, n)
    k = np.arange(1, n, 4)  # every fourth blob overlaps its predecessor
    r[k] = r[k - 1] + rng.uniform(0.2, 0.9, (k.size, 3)) * a
    return r, rng.standard_normal(3 * n)


@pytest.mark.parametrize("n", [256, 257, 319, 320, 321, 383, 385, 449, 1153])
def test_mixed_tiles_match_oracle(cuda_device, n):
    a = 0.4
    r, v = _blobs(n, n, a)
    mob.autotune_clear()
    mob.autotune_set("uf", n, "mixed", -1)
    try:
        got = mob.wall_product("uf", r, v, 1.0, a, mode="mixed")
        again = mob.wall_product("uf", r, v, 1.0, a, mode="mixed")
    finally:
        mob.autotune_clear()
    assert rel_err(got, owall.wall_product("uf", r, v, 1.0, a)) <= TOL
    assert np.array_equal(got, again)


def test_mixed_batch_of_tile_edges_matches_oracle(cuda_device):
    import torch
    a, sizes = 0.4, [1, 63, 64, 65, 127, 129, 200, 321]
    off = np.concatenate([[0], np.cumsum(sizes)])
    parts = [_blobs(m, m, a) for m in sizes]
    r, v = np.concatenate([p[0] for p in parts]), np.concatenate([p[1] for p in parts])
    got = mob.SuspensionBatch(off).product("uf", torch.tensor(r, device="cuda"), torch.tensor(v, device="cuda"), 1.0, a,
                                           mode="mixed").cpu().numpy()
    for k, m in enumerate(sizes):
        ref = owall.wall_product("uf", *parts[k], 1.0, a)
        assert rel_err(got[3 * off[k]:3 * off[k + 1]], ref) <= TOL
