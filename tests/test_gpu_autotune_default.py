"""GPU: the time that autotuning reports for the built-in rule is that of the kernel which an untuned product runs."""
import pytest

from rigidmultiblobswall_gb300 import mobility as mob

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,mode,n", [("uf", "df64", 2048), ("uf", "fp64", 1000), ("wt", "df64", 5003),
                                         ("uf", "mixed", 20000)])
def test_default_time_is_the_rules(cuda_device, kind, mode, n):
    mob.autotune_clear()
    res = mob.autotune(kind, n, mode, reps=3)
    mob.autotune_clear()
    # the rule takes the symmetric kernel at these sizes, which is also the fastest: one measurement, reported twice
    assert res["nchunks"] == -1
    assert res["default_ms"] == res["ms"]
