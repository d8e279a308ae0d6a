"""Small batches in one launch against the separate kernels.

Profiling needs the kernels apart, so a context with profiling on takes them.
Both forms sum the same terms in the same order: det D, the tensors and the
fields agree to 1e-13 of their size (a few rounding errors: the compiler may
contract a product differently in each kernel), whatever the batch size, and
calls in a row agree bit for bit (the counters return to zero).
"""
import numpy as np
import pytest

from alps_gb300 import workloads

pytestmark = pytest.mark.gpu

OMS = np.array([0.45 - 0.2j, 1.3 - 0.004j, 0.9 + 0.003j, 0.7 + 0.0j, 2.2 - 0.35j, 0.05 + 0.1j, -1.1 - 0.02j])
RTOL = 1e-13


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("kpar", [0.3, -0.05])
def test_one_launch_and_many(precision, kpar):
    from alps_gb300 import api
    w = workloads.proton_electron(24, 51, 1.0, kpar, 1e-14)
    system, species = workloads.build(w, api.generate_f0)
    G = api.Plasma(system, species, precision=precision)
    G.set_k(1.0, kpar)
    for n in [1, 2, 5, 31, 32, 64, 65, 130, 300]:
        om = np.resize(OMS, n)
        one = G.disp_batch(om)
        assert G.stats().kernels_launched == 1 or n > 64
        assert np.array_equal(one, G.disp_batch(om))
        G.set_profiling(True)
        many = G.disp_batch(om)
        assert G.stats().kernels_launched > 1
        G.set_profiling(False)
        assert np.all(np.abs(one - many) <= RTOL * np.abs(many)), (n, np.abs(one / many - 1).max())
    for om in OMS:
        one = G.disp(om)
        G.set_profiling(True)
        many = G.disp(om)
        G.set_profiling(False)
        for a, b in zip(one, many):
            a, b = np.asarray(a), np.asarray(b)
            assert np.all(np.abs(a - b) <= RTOL * np.abs(b).max())
