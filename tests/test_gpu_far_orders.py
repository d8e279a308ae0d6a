"""Orders beyond a frequency's reach as one power series in omega, from 25000
warps of orders on, against batches below that line (order by order).

Both sum the same terms; each double-float sum is within 2^-40 of its terms'
magnitudes, each FP64 sum within 2^-48, and det D loses up to four digits to
cancellation: 1e-8 and 1e-10 of |D|.  The frequencies range from zero to past
the series' last level, above and below the axis; grids at and off zero, both
signs of k_par.
"""
import numpy as np
import pytest

from alps_gb300 import workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,rtol", [("fp64", 1e-10), ("mixed", 1e-8)])
@pytest.mark.parametrize("kpar,drift,npar", [(0.3, 0.0, 48), (-0.3, 0.0, 51), (0.2, 1.5, 48), (0.02, 0.0, 60)])
def test_far_series_and_single_orders(precision, rtol, kpar, drift, npar):
    from alps_gb300 import api
    w = workloads.proton_electron(24, npar, 3.0, kpar, 1e-20)
    if drift:
        w["dists"][0] = workloads._dist(ms=1.0, p_drift=drift)
        w["species"][0].fit_init[0][2] = drift
    system, species = workloads.build(w, api.generate_f0)
    G = api.Plasma(system, species, precision=precision)
    G.set_k(3.0, kpar)
    orders = sum(2 * n + 1 for n in G.nmax())
    rng = np.random.default_rng(8)
    n = 25000 * 32 // orders + 64
    om = rng.uniform(-1, 1, n) * 10.0 ** rng.uniform(-3, 1.3, n) + 1j * abs(kpar) * rng.choice([-0.6, -0.05, 0.03, 1.0], n)
    om[:7] = [1e-6j, 3.0 + 0.01j, -3.0 + 0.01j, 8.0 + 0.1j, 30.0 + 0.1j, 0.5 + 2.0j, 0.01 + 9.0j]
    large = G.disp_batch(om)
    small = np.concatenate([G.disp_batch(om[i:i + 1000]) for i in range(0, n, 1000)])
    err = np.abs(large - small) / np.abs(small)
    assert np.all(err <= rtol), (np.nanmax(err), om[np.nanargmax(err)])
    assert np.array_equal(large, G.disp_batch(om))
