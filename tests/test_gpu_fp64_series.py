"""The FP64 path's Laurent series and factorised Landau term against the oracle,
at test_gpu_parity's bounds: poles on both sides of the series' line (rho^2 =
0.58, rho the grid's half-width over the pole's distance from its centre), far
poles, a grid off zero, both signs of k_par; continuation fits whose rows share
one Gaussian (factorised) and rows that differ by 1e-3 (summed one by one).
"""
import numpy as np
import pytest

from alps_gb300 import workloads
from test_gpu_parity import _disp_close, _oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kpar,drift", [(0.3, 0.0), (-0.3, 0.0), (0.3, 1.5)])
@pytest.mark.parametrize("rows", ["shared", "uneven"])
def test_series_and_factorised_landau(kpar, drift, rows):
    from alps_gb300 import api
    po = _oracle()
    w = workloads.proton_electron(24, 48, 1.0, kpar, 1e-14)
    if drift:
        w["dists"][0] = workloads._dist(ms=1.0, p_drift=drift)
        w["species"][0].fit_init[0][2] = drift
    system, species = workloads.build(w, po.generate_f0)
    O = po.OraclePlasma(system, species)
    G = api.Plasma(system, species, precision="fp64")
    for i in range(system.nspec):
        fit = O.get_fit(i)
        if rows == "uneven":
            fit = np.array(fit)
            flat = fit.reshape(-1, 5)
            flat[::2, 1] *= 1.0 + 1e-3
            O.set_fit(i, fit)
        G.set_fit(i, fit)
    O.set_k(1.0, kpar)
    G.set_k(1.0, kpar)
    edge = abs(kpar) * 5.75 / np.sqrt(0.58)  # |Re omega| at which the order n = 0 starts its series
    oms = [edge * f + g for f in (0.99, 0.9999, 1.0001, 1.02) for g in (-0.01j, 0.2j)]
    oms += [0.6 - 0.15j, 1.1 + 0.05j, 0.4 + 1j * edge, 25.0 - 0.02j]
    for om in oms:
        _disp_close(O, G, om, "%s kpar=%s %s" % (om, kpar, rows))
