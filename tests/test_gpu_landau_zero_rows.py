"""A continuation fit with a row of amplitude zero: landau_integrate returns
nothing where the continuation of a row is exactly zero (src/ALPS_fns.f90:
1380-1400), so the whole Landau term is zero, in either precision and on
either form of the term; row 0 takes no part in that test and leaves it.
Against the oracle at test_gpu_parity's bounds.
"""
import numpy as np
import pytest

from alps_gb300 import workloads
from test_gpu_parity import _disp_close, _oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("row", [0, 1, 11, 24])
@pytest.mark.parametrize("rows", ["shared", "uneven"])
def test_zero_row(precision, row, rows):
    from alps_gb300 import api
    po = _oracle()
    w = workloads.proton_electron(24, 48, 1.0, 0.3, 1e-14)
    system, species = workloads.build(w, po.generate_f0)
    O = po.OraclePlasma(system, species)
    G = api.Plasma(system, species, precision=precision)
    for i in range(system.nspec):
        fit = np.array(O.get_fit(i))
        flat = fit.reshape(-1, 5)
        if rows == "uneven":
            flat[::2, 1] *= 1.0 + 1e-3
        flat[row, 0] = 0.0
        O.set_fit(i, fit)
        G.set_fit(i, fit)
    O.set_k(1.0, 0.3)
    G.set_k(1.0, 0.3)
    for om in (0.6 - 0.15j, 0.3 + 0j, 1.2 - 0.02j, 0.8 + 0.1j):
        _disp_close(O, G, om, "%s row %d %s %s" % (om, row, rows, precision))
