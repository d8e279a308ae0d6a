"""Principal-value windows of many nodes (positions_principal has no upper
limit but the grid's): the window's pieces and weights are held on the chip up
to 48 nodes to a side, wider ones are summed sample by sample, and beyond 128
a relativistic row takes its pieces in parts.  Against the oracle at the bounds
of the parity tests.
"""
import numpy as np
import pytest

from alps_gb300 import workloads
from test_gpu_parity import _disp_close, _oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("M_I,M_P", [(48, 100), (49, 300), (128, 100), (370, 100)])
def test_wide_window(precision, M_I, M_P):
    from alps_gb300 import api
    po = _oracle()
    w = workloads.proton_electron(8, 2 * M_I + 61, 1.0, 0.3, 1e-9)
    w["system"].positions_principal = M_I
    w["system"].n_resonance_interval = M_P
    system, species = workloads.build(w, po.generate_f0)
    O = po.OraclePlasma(system, species)
    G = api.Plasma(system, species, precision=precision)
    for i in range(system.nspec):
        G.set_fit(i, O.get_fit(i))
    O.set_k(1.0, 0.3)
    G.set_k(1.0, 0.3)
    for om in (0.05 - 0.01j, -0.02 + 0.03j, 0.011 + 0.001j, 0.03 - 0.1j):
        _disp_close(O, G, om, "%s M_I %d %s" % (om, M_I, precision))


@pytest.mark.parametrize("M_I", [128, 136, 316])
def test_wide_relativistic_window(M_I):
    from alps_gb300 import api
    from test_gpu_relativistic import _check_disp, _limit_case, _pair
    sysd, species = _limit_case(N=4, M=2 * M_I + 8)
    sysd.positions_principal, sysd.ngamma, sysd.npparbar = M_I, 24, 8 * M_I
    sysd.kpar = 0.2
    O, G = _pair(api, sysd, species)
    for om in (0.2 + 0.02j, 0.21 + 0.05j, 0.205 - 0.01j):
        _check_disp(O, G, om)
