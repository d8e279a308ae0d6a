"""positions_principal = 0: the principal-value window is the one interval from
the node below the pole, and its rest takes rest/width times the window's
samples: none where the pole lies on the node (the quotient fits no int), a
hundred thousand a thousandth of a spacing above it.  On nodes the calls end
and both precisions agree; beside them, and for a relativistic species, the
oracle's values at the parity tests' bounds.
"""
import numpy as np
import pytest

from alps_gb300 import workloads
from test_gpu_parity import _disp_close, _oracle

pytestmark = pytest.mark.gpu

RTOL = 1e-8  # as test_gpu_resonant_forms


def _built(generate):
    w = workloads.proton_electron(24, 48, 1.0, 0.25, 1e-14)
    w["system"].positions_principal = 0
    w["system"].nspec = 1
    w["dists"], w["species"] = w["dists"][:1], w["species"][:1]
    return workloads.build(w, generate)


@pytest.mark.parametrize("n", [1, 31, 700, 2600])
def test_poles_on_nodes(n):
    """At k_par = 0.25 an order's pole moves by 16 spacings of 0.25 and a
    sixteenth of the frequency by one: every pole is on a node."""
    from alps_gb300 import api
    rng = np.random.default_rng(3)
    om = rng.integers(-40, 41, n) / 16.0 + 1j * rng.choice([0.01, 0.05, -0.03], n)
    om[0] = 0.5 + 0.02j
    D = []
    for precision in ("fp64", "mixed"):
        system, species = _built(api.generate_f0)
        G = api.Plasma(system, species, precision=precision)
        G.set_k(1.0, 0.25)
        D.append(G.disp_batch(om))
    assert np.all(np.isfinite(D[0]))
    assert np.all(np.abs(D[1] - D[0]) <= RTOL * np.abs(D[0]))


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_poles_beside_nodes(precision):
    from alps_gb300 import api
    po = _oracle()
    system, species = _built(po.generate_f0)
    O = po.OraclePlasma(system, species)
    G = api.Plasma(system, species, precision=precision)
    G.set_fit(0, O.get_fit(0))
    O.set_k(1.0, 0.25)
    G.set_k(1.0, 0.25)
    for f in (1e-3, 0.03, 0.3, 0.49, 0.51, 0.9):
        for om in ((7 + f) / 16.0 + 0.02j, (11 + f) / 16.0 - 0.02j, (9 + f) / 16.0 + 0.001j):
            _disp_close(O, G, om, "%g %s %s" % (f, om, precision))


def test_relativistic():
    from alps_gb300 import api
    from test_gpu_relativistic import _check_disp, _limit_case, _pair
    sysd, species = _limit_case()
    sysd.positions_principal, sysd.ngamma, sysd.npparbar = 0, 60, 80
    O, G = _pair(api, sysd, species)
    for om in (0.5 + 0.1j, 0.9 - 0.05j):
        _check_disp(O, G, om)
