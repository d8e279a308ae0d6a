"""A p_par grid of 8000 intervals whose spacings differ by the 1e-9 that
alps_set_species accepts: the first spacings leave the last nodes 1.4e-5 of a
spacing off their uniform places, more than the distance to a node from which
a resonance momentum's place used to be taken as settled.  Resonances just
beside a node and a half-way point near the grid's end, against the oracle at
test_gpu_parity's bounds.
"""
import numpy as np
import pytest

from alps_gb300 import _abi
from test_gpu_parity import _disp_close, _oracle

pytestmark = pytest.mark.gpu

N, M, KPAR = 4, 8000, 0.3


def _species():
    d = 12.0 / M
    step = np.full(M, d * (1.0 + 0.9e-9))
    step[0], step[1] = d, d * (1.0 - 0.9e-9)
    pz = -11.5 + np.concatenate([[0.0], np.cumsum(step)])
    pp = np.arange(N + 1) * 1.5
    f0 = np.pi ** -1.5 * np.exp(-pz[None, :] ** 2 - pp[:, None] ** 2)
    sysd = _abi.system_defaults(nspec=1, nperp=N, npar=M, kperp=0.5, kpar=KPAR, vA=1e-4, Bessel_zero=1e-4,
                                kperp_norm=1, positions_principal=3, n_resonance_interval=100, Tlim=0.01)
    sp = _abi.species_defaults(ns=1.0, qs=1.0, ms=1.0, fits=[(1, [np.pi ** -1.5, 1.0, 0, 0, 0], 1.0)])
    return sysd, [(sp, np.repeat(pp, M + 1), np.tile(pz, N + 1), f0.ravel())], pz


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_beside_nodes_and_half_way_points(precision):
    from alps_gb300 import api
    sysd, species, pz = _species()
    O = _oracle().OraclePlasma(sysd, species)
    G = api.Plasma(sysd, species, precision=precision)
    G.set_fit(0, O.get_fit(0))
    O.set_k(0.5, KPAR)
    G.set_k(0.5, KPAR)
    dp = pz[1] - pz[0]
    for j in (7700, 7900, 7950):
        for place in (0.0, 0.5):
            for off in (-3e-6, 3e-6, -1.2e-5, 1.2e-5):
                om = (pz[j] + (place + off) * dp) * KPAR - 0.02j
                _disp_close(O, G, om, "node %d + %g %s" % (j, place + off, precision))
