"""Kappa continuation rows, whose three points share one complex power where
the spacing is small against the local scale (disp_kernels.cu eval_fit3_d),
against the oracle at test_gpu_parity's bounds: spacings on both sides of that
line (npar 16: beyond, 48 and 96: within), small and large kappa, a kappa term
beside a Maxwellian one in a species, shallow to strong damping, and a pole
past the point where z's real part turns negative.
"""
import numpy as np
import pytest

from alps_gb300 import _abi, workloads
from test_gpu_parity import _disp_close, _oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("npar,kappa,two", [(16, 3.0, False), (48, 8.0, False), (96, 3.0, False), (48, 4.0, True)])
def test_kappa_rows(precision, npar, kappa, two):
    from alps_gb300 import api
    po = _oracle()
    sysd = _abi.system_defaults(
        nspec=2, nperp=24, npar=npar, kperp=1.0, kpar=0.4, vA=1e-4, Bessel_zero=1e-9, secant_method=2, numiter=50,
        kperp_norm=1, D_threshold=1e-15, positions_principal=3, n_resonance_interval=100, Tlim=0.01)
    species = []
    for ms, qs, kind in ((1.0, 1.0, 2), (1.0 / 1836.0, -1.0, 1)):
        d = workloads._dist(kind=kind, ms=ms, kappa=kappa, kappa1=kappa)
        pp, pl, f0, ideal = po.generate_f0(d, 24, npar)
        fits = [(kind, list(ideal[:5]), ideal[5])]
        if two and kind == 2:
            fits.append((1, [0.01 * ideal[0], 1.0 / ms, 0.3, 0.0, 0.0], 1.0 / ms))
        species.append((_abi.species_defaults(ns=1.0, qs=qs, ms=ms, fits=fits), pp, pl, f0))
    O = po.OraclePlasma(sysd, species)
    G = api.Plasma(sysd, species, precision=precision)
    for i in range(2):
        G.set_fit(i, O.get_fit(i))
    O.set_k(1.0, 0.4)
    G.set_k(1.0, 0.4)
    for om in [0.5 - 0.001j, 0.9 - 0.1j, 1.4 - 0.4j, 0.2 - 0.02j, 1.0 - 0.9j]:
        _disp_close(O, G, om, "%s npar=%d kappa=%g" % (om, npar, kappa))
