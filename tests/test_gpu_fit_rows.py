"""The continuation fit on the device against the oracle's, at the sizes where
its row loop changes form: rows shorter and longer than a warp and than a
block, an odd number of points, and a fit whose points do not fit in shared
memory; the exponential-free form of one Maxwellian in log space and the
general form (bi-kappa, two terms, linear space), from seeds off the table's
own parameters.  Parameters agree to 1e-10 of the largest, the gate of the
other fit tests: both stop at the same iteration, where the last step is far
below it.
"""
import os

import numpy as np
import pytest

from alps_gb300 import _abi

pytestmark = pytest.mark.gpu

FIT_RTOL = 1e-10


def _table(kind, nperp, npar):
    """(pperp, ppar, f0, fits, log_fit) of one proton species."""
    pp = np.arange(nperp + 1) * (4.0 / nperp)
    pz = np.arange(npar + 1) * (8.0 / npar) - 4.0
    a, b = np.meshgrid(pp, pz, indexing="ij")
    norm = np.pi ** -1.5
    maxw = norm * np.exp(-a * a - b * b)
    if kind == "maxwellian":
        return a, b, maxw, [(1, [1.03 * norm, 1.02, 0.01, 0, 0], 1.0)], 1
    if kind == "linear":
        return a, b, maxw, [(1, [1.03 * norm, 1.02, 0.01, 0, 0], 1.0)], 0
    if kind == "kappa":
        kap, a2 = 5.0, 0.7
        f = 0.2 * (1.0 + b * b / (kap * a2) + a * a / (kap * a2)) ** (-1.0 - kap)
        return a, b, f, [(2, [0.201, 1.01 / (kap * a2), 0.002, -1.0 - kap, 1.0], 1.0 / (kap * a2))], 1
    beam = 0.1 * norm * np.exp(-a * a - 4.0 * (b - 2.0) ** 2)
    return a, b, maxw + beam, [(1, [1.01 * norm, 1.01, 0.005, 0, 0], 1.0),
                               (1, [0.101 * norm, 4.02, 2.005, 0, 0], 1.0)], 1


@pytest.mark.parametrize("kind,nperp,npar", [("maxwellian", 5, 30), ("maxwellian", 7, 33), ("maxwellian", 5, 255),
                                             ("maxwellian", 4, 601), ("linear", 5, 64), ("kappa", 5, 48),
                                             ("kappa", 4, 1500), ("two", 5, 96), ("two", 4, 1301)])
def test_fit_rows_match_oracle(kind, nperp, npar):
    from alps_gb300 import api
    from oracle import pyoracle as po
    po.set_threads(os.cpu_count() or 1)
    a, b, f, fits, log_fit = _table(kind, nperp, npar)
    system = _abi.system_defaults(nspec=1, nperp=nperp, npar=npar, kperp=0.5, kpar=0.2, vA=1e-4, Bessel_zero=1e-6)
    sp = _abi.species_defaults(ns=1.0, qs=1.0, ms=1.0, fits=fits, log_fit=log_fit)
    species = [(sp, a.ravel(), b.ravel(), f.ravel())]
    want = po.OraclePlasma(system, species).get_fit(0)
    got = api.Plasma(system, species).get_fit(0)
    assert np.all(np.isfinite(want))
    assert np.abs(got - want).max() <= FIT_RTOL * np.abs(want).max()
