"""Resonant orders of a mixed batch: one item per lane from 2560 frequencies
on, one item per warp below.

Both forms, and the FP64 path, sum the same samples.  Each double-float sum
is within 2^-40 of its terms' magnitudes; with four digits lost to the
cancellation in det D that is 1e-8 of |D|.  The frequencies put poles over
the whole grid and past both ends, on nodes, half-way between nodes, and on
both sides of the analytic branch's limit in Im(p).
"""
import numpy as np
import pytest

from alps_gb300 import workloads

pytestmark = pytest.mark.gpu

RTOL = 1e-8


def _frequencies(n, kpar, npar):
    rng = np.random.default_rng(7)
    im = rng.choice([-0.3, -0.05, -0.011, -0.002, 0.002, 0.05, 0.4], n) * abs(kpar) / 0.3
    om = rng.uniform(-2.6, 2.6, n) + 1j * im
    # poles of the protons' orders -1, 0, 1 on nodes and half-way (p = -6 + 12 j / npar)
    half = rng.integers(1, 2 * npar, n // 8)
    om.real[:len(half)] = kpar * (-6.0 + 6.0 * half / npar) + rng.integers(-1, 2, len(half))
    return om


@pytest.mark.parametrize("kpar,npar,M_I,M_P", [
    (0.3, 48, 3, 100), (-0.3, 51, 3, 100), (0.3, 51, 1, 127), (0.3, 48, 5, 16),
    (0.7, 48, 2, 1), (0.3, 48, 6, 100), (0.3, 51, 3, 128), (-0.3, 20, 5, 30)])
def test_lane_and_warp_forms(kpar, npar, M_I, M_P):
    from alps_gb300 import api
    w = workloads.proton_electron(24, npar, 1.0, kpar, 1e-12)
    w["system"].positions_principal = M_I
    w["system"].n_resonance_interval = M_P
    system, species = workloads.build(w, api.generate_f0)
    om = _frequencies(2561, kpar, npar)
    D = {}
    for precision in ("mixed", "fp64"):
        G = api.Plasma(system, species, precision=precision)
        G.set_k(1.0, kpar)
        D[precision, "large"] = G.disp_batch(om)
        D[precision, "small"] = np.concatenate([G.disp_batch(om[i:i + 500]) for i in range(0, len(om), 500)])
    ref = D["fp64", "small"]
    for key, d in D.items():
        err = np.abs(d - ref) / np.abs(ref)
        assert np.all(err <= RTOL), (key, np.nanmax(err), om[np.nanargmax(err)])
