"""Mixed batches around 2560 frequencies, where the resonant orders go to an
item per lane, with continuations whose Landau terms do not factorise (two
Maxwellians, a Chebyshev series): the rows of every damped order are left to
the warps.  det D agrees with the FP64 path's at test_gpu_resonant_forms's
1e-8, and a batch beyond the line takes no more than twice the time of one
below (the rows' work is the same; leaving them to too few warps took 3.6
times as long).
"""
import time

import numpy as np
import pytest

from alps_gb300 import workloads

pytestmark = pytest.mark.gpu

RTOL = 1e-8


def _plasma(kind, precision):
    from alps_gb300 import _abi, api
    w = workloads.proton_electron(48, 96, 1.0, 0.3, 1e-14)
    species = []
    for sp in w["species"]:
        p = [sp.fit_init[0][i] for i in range(3)]
        pc = sp.perp_correction[0]
        if kind == "two":
            sp = _abi.species_defaults(ns=sp.ns, qs=sp.qs, ms=sp.ms, fits=[
                (1, [0.9 * p[0], p[1], p[2], 0, 0], pc), (1, [0.1 * p[0], 0.8 * p[1], p[2], 0, 0], 0.8 * pc)])
        else:
            sp.ac_method, sp.poly_kind, sp.poly_order, sp.poly_log_max = 2, 1, 12, 100.0
        species.append(sp)
    w["species"] = species
    system, tables = workloads.build(w, api.generate_f0)
    G = api.Plasma(system, tables, precision=precision)
    G.set_k(1.0, 0.3)
    return G


@pytest.mark.parametrize("kind", ["two", "chebyshev"])
def test_rows_left_to_the_warps(kind):
    rng = np.random.default_rng(9)
    om = rng.uniform(0.05, 2.5, 2600) - 1j * rng.uniform(0.0, 0.3, 2600)
    G = _plasma(kind, "mixed")
    ref = _plasma(kind, "fp64").disp_batch(om)
    assert np.all(np.abs(G.disp_batch(om) - ref) <= RTOL * np.abs(ref))

    def best(n):
        t = []
        for _ in range(8):
            t0 = time.perf_counter()
            G.disp_batch(om[:n])
            t.append(time.perf_counter() - t0)
        return min(t)

    assert best(2600) <= 2.0 * best(2500)
