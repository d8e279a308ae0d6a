"""Batches with tensors (calc_eigen) of one to thousands of roots: the lanes
per frequency change at fixed products of batch size and signed orders (100,
300, 900, 1500 and 7000 warps of orders).  Just below and above each line a
root's fields are those of the root alone to 1e-9 (E, B, U and delta n are
quotients of sums that agree to some 1e-13, with four digits of cancellation),
copies of a root agree bit for bit, and a large batch takes no more than five
times its det D (a lane in 32 at work took six to eight).
"""
import time

import numpy as np
import pytest

from alps_gb300 import _abi, workloads

pytestmark = pytest.mark.gpu

OMS = np.array([0.45 - 0.2j, 1.3 - 0.004j, 0.9 + 0.003j, 0.7 + 0.0j, 2.2 - 0.35j])
LINES = (100, 300, 900, 1500, 7000)


def _plasma(precision, kperp, bz):
    from alps_gb300 import api
    w = workloads.proton_electron(24, 51, kperp, 0.3, bz)
    system, species = workloads.build(w, api.generate_f0)
    G = api.Plasma(system, species, precision=precision)
    G.set_k(kperp, 0.3)
    return G


def _fields(e):
    return np.array(_abi.eigen_columns(e, 2)[0])


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_lines(precision):
    G = _plasma(precision, 3.0, 1e-20)
    orders = sum(2 * m + 1 for m in G.nmax())
    one = [_fields(G.calc_eigen([om], eigen=True, heat=False)[0]) for om in OMS]
    for u in LINES:
        first = -(-u * 32 // orders)  # the first n of the next shape
        for n in (first - 1, first):
            many = G.calc_eigen(np.resize(OMS, n), eigen=True, heat=False)
            for k, ref in enumerate(one):
                got = [_fields(many[q]) for q in range(k, n, len(OMS))]
                if got:
                    assert np.all(np.abs(got[0] - ref) <= 1e-9 * np.abs(ref).max()), (n, k)
                    assert all(np.array_equal(g, got[0]) for g in got), (n, k)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_time_of_many(precision):
    G = _plasma(precision, 8.0, 1e-20)
    om = np.resize(OMS, 1200)

    def best(f):
        t = []
        for _ in range(6):
            t0 = time.perf_counter()
            f()
            t.append(time.perf_counter() - t0)
        return min(t)

    assert best(lambda: G.calc_eigen(om, eigen=True, heat=False)) <= 5.0 * best(lambda: G.disp_batch(om))
