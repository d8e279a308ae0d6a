"""Batch sizes on both sides of every line of the launch shapes: lanes per
frequency and orders per chunk at fixed products of batch size and signed
orders (in warps of 32: mixed 100, 300, 440, 3000 and 7700, FP64 8, 50, 180, 400,
600 and 20000), the item-per-lane form of the resonant orders from 2560
frequencies (mixed), the last step by warps up to 4096, and the one launch of
small batches.  Every frequency's det D is that of a batch of its own to 1e-12
(the sums' order differs, each double-float sum is within 2^-40 of its terms'
magnitudes), and its copies within a batch agree bit for bit.
"""
import numpy as np
import pytest

from alps_gb300 import workloads

pytestmark = pytest.mark.gpu

OMS = np.array([0.45 - 0.2j, 1.3 - 0.004j, 0.9 + 0.003j, 0.7 + 0.0j, 2.2 - 0.35j])
RTOL = 1e-12
LINES = {"mixed": (100, 300, 440, 3000, 7700), "fp64": (8, 50, 180, 400, 600, 20000)}


def _plasma(precision, npar):
    from alps_gb300 import api
    w = workloads.proton_electron(24, npar, 1.0, 0.3, 1e-14)
    system, species = workloads.build(w, api.generate_f0)
    G = api.Plasma(system, species, precision=precision)
    G.set_k(1.0, 0.3)
    return G


def _check(G, ref, n):
    D = G.disp_batch(np.resize(OMS, n))
    for k in range(len(OMS)):
        got = D[k::len(OMS)]
        if len(got):
            assert np.all(np.abs(got[0] - ref[k]) <= RTOL * np.abs(ref[k])), (n, k, abs(got[0] / ref[k] - 1))
            assert np.all(got == got[0]), (n, k)


@pytest.mark.parametrize("npar", [48, 51])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_lines(precision, npar):
    G = _plasma(precision, npar)
    orders = sum(2 * m + 1 for m in G.nmax())
    ref = np.array([G.disp_batch(np.array([om]))[0] for om in OMS])
    first = [-(-u * 32 // orders) for u in LINES[precision]]  # the first n of the next shape
    for n in [f + d for f in first for d in (-1, 0)] + [2559, 2560, 4096, 4097]:
        _check(G, ref, n)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_end_of_the_one_launch(precision):
    G = _plasma(precision, 48)
    ref = np.array([G.disp_batch(np.array([om]))[0] for om in OMS])
    lo, hi = 1, 2559  # one launch; several
    while hi - lo > 1:
        mid = (lo + hi) // 2
        G.disp_batch(np.resize(OMS, mid))
        if G.stats().kernels_launched == 1:
            lo = mid
        else:
            hi = mid
    for n in (lo, hi):
        _check(G, ref, n)
        assert (G.stats().kernels_launched == 1) == (n == lo)
