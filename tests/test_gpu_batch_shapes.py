"""The launch shapes of a frequency batch: lanes per frequency and orders per
chunk of the pole sums, and one warp or one thread per frequency at the end.

The shape changes at fixed products of batch size and signed orders (220, 440,
3000, 7700 warps of orders) and at 4096 frequencies.  Batches just below and
above each line give every frequency the same det D as a batch of its own
(1e-12 relative: the sums' order differs, each double-float sum is within
2^-40 of its terms' magnitudes), and the copies of a frequency within a batch
agree bit for bit, wherever in the batch they sit.
"""
import numpy as np
import pytest

from alps_gb300 import workloads

pytestmark = pytest.mark.gpu

OMS = np.array([0.45 - 0.2j, 1.3 - 0.004j, 0.9 + 0.003j, 0.7 + 0.0j, 2.2 - 0.35j])
RTOL = 1e-12


@pytest.mark.parametrize("npar", [48, 51])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_batch_sizes_agree(precision, npar):
    from alps_gb300 import api
    w = workloads.proton_electron(24, npar, 1.0, 0.3, 1e-14)
    system, species = workloads.build(w, api.generate_f0)
    G = api.Plasma(system, species, precision=precision)
    G.set_k(1.0, 0.3)
    orders = sum(2 * n + 1 for n in G.nmax())
    ref = np.array([G.disp_batch(np.array([om]))[0] for om in OMS])
    edges = [-(-u * 32 // orders) for u in (220, 440, 3000, 7700)]  # first n of the next shape
    sizes = [2, 31, 33] + [n + d for n in edges for d in (-1, 0)] + [4096, 4097]
    for n in sizes:
        D = G.disp_batch(np.resize(OMS, n))
        for k in range(len(OMS)):
            got = D[k::len(OMS)]
            if len(got):
                assert np.all(np.abs(got - ref[k]) <= RTOL * abs(ref[k])), (n, k, np.abs(got / ref[k] - 1).max())
                assert np.all(got == got[0]), (n, k)


def test_tensors_of_many_frequencies():
    """calc_eigen's tensors: every order a chunk of its own; the fields of
    many roots together are those of each root alone."""
    from alps_gb300 import api
    w = workloads.proton_electron(24, 51, 1.0, 0.3, 1e-14)
    system, species = workloads.build(w, api.generate_f0)
    G = api.Plasma(system, species, precision="mixed")
    G.set_k(1.0, 0.3)
    many = G.calc_eigen(np.resize(OMS, 37), eigen=True, heat=False)
    for k, om in enumerate(OMS):
        one = G.calc_eigen([om], eigen=True, heat=False)[0]
        for q in range(k, 37, len(OMS)):
            for i in range(3):
                a, b = many[q].electric[i], one.electric[i]
                assert (a.re, a.im) == (b.re, b.im)
