"""Small batches in one launch (k_disp_one, k_disp_many) give the bits of the
separate kernels, which a round takes where a job is large or the jobs
together are too many: a context's results do not depend on what it is
batched with.  Profiling takes a lone batch to the separate kernels; a solve
of 400 plasmas is past the line of 7296 warps (28 slots and at least 8 warps of
pole sums each), one of 20 below it.
"""
import numpy as np
import pytest

from alps_gb300 import workloads

pytestmark = pytest.mark.gpu

OMS = np.array([0.45 - 0.2j, 1.3 - 0.004j, 0.9 + 0.003j, 0.7 + 0.0j, 2.2 - 0.35j, 0.05 + 0.1j, -1.1 - 0.02j])


@pytest.mark.parametrize("rows", ["shared", "uneven"])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("kpar", [0.3, -0.05])
def test_lone_batches(precision, kpar, rows):
    from alps_gb300 import api
    w = workloads.proton_electron(24, 51, 1.0, kpar, 1e-14)
    system, species = workloads.build(w, api.generate_f0)
    G = api.Plasma(system, species, precision=precision)
    if rows == "uneven":  # the Landau term by its rows
        for i in range(system.nspec):
            fit = np.array(G.get_fit(i))
            fit.reshape(-1, 5)[::2, 1] *= 1.001
            G.set_fit(i, fit)
    G.set_k(1.0, kpar)
    for n in (1, 2, 7, 31, 64, 65, 130):
        om = np.resize(OMS, n)
        one = G.disp_batch(om)
        assert G.stats().kernels_launched == 1
        G.set_profiling(True)
        many = G.disp_batch(om)
        assert G.stats().kernels_launched == 5
        G.set_profiling(False)
        assert np.array_equal(one, many), n
    for om in OMS:
        one = G.disp(om)
        G.set_profiling(True)
        many = G.disp(om)
        G.set_profiling(False)
        for a, b in zip(one, many):
            assert np.array_equal(a, b), om


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_rounds_on_both_sides_of_the_line(precision):
    from alps_gb300 import api
    rng = np.random.default_rng(13)
    n = 400
    ks = [(1.0, 0.05 + 0.002 * i) for i in range(n)]
    built = [workloads.build(workloads.proton_electron(24, 48, k[0], k[1], 1e-14), api.generate_f0) for k in ks]
    P = api.make_many(built, precision=precision, ks=ks)
    g = np.array([k[1] * (1.2 - 0.02j) * (1.0 + rng.uniform(-0.01, 0.01)) for k in ks])
    roots, iters, D, _ = api.solve_many(P, g)
    few = api.solve_many(P[:20], g[:20])
    assert np.array_equal(few[0], roots[:20]) and np.array_equal(few[1], iters[:20])
    assert np.array_equal(few[2], D[:20])
    for k in (0, 7, 399):
        r, i, d, _ = api.solve_many([P[k]], [g[k]])
        assert r[0] == roots[k] and i[0] == iters[k] and d[0] == D[k]
