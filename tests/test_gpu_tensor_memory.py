"""Tensors of thousands of roots at many Bessel orders: the partial sums, one
per order, are held for a part of the roots at a time (64 MiB), whatever their
number; copies of a root agree bit for bit over the parts, and with the root
alone to 1e-9 (see test_gpu_tensor_batches).
"""
import numpy as np
import pytest

from alps_gb300 import _abi, workloads

pytestmark = pytest.mark.gpu

OMS = np.array([0.45 - 0.2j, 1.3 - 0.004j, 0.9 + 0.003j, 0.7 + 0.0j, 2.2 - 0.35j, 0.6 - 0.1j, 1.9 - 0.02j])


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_parts(precision):
    import torch
    from alps_gb300 import api
    w = workloads.proton_electron(24, 51, 20.0, 0.3, 1e-20)
    system, species = workloads.build(w, api.generate_f0)
    G = api.Plasma(system, species, precision=precision)
    G.set_k(20.0, 0.3)
    n = 6001
    assert n * 2 * (2 * max(G.nmax()) + 1) * 96 > 4 * (64 << 20)  # all at once
    fields = lambda e: np.array(_abi.eigen_columns(e, 2)[0])
    one = [fields(G.calc_eigen([om], eigen=True, heat=False)[0]) for om in OMS]
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    many = G.calc_eigen(np.resize(OMS, n), eigen=True, heat=False)
    assert free - torch.cuda.mem_get_info()[0] < 128 << 20
    assert G.stats().n_eval == n
    got = np.array([fields(e) for e in many])
    for k, ref in enumerate(one):
        assert np.all(np.abs(got[k] - ref) <= 1e-9 * np.abs(ref).max())
        assert np.all(got[k::len(OMS)] == got[k])
