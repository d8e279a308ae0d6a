"""Calls from host memory after small device batches that a caller left
running.  The overlapping call's own values are undefined (a context's batches
share its workspace), but every call after it gives its own det D, bit for
bit, and not what an earlier call left.
"""
import numpy as np
import pytest

from alps_gb300 import workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_host_calls_after_an_overlap(precision):
    import torch
    from alps_gb300 import api
    w = workloads.proton_electron(24, 51, 1.0, 0.3, 1e-14)
    system, species = workloads.build(w, api.generate_f0)
    G = api.Plasma(system, species, precision=precision)
    G.set_k(1.0, 0.3)
    rng = np.random.default_rng(4)
    oms = [rng.uniform(0.05, 2.5, n) + 1j * rng.uniform(-0.4, 0.05, n) for n in (64, 63, 48, 1)]
    ref = [G.disp_batch(o) for o in oms]
    other = torch.from_numpy(rng.uniform(0.05, 2.5, 64) + 1j * rng.uniform(-0.4, 0.05, 64)).cuda()
    out = torch.empty_like(other)
    s = torch.cuda.Stream()
    torch.cuda.synchronize()
    for _ in range(30):
        for _ in range(4):
            G.disp_batch_device(64, other.data_ptr(), out.data_ptr(), s.cuda_stream)
        G.disp_batch(oms[0])
        torch.cuda.synchronize()
        for o, r in zip(oms, ref):
            assert np.array_equal(G.disp_batch(o), r)
