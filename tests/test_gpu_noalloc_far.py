"""alps_disp_batch_noalloc with the far-order series (batches of 25000 warps of
orders and more): the series' coefficients, which belong to one k_par, come
from the call's static scratch like the rest.  The call gives the bits of
alps_disp_batch_device, alone and while batches of the same context at
another k_par run on another stream.
"""
import ctypes as C

import numpy as np
import pytest

from alps_gb300 import workloads

pytestmark = pytest.mark.gpu

KPERP, KPARS = 20.0, (0.3, 0.2)


def _call(G, om, out, stream):
    from alps_gb300._native import lib
    need = C.c_size_t()
    st = lib().alps_disp_batch_noalloc(G.handle, len(om), C.c_void_p(om.data_ptr()), C.c_void_p(out.data_ptr()),
                                       C.c_void_p(stream.cuda_stream), C.byref(need))
    assert st == 0 and 0 < need.value <= 16 << 20, (st, need.value)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_far_series_in_the_static_scratch(precision):
    import torch
    from alps_gb300 import api
    w = workloads.proton_electron(24, 48, KPERP, KPARS[0], 1e-20)
    system, species = workloads.build(w, api.generate_f0)
    G = api.Plasma(system, species, precision=precision)
    G.set_k(KPERP, KPARS[0])
    n = 25000 * 32 // sum(2 * m + 1 for m in G.nmax()) + 8
    rng = np.random.default_rng(11)
    om = torch.from_numpy(rng.uniform(0.05, 2.5, n) + 1j * rng.uniform(-0.3, 0.05, n)).cuda()
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    ref = []
    for k in KPARS:
        G.set_k(KPERP, k)
        d = torch.empty_like(om)
        G.disp_batch_device(n, om.data_ptr(), d.data_ptr(), b.cuda_stream)
        assert G.batch_status(b.cuda_stream) == 0
        assert G.stats().kernels_launched == 7  # stage, four, and the far orders' two
        ref.append(d.cpu().numpy())
    for k, r in zip(KPARS, ref):
        G.set_k(KPERP, k)
        d = torch.full_like(om, float("nan"))
        torch.cuda.synchronize()
        _call(G, om, d, a)
        assert G.batch_status(a.cuda_stream) == 0
        assert np.array_equal(d.cpu().numpy(), r)
    outs = [(torch.full_like(om, float("nan")), torch.full_like(om, float("nan"))) for _ in range(24)]
    torch.cuda.synchronize()
    for x, y in outs:
        G.set_k(KPERP, KPARS[0])
        _call(G, om, x, a)
        G.set_k(KPERP, KPARS[1])
        G.disp_batch_device(n, om.data_ptr(), y.data_ptr(), b.cuda_stream)
    torch.cuda.synchronize()
    for x, y in outs:
        assert np.array_equal(x.cpu().numpy(), ref[0])
        assert np.array_equal(y.cpu().numpy(), ref[1])


def test_batches_with_and_without_room_for_the_tables():
    """Of the batches that the scratch holds, those that leave no room for the
    series' tables sum order by order: the same bits through both entry points
    at every size, and both forms occur."""
    import torch
    from alps_gb300 import api
    from alps_gb300._native import lib
    w = workloads.proton_electron(24, 48, KPERP, KPARS[0], 1e-20)
    system, species = workloads.build(w, api.generate_f0)
    G = api.Plasma(system, species, precision="fp64")
    G.set_k(KPERP, KPARS[0])
    top = 20000
    rng = np.random.default_rng(12)
    om = torch.from_numpy(rng.uniform(0.05, 2.5, top) + 1j * rng.uniform(-0.3, 0.05, top)).cuda()
    s = torch.cuda.Stream()
    torch.cuda.synchronize()
    need = C.c_size_t()
    launches = set()
    for n in range(25000 * 32 // sum(2 * m + 1 for m in G.nmax()) + 1, top, 150):
        d, e = torch.empty_like(om[:n]), torch.empty_like(om[:n])
        torch.cuda.synchronize()
        if lib().alps_disp_batch_noalloc(G.handle, n, C.c_void_p(om.data_ptr()), C.c_void_p(d.data_ptr()),
                                         C.c_void_p(s.cuda_stream), C.byref(need)) != 0:
            assert need.value > 16 << 20
            continue
        G.disp_batch_device(n, om.data_ptr(), e.data_ptr(), s.cuda_stream)
        assert G.batch_status(s.cuda_stream) == 0
        assert torch.equal(d, e), n
        launches.add(G.stats().kernels_launched)
    assert launches == {5, 7}
