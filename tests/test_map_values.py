"""A map's values log10 |det D|: the library's own logarithm (map_value.cuh)
against extended precision on the CPU, and the device's values against the
host's, bit for bit."""
import ctypes as C

import numpy as np
import pytest

from alps_gb300 import _abi, _native, build, workloads


def _finish(D):
    build.build()
    lib = C.CDLL(_native.LIB_PATH)
    D = np.ascontiguousarray(D, dtype=np.complex128)
    cal, val = np.empty_like(D), np.empty(len(D))
    f = lib.map_finish
    f.restype = None
    f(C.c_int(len(D)), D.ctypes.data_as(C.c_void_p), cal.ctypes.data_as(C.c_void_p), val.ctypes.data_as(C.c_void_p))
    return cal, val


def test_values_against_extended_precision():
    rng = np.random.default_rng(4)
    n = 60000
    e = 10.0 ** rng.uniform(-90, 90, n)
    D = (rng.uniform(-1, 1, n) + 1j * rng.uniform(-1, 1, n) * 10.0 ** -rng.integers(0, 12, n)) * e
    D[:200].imag = 0.0
    D[200:400].real = 0.0
    cal, val = _finish(D)
    assert np.array_equal(cal, D)
    x, y = D.real.astype(np.longdouble), D.imag.astype(np.longdouble)
    ref = np.log10(np.sqrt(x * x + y * y))
    far = np.abs(ref) > 0.01
    err = np.abs(val.astype(np.longdouble) - ref) / np.spacing(np.abs(ref).astype(float))
    assert np.all(err[far] <= 0.75)
    # near |D| = 1 the absolute error counts
    assert np.all(np.abs(val.astype(np.longdouble) - ref)[~far] <= 1e-18 + 1e-16 * np.abs(ref[~far]) + 3e-19)


def test_sentinels():
    nan, inf = np.nan, np.inf
    D = np.array([0.0, complex(nan, 0.0), 2e100, complex(-2e100, 5.0), complex(1.0, nan), complex(inf, 1.0),
                  complex(3.0, inf), 5e-324, 1e-310 + 1e-310j])
    cal, val = _finish(D)
    assert val[0] == -inf and cal[0] == 0.0
    assert val[1] == 999999.0 and cal[1] == 999999.0
    assert val[2] == val[3] == 899999.0 and cal[3] == 899999.0
    assert np.isnan(val[4]) and val[5] == 899999.0 and val[6] == inf
    assert abs(val[7] - np.log10(5e-324)) < 1e-12 and abs(val[8] - np.log10(np.sqrt(2.0)) + 310.0) < 1e-9


@pytest.mark.gpu
@pytest.mark.parametrize("nr,ni,log", [(1, 1, 0), (1, 7, 0), (37, 1, 1), (67, 45, 0), (50, 61, 1)])
def test_device_values_are_the_hosts(nr, ni, log):
    from alps_gb300 import api
    w = workloads.proton_electron(24, 48, 1.0, 0.3, 1e-9)
    system, species = workloads.build(w, api.generate_f0)
    G = api.Plasma(system, species, precision="mixed")
    G.set_k(1.0, 0.3)
    mp = _abi.alps_map_params()
    mp.omi, mp.omf, mp.gami, mp.gamf, mp.nr, mp.ni = 0.05, 2.5, 0.01, 0.2, nr, ni
    mp.loggridw = mp.loggridg = log
    om, cal, val = G.map_search(mp)
    wr = 0.05 * (2.5 / 0.05) ** (np.arange(nr) / max(nr - 1, 1)) if log else np.linspace(0.05, 2.5, nr)
    wi = 0.01 * (0.2 / 0.01) ** (np.arange(ni) / max(ni - 1, 1)) if log else np.linspace(0.01, 0.2, ni)
    assert np.allclose(om, (wr[:, None] + 1j * wi[None, :]).ravel(), rtol=1e-13)
    host_cal, host_val = _finish(cal)
    assert np.array_equal(host_cal, cal) and np.array_equal(host_val, val)
    assert np.array_equal(G.disp_batch(om), cal)
