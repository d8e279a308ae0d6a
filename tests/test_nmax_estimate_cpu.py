"""Debye's leading term as determine_nmax's screen (setup_kernels.cu nmax_body):
for z < 0.95 n it is above J_n(z) and less than a factor 8 (e^2.08) above it,
in FP32 too, and J_n rises on (0, n), so that the last node decides."""
import numpy as np
from scipy.special import jv


def _debye32(n, z):
    f = np.float32
    x = f(z) / f(n)
    ta = np.sqrt((f(1) - x) * (f(1) + x))
    return f(n) * (ta - np.log((f(1) + ta) / x)) - f(0.5) * np.log(f(6.2831853) * f(n) * ta)


def test_debye_brackets_bessel():
    rng = np.random.default_rng(2)
    seen = 0
    for n in list(range(1, 60)) + [100, 300, 1000, 1999]:
        for x in np.concatenate([rng.uniform(1e-3, 0.95, 200), [0.9499, 1e-6]]):
            j = jv(n, x * n)
            if not 1e-300 < j:
                continue
            tol = 1e-6 * n * (1.0 + abs(np.log(x)))
            d = float(_debye32(n, x * n)) - np.log(j)
            assert -tol <= d < 2.08 + tol, (n, x, d)
            seen += 1
    assert seen > 5000


def test_bessel_rises_below_its_order():
    for n in [1, 2, 5, 17, 60, 400]:
        z = np.linspace(0.0, 0.95 * n, 97)
        j = jv(n, z)
        j = j[j > 1e-300]
        assert np.all(j[1:] > j[:-1])
