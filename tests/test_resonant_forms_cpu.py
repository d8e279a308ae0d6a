"""The resonant orders' fast forms, restated in numpy and checked against the
general ones.

  * device_math.cuh res_geometry_fast finds the window from one product and a
    floor on the uniform grid, and hands poles within 1e-5 spacings of a node
    or a half-way point to the general search: where it answers, both agree.
  * disp_kernels.cu sums the principal value as node weights: over the samples
    that interpolate about node j, with r = 1/(dx^2 + y^2), the sum of
    f H(p), H(p) = V_j + (p - p_j) (V_{j+1} - V_{j-1})/(2 dp), is A_j V_j +
    B_j (V_{j+1} - V_{j-1})/(2 dp), and so sum_j W_j V_j with W_j = A_j +
    (B_{j-1} - B_{j+1})/(2 dp).
"""
import numpy as np
import pytest


def _general(pp, M, MI, dpp, x):
    res = pp[1] <= x < pp[M] or pp[1] - MI * dpp <= x < pp[1] or pp[M - 1] <= x < pp[M - 1] + MI * dpp
    if not res:
        return (0, 1, M - 1, 1, 0)
    i = 0
    if pp[1] <= x < pp[M - 1]:
        i = max(j for j in range(1, M - 1) if pp[j] <= x)
    for ip in range(MI + 1):
        if pp[0] - dpp * ip <= x < pp[0] - dpp * (ip - 1):
            i = -ip
        if pp[M - 1] + dpp * ip <= x < pp[M - 1] + dpp * (ip + 1):
            i = M - 1 + ip
    if i - MI <= 2:
        return (1, i + MI, M - 1, 1, 0)
    if i + MI >= M - 2:
        return (2, 1, i - MI, 1, 0)
    up = i + MI + (1 if abs(x - pp[i]) < 0.5 * dpp else 2)
    return (3, 1, i - MI, up, M - 1)


def _fast(pp, M, MI, dpp, x):
    v = (x - pp[0]) / dpp
    if not (-MI < v < M + MI + 1):
        return None
    i, fr = int(np.floor(v)), np.float32(v - np.floor(v))
    if not (1e-5 < fr < 0.99999 and abs(fr - np.float32(0.5)) > 1e-5):
        return None
    if not (1 - MI <= i < M - 1 + (MI if MI > 1 else 1)):
        return (0, 1, M - 1, 1, 0)
    if i - MI <= 2:
        return (1, i + MI, M - 1, 1, 0)
    if i + MI >= M - 2:
        return (2, 1, i - MI, 1, 0)
    return (3, 1, i - MI, i + MI + (1 if fr < 0.5 else 2), M - 1)


@pytest.mark.parametrize("MI", [1, 2, 3, 5])
@pytest.mark.parametrize("M,lo,hi", [(24, -6.0, 6.0), (51, -5.5, 7.25), (13, 3.0, 3.5)])
def test_window_of_a_pole(MI, M, lo, hi):
    rng = np.random.default_rng(11)
    pp = lo + (hi - lo) * np.arange(M + 1) / M
    dpp = pp[2] - pp[1]
    x = np.concatenate([rng.uniform(lo - (MI + 3) * dpp, hi + (MI + 3) * dpp, 4000),
                        (pp[:, None] + dpp * np.array([0.0, 1e-4, -1e-4, 0.5, 0.4999, 0.5001])).ravel()])
    answered = 0
    for p in x:
        f = _fast(pp, M, MI, dpp, p)
        if f is not None:
            answered += 1
            assert f == _general(pp, M, MI, dpp, p), p
    assert answered > 3000 * (M + 1) / (M + 7)


@pytest.mark.parametrize("pr", [0.013, -0.21, 0.249])
def test_node_weights(pr):
    rng = np.random.default_rng(5)
    M, dp, y, MP = 40, 0.25, 0.07, 100
    pp = -5.0 + dp * np.arange(M + 1)
    V = rng.standard_normal(M + 1)
    i = int(np.floor((pr - pp[0]) / dp))
    lower, upper = i - 3, i + 5 if pr - pp[i] >= dp / 2 else i + 4
    cap = pr - pp[lower]
    sm = cap / MP
    nt = int((pp[upper] - pr - cap) / sm)
    cor = (pp[upper] - pr - cap) / sm / max(nt, 1)
    k = np.arange(MP + 1)
    kt = np.arange(nt + 1 if nt > 0 else 0)
    end = np.where((k == 0) | (k == MP), 1.0, 2.0)
    endt = np.where((kt == 0) | (kt == nt), 1.0, 2.0) * cor
    pts = [(pr + sm * k, end, 1.0), (pr - sm * k, end, -1.0), (pr + cap + cor * sm * kt, endt, 1.0)]
    direct, mag = 0.0, 0.0
    A = np.zeros(M + 2, complex)
    B = np.zeros(M + 2, complex)
    for p, w, sign in pts:
        dx = sign * np.abs(p - pr)
        f = w * (dx + 1j * y) / (dx * dx + y * y)
        j = np.rint((p - pp[0]) / dp).astype(int)
        H = V[j] + (p - pp[j]) * (V[j + 1] - V[j - 1]) / (2 * dp)
        direct += np.sum(f * H)
        mag += np.sum(np.abs(f * H))
        # a side's piece from its sums S1 = w r dx, S2 = w r, S3 = w r dx^2
        r = w / (dx * dx + y * y)
        for q in np.unique(j):
            s = j == q
            s1, s2, s3 = np.sum(r[s] * dx[s]), np.sum(r[s]), np.sum(w[s] - y * y * r[s])
            a = s1 + 1j * y * s2
            A[q] += a
            B[q] += (s3 + 1j * y * s1) + (pr - pp[q]) * a
    W = A.copy()
    W[1:-1] += (B[:-2] - B[2:]) / (2 * dp)
    W[0] -= B[1] / (2 * dp)
    assert abs(np.sum(W[:M + 1] * V) - direct) <= 1e-13 * mag
