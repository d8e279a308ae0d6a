"""What a user of the dispersion library has it do, as timed cases.

A case is a dict of plain values.  ``prepare`` builds what a user's program
holds before the call (f0 tables, plasmas at their k, frequencies),
``run`` makes one pass through the public entry points of alps_gb300.api,
``exact`` restates the same result in 64-bit numpy.

Sizes, k ranges and species follow the configurations of this repository:
the 60x120 k-scan, the 120x240 quick test, the 128x256 frequency map, the
uneven draws on 64x128 to 256x512 grids, the Juettner electrons.  The seed
moves the species' betas and anisotropies by a few per cent and draws the
frequencies and guesses.
"""
import math

import numpy as np
import torch

from alps_gb300 import _abi, api, workloads

M_E = 1.0 / 1836.0
V_A = 1e-4
M_I, M_P, T_LIM = 3, 100, 0.01   # principal-value window and samples of every case
RTOL = 1e-12                     # relative-step stop of the root polishes

# the entries xx yy zz xy xz yz of a symmetric tensor
ROWS, COLS = [0, 1, 2, 0, 0, 1], [0, 1, 2, 1, 2, 2]


# ---------------------------------------------------------------------------
# cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # one det D with chi, chi_low and the wave tensor: what calc_eigen and
        # a user's own root finder ask for, on the quick test's grid
        dict(name="tensor_120x240_fp64", kind="tensor", precision="fp64", nperp=120, npar=240, kperp=0.5, kpar=0.2,
             bessel_zero=1e-50),
        # a few frequencies from host memory: the step of a root finder that
        # advances a handful of roots on one plasma
        dict(name="batch_31_64x128_mixed", kind="batch", precision="mixed", plasma="bimax", nperp=64, npar=128,
             kperp=1.0, kpar=0.3, bessel_zero=1e-20, n=31, device=False),
        # an odd number of frequencies already on the device, on a caller's stream
        dict(name="batch_2999_128x256_mixed", kind="batch", precision="mixed", plasma="bimax", nperp=128, npar=256,
             kperp=2.0, kpar=0.3, bessel_zero=1e-9, n=2999, device=True),
        # three species on an odd grid, with a beam and a kappa continuation
        dict(name="batch_700_193x385_mixed", kind="batch", precision="mixed", plasma="kappa", nperp=193, npar=385,
             kperp=1.5, kpar=0.7, bessel_zero=1e-20, n=700, device=False),
        # the complex-frequency map of the benchmark configuration
        dict(name="map_512x512_128x256_mixed", kind="map", precision="mixed", nperp=128, npar=256, kperp=2.0,
             kpar=0.3, bessel_zero=1e-9, nr=512, ni=512),
        # a coarse map on the all-FP64 path
        dict(name="map_61x47_128x256_fp64", kind="map", precision="fp64", nperp=128, npar=256, kperp=2.0, kpar=0.3,
             bessel_zero=1e-9, nr=61, ni=47),
        # the k-scan configuration, up to where the wave is strongly damped: one
        # root followed along k_par, the k tables kept
        dict(name="scan_kpar_60x120_mixed", kind="scan", precision="mixed", nperp=60, npar=120, kperp=1.0,
             kpar=0.05, bessel_zero=1e-50, type_s=4, end=0.4, steps=32),
        # a root followed in |k| at fixed angle: the k tables are built at every step
        dict(name="scan_k_96x192_fp64", kind="scan", precision="fp64", nperp=96, npar=192, kperp=0.4, kpar=0.1,
             bessel_zero=1e-20, type_s=2, end=0.8, steps=16),
        # many roots, each on a plasma and grid of its own, in one call
        dict(name="solves_48_mixed", kind="solves", precision="mixed", plasmas=48, nperp_max=192),
        # Juettner electrons on the (Gamma, p_par) grid beside closed-form protons
        dict(name="relativistic_100x200", kind="relativistic", nperp=24, npar=48, ngamma=100, npparbar=200,
             theta_e=0.3, kpar_de=0.25, n=8),
        # a new plasma from its tables: derivatives, continuation fits, k tables, first values
        dict(name="setup_192x384_mixed", kind="setup", precision="mixed", nperp=192, npar=384, kperp=1.0, kpar=0.5,
             bessel_zero=1e-20),
        # requests on many plasmas through one server: polishes, a k_par scan, a map
        dict(name="served_32_mixed", kind="served", precision="mixed", polishes=32, nperp_max=128, nr=48, ni=48),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["tensor", "batch", "batch", "batch", "map", "map", "scan", "solves", "relativistic", "setup",
                       "served"])
    precision = rng.choice(["mixed", "mixed", "fp64"])
    nperp = _log_int(rng, 48, 200)
    c = dict(kind=kind, precision=precision, nperp=nperp, npar=2 * nperp + rng.choice([0, 1]),
             kperp=round(math.exp(rng.uniform(math.log(0.3), math.log(3.0))), 3),
             kpar=round(math.exp(rng.uniform(math.log(0.1), math.log(1.0))), 3),
             bessel_zero=rng.choice([1e-9, 1e-20, 1e-50]))
    if kind == "batch":
        c["plasma"] = rng.choice(["bimax", "bimax", "kappa"])
        top = 20000 if precision == "mixed" else 2000
        c["n"] = _log_int(rng, 1, top // 10 if c["plasma"] == "kappa" else top)
        c["device"] = rng.choice([True, False])
    elif kind == "map":
        top = 300 if precision == "mixed" else 60
        c["nr"], c["ni"] = _log_int(rng, 8, top), _log_int(rng, 8, top)
    elif kind == "scan":
        c["kperp"], c["kpar"] = round(rng.uniform(0.3, 1.0), 3), round(rng.uniform(0.03, 0.1), 3)
        c["type_s"] = rng.choice([2, 4])
        k0 = c["kpar"] if c["type_s"] == 4 else math.hypot(c["kperp"], c["kpar"])
        c["end"] = round(rng.uniform(1.5, 3.0) * k0, 4)
        c["steps"] = _log_int(rng, 4, 32)
    elif kind == "solves":
        c = dict(kind=kind, precision=precision, plasmas=_log_int(rng, 1, 64), nperp_max=rng.choice([96, 128, 192]))
    elif kind == "served":
        c = dict(kind=kind, precision=precision, polishes=_log_int(rng, 2, 32), nperp_max=rng.choice([64, 96, 128]),
                 nr=_log_int(rng, 8, 48), ni=_log_int(rng, 8, 48))
    elif kind == "relativistic":
        c = dict(kind=kind, nperp=rng.choice([20, 24]), npar=rng.choice([40, 48]), ngamma=rng.randint(60, 100),
                 npparbar=rng.randint(121, 200), theta_e=round(rng.uniform(0.1, 0.3), 3),
                 kpar_de=round(rng.uniform(0.1, 0.3), 3), n=_log_int(rng, 1, 8))
    return c


# ---------------------------------------------------------------------------
# plasmas
# ---------------------------------------------------------------------------
def _species(kind, ms, qs, ns, beta, alph, nperp, npar, drift=0.0, kappa=0.0):
    """One species: its f0 table (bi-Maxwellian, drifting beam or bi-kappa)
    on the uniform grid of six thermal momenta, and the parameters of its
    analytic continuation."""
    thp, thz = beta * ms * alph, beta * ms
    pp = np.arange(nperp + 1) * (6.0 * math.sqrt(thp) / nperp)
    pz = np.arange(npar + 1) * (12.0 * math.sqrt(thz) / npar) - 6.0 * math.sqrt(thz) + drift
    d = pz[None, :] - drift
    if kind == "kappa":
        a2 = (2.0 * kappa - 3.0) / (2.0 * kappa)
        norm = math.gamma(kappa + 1.0) / math.gamma(kappa - 0.5) / ((math.pi * thz * kappa * a2) ** 1.5 * alph)
        f0 = norm * (1.0 + d * d / (thz * kappa * a2) + pp[:, None] ** 2 / (thp * kappa * a2)) ** (-1.0 - kappa)
        fit, pc, ftype = [norm, 1.0 / (thz * kappa * a2), drift, -1.0 - kappa, 1.0], 1.0 / (thp * kappa * a2), 2
    else:
        norm = math.pi ** -1.5 / (thz ** 1.5 * alph)
        f0 = norm * np.exp(-(d * d) / thz - pp[:, None] ** 2 / thp)
        fit, pc, ftype = [norm, 1.0 / thz, drift, 0.0, 0.0], 1.0 / thp, 1
    return dict(ms=ms, qs=qs, ns=ns, pp=pp, pz=pz, f0=f0, fit=fit, pc=pc, ftype=ftype)


def _bimax(nperp, npar, rng, beta=1.0):
    """Protons and electrons, bi-Maxwellian."""
    return [_species("bimax", ms, qs, 1.0, beta * rng.uniform(0.9, 1.1), rng.uniform(0.9, 1.1), nperp, npar)
            for ms, qs in ((1.0, 1.0), (M_E, -1.0))]


def _with_kappa(nperp, npar, rng):
    """A proton core, a drifting proton beam and kappa electrons."""
    b = rng.uniform(0.9, 1.1)
    return [_species("bimax", 1.0, 1.0, 1.0, b, rng.uniform(0.9, 1.1), nperp, npar),
            _species("beam", 1.0, 1.0, 0.1, b, 1.0, nperp, npar, drift=rng.uniform(0.8, 1.2)),
            _species("kappa", M_E, -1.0, 1.1, b, 1.0, nperp, npar, kappa=rng.uniform(4.5, 5.5))]


def _system(case, nspec):
    return _abi.system_defaults(
        nspec=nspec, nperp=case["nperp"], npar=case["npar"], kperp=case["kperp"], kpar=case["kpar"], vA=V_A,
        Bessel_zero=case["bessel_zero"], secant_method=2, numiter=50, kperp_norm=1, D_threshold=1e-15,
        positions_principal=M_I, n_resonance_interval=M_P, Tlim=T_LIM)


def _tables(species, fit_scale=1.0):
    """(alps_species, pperp, ppar, f0) tuples; fit_scale moves the seeds of
    the continuation fit away from the table's own parameters."""
    out = []
    for s in species:
        n, m = s["f0"].shape
        fit = [s["fit"][0] * fit_scale, s["fit"][1] * fit_scale] + s["fit"][2:]
        out.append((_abi.species_defaults(ns=s["ns"], qs=s["qs"], ms=s["ms"], fits=[(s["ftype"], fit, s["pc"])]),
                    np.repeat(s["pp"], m), np.tile(s["pz"], n), s["f0"].ravel()))
    return out


def _plasma_of(case, seed):
    rng = np.random.default_rng(seed)
    species = (_with_kappa if case.get("plasma") == "kappa" else _bimax)(case["nperp"], case["npar"], rng)
    return species, rng


def _alfven_guess(species, kperp, kpar):
    """The kinetic Alfven wave's frequency, omega^2 = k_par^2 (1 + k_perp^2
    rho^2 / (beta + 1)), weakly damped."""
    beta = 1.0 / species[0]["fit"][1]
    w = kpar * math.sqrt(1.0 + kperp ** 2 * beta / (1.0 + beta))
    return w * (1.0 - 0.03j)


def _uneven(case, seed, count):
    """(case, species, guess) of ``count`` plasmas, each with a grid, beta
    and k of its own, with a guess within a per cent of the Alfven wave."""
    rng = np.random.default_rng(seed)
    grids = [g for g in (64, 96, 128, 192, 256) if g <= case["nperp_max"]]
    out = []
    for i in range(count):
        n = grids[i % len(grids)]
        beta = 10.0 ** rng.uniform(-0.5, 0.3)
        kperp, kpar = 10.0 ** rng.uniform(-0.7, 0.1), 10.0 ** rng.uniform(-1.7, -1.0)
        c = dict(nperp=n, npar=2 * n, kperp=kperp, kpar=kpar, bessel_zero=1e-20, precision=case["precision"])
        species = _bimax(n, 2 * n, rng, beta)
        g = _alfven_guess(species, kperp, kpar)
        out.append((c, species, g * (1.0 + rng.uniform(-0.01, 0.01) + 0.01j * rng.uniform(-1.0, 1.0))))
    return out


def _make_uneven(case, plasmas):
    return api.make_many([(_system(c, 2), _tables(s)) for c, s, _ in plasmas], precision=case["precision"],
                         ks=[(c["kperp"], c["kpar"]) for c, _, _ in plasmas])


def _damping(kpar):
    """The strongest damping searched, in units of that at k_par = 0.3: the
    continuation grows as exp((Im omega / k_par)^2), and with it the
    cancellation in det D."""
    return min(1.0, kpar / 0.3)


def _frequencies(rng, n, kpar):
    return rng.uniform(0.05, 2.5, n) + 1j * _damping(kpar) * rng.uniform(-0.4, 0.05, n)


def _map(nr, ni, rng, kpar):
    mp = _abi.alps_map_params()
    mp.omi, mp.omf = 0.02 * (1.0 + rng.uniform()), 3.0
    mp.gami, mp.gamf = (-0.5 + 0.01 * rng.uniform()) * _damping(kpar), 0.1 * _damping(kpar)
    mp.nr, mp.ni, mp.loggridw, mp.loggridg = nr, ni, 0, 0
    return mp


def _lattice(mp):
    wr = mp.omi + (mp.omf - mp.omi) / (mp.nr - 1) * np.arange(mp.nr)
    wi = mp.gami + (mp.gamf - mp.gami) / (mp.ni - 1) * np.arange(mp.ni)
    return (wr[:, None] + 1j * wi[None, :]).ravel()


# the scan among a server's requests
SERVED_SCAN = dict(kpar_factor=1.3, steps=8)


# ---------------------------------------------------------------------------
# preparation and the timed pass
# ---------------------------------------------------------------------------
def prepare(case, seed):
    kind = case["kind"]
    if kind == "relativistic":
        rng = np.random.default_rng(seed)
        w = workloads.config_relativistic(case["theta_e"] * rng.uniform(0.98, 1.02), nperp=case["nperp"],
                                          npar=case["npar"], ngamma=case["ngamma"], npparbar=case["npparbar"],
                                          kpar_de=case["kpar_de"])
        system, tables = workloads.build_relativistic(w, api.generate_f0)
        P = api.Plasma(system, tables)
        P.set_k(*w["k"])
        g = w["extra"]["guess"][0]
        om = g * (1.0 + rng.uniform(-0.05, 0.05, case["n"])) + 1j * abs(g) * rng.uniform(-0.1, 0.02, case["n"])
        return dict(case=case, plasma=P, om=om)
    if kind in ("solves", "served"):
        plasmas = _uneven(case, seed, case["plasmas"] if kind == "solves" else case["polishes"] + 2)
        st = dict(case=case, plasmas=_make_uneven(case, plasmas), guesses=np.array([p[2] for p in plasmas]))
        if kind == "served":
            st["map"] = _map(case["nr"], case["ni"], np.random.default_rng(seed + 1), plasmas[-1][0]["kpar"])
            st["server"] = api.Server()
        return st
    species, rng = _plasma_of(case, seed)
    system = _system(case, len(species))
    if kind == "setup":
        return dict(case=case, system=system, tables=_tables(species, 1.0 + rng.uniform(0.02, 0.03)),
                    om=_frequencies(rng, 3, case["kpar"]))
    P = api.Plasma(system, _tables(species), precision=case["precision"])
    P.set_k(case["kperp"], case["kpar"])
    st = dict(case=case, plasma=P)
    if kind == "tensor":
        st["om"] = complex(_frequencies(rng, 1, case["kpar"])[0])
    elif kind == "batch":
        st["om"] = _frequencies(rng, case["n"], case["kpar"])
        if case["device"]:
            st["om"] = torch.from_numpy(st["om"]).cuda()
            st["D"] = torch.empty_like(st["om"])
            st["stream"] = torch.cuda.Stream()
    elif kind == "map":
        st["map"] = _map(case["nr"], case["ni"], rng, case["kpar"])
    elif kind == "scan":
        st["guess"] = _alfven_guess(species, case["kperp"], case["kpar"])
    return st


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "tensor":
        D, chi0, chi0_low, wave = state["plasma"].disp(state["om"])
        return {"D": np.array([D]), "chi0": chi0, "chi0_low": chi0_low, "wave": wave}
    if kind == "batch" and case["device"]:
        state["plasma"].disp_batch_device(case["n"], state["om"].data_ptr(), state["D"].data_ptr(),
                                          state["stream"].cuda_stream)
        return {"D": state["D"]}
    if kind in ("batch", "relativistic"):
        return {"D": state["plasma"].disp_batch(state["om"])}
    if kind == "map":
        om, cal, val = state["plasma"].map_search(state["map"])
        return {"om": om, "cal": cal, "val": val}
    if kind == "scan":
        P = state["plasma"]
        P.set_k(case["kperp"], case["kpar"])
        roots = P.polish([state["guess"]], om_rtol=RTOL)[0]
        rows, _ = P.om_scan(case["type_s"], 0.0, case["end"], True, case["steps"], 1, roots, om_rtol=RTOL)
        return {"rows": rows}
    if kind == "solves":
        return {"roots": api.solve_many(state["plasmas"], state["guesses"], om_rtol=RTOL)[0]}
    if kind == "setup":
        P = api.Plasma(state["system"], state["tables"], precision=case["precision"])
        P.set_k(case["kperp"], case["kpar"])
        return {"fits": [P.get_fit(i) for i in range(P.nspec)], "nmax": np.array(P.nmax()),
                "D": P.disp_batch(state["om"])}
    # served: the last two plasmas take the scan and the map, the others a polish each
    srv, plasmas, guesses = state["server"], state["plasmas"], state["guesses"]
    s = plasmas[-2]
    k0 = (state.setdefault("k0", (s.kperp, s.kpar)))
    s.set_k(*k0)
    sc = api.scan_def(4, 0.0, k0[1] * SERVED_SCAN["kpar_factor"], True, SERVED_SCAN["steps"], 1, *k0)
    scan = srv.scan(s, sc, [guesses[-2]], om_rtol=RTOL)
    mapped = srv.map(plasmas[-1], state["map"])
    polished = [srv.polish(p, [g], om_rtol=RTOL) for p, g in zip(plasmas[:-2], guesses[:-2])]
    cal, val = mapped.wait()
    return {"roots": np.concatenate([r.wait() for r in polished]), "rows": scan.wait()[0][1:], "cal": cal, "val": val}


# ---------------------------------------------------------------------------
# the least work of a pass
# ---------------------------------------------------------------------------
def _orders(case, qs, pmax):
    """About the Bessel orders a species keeps: the argument's largest value
    z and the orders beyond it until J_n falls below the cutoff."""
    z = case["kperp"] * pmax / abs(qs)
    n = z
    while n * math.log(max(n, 1.0) * 2.0 / (math.e * max(z, 1e-30))) < -math.log(case["bessel_zero"]):
        n += 1.0
    return n


def _eval_flops(case, species=None):
    """Flops of one det D: per species, order and p_par node 150 (two complex
    reciprocals, three numerators, twelve entry sums), per resonant order 24
    per principal-value sample and 60 per p_perp row."""
    total = 0.0
    for ms, qs in species or ((1.0, 1.0), (M_E, -1.0)):
        n = _orders(case, qs, 6.0 * math.sqrt(ms))
        items = min(2.0 * n + 1.0, 12.0 * math.sqrt(ms) * case["kpar"] / abs(qs) + 1.0)
        total += 150.0 * (n + 1.0) * (case["npar"] - 1) + items * (24.0 * M_P + 60.0 * (case["nperp"] + 1))
    return total


def _contraction_flops(case):
    """Flops of the p_perp sums of one k."""
    return sum(2.0 * 3.0 * (_orders(case, 1.0, 6.0 * math.sqrt(ms)) + 1.0) * case["nperp"] * 2.0 * case["npar"]
               for ms in (1.0, M_E))


def _table_bytes(case, nspec=2):
    """The tables an evaluation reads: two real vectors of three Bessel
    families per order and p_par node."""
    return 48.0 * case["npar"] * nspec * (_orders(case, 1.0, 6.0) + 1.0)


def work(case):
    kind = case["kind"]
    if kind == "relativistic":
        rows, nodes, orders = case["ngamma"] - 1, case["npparbar"] + 4 * M_P, 2 * 20 + 1
        return {"bytes": 32.0 * case["n"] + 24.0 * case["ngamma"] * case["npparbar"],
                "flops": 60.0 * case["n"] * orders * rows * nodes}
    if kind in ("solves", "served"):
        c = dict(nperp=case["nperp_max"], npar=2 * case["nperp_max"], kperp=0.5, kpar=0.02, bessel_zero=1e-20)
        n = case["plasmas"] if kind == "solves" else case["polishes"]
        evals = 8.0 * n + (0.0 if kind == "solves" else 8.0 * SERVED_SCAN["steps"] + case["nr"] * case["ni"])
        return {"bytes": n * _table_bytes(c), "flops": evals * _eval_flops(c)}
    grid = (case["nperp"] + 1) * (case["npar"] + 1)
    if kind == "setup":
        # per point of a row 100 flops and two iterations of the fit, and the k tables
        return {"bytes": 2.0 * 8.0 * grid, "flops": 2.0 * 200.0 * grid + _contraction_flops(case)}
    if kind == "scan":
        evals = 8.0 * (case["steps"] + 1)
        ks = case["steps"] + 1 if case["type_s"] == 2 else 0
        return {"bytes": (_table_bytes(case) if not ks else ks * 32.0 * grid),
                "flops": evals * _eval_flops(case) + ks * _contraction_flops(case)}
    species = ((1.0, 1.0), (1.0, 1.0), (M_E, -1.0)) if case.get("plasma") == "kappa" else None
    n = {"tensor": 1, "batch": case.get("n", 0), "map": case.get("nr", 0) * case.get("ni", 0)}[kind]
    out = {"tensor": 16.0 * (1 + 36 * 2 + 9), "batch": 32.0, "map": 16.0 + 16.0 + 8.0}[kind]
    return {"bytes": _table_bytes(case, 3 if species else 2) + out * n, "flops": n * _eval_flops(case, species)}


# ---------------------------------------------------------------------------
# the same results in 64-bit numpy
# ---------------------------------------------------------------------------
def _j0(x):
    """J0 by the rational approximations ALPS uses (src/ALPS_fns_rel.f90:1651-1692)."""
    ax = np.abs(x)
    y = x * x
    small = (np.polynomial.polynomial.polyval(y, [57568490574.0, -13362590354.0, 651619640.7, -11214424.18, 77392.33017,
                                                  -184.9052456]) /
             np.polynomial.polynomial.polyval(y, [57568490411.0, 1029532985.0, 9494680.718, 59272.64853, 267.8532712,
                                                  1.0]))
    z = 8.0 / np.maximum(ax, 8.0)
    y = z * z
    p = np.polynomial.polynomial.polyval(y, [1.0, -.1098628627e-2, .2734510407e-4, -.2073370639e-5, .2093887211e-6])
    q = np.polynomial.polynomial.polyval(y, [-.1562499995e-1, .1430488765e-3, -.6911147651e-5, .7621095161e-6,
                                             -.9349451520e-7])
    xx = ax - .785398164
    large = np.sqrt(.636619772 / np.maximum(ax, 8.0)) * (p * np.cos(xx) - z * q * np.sin(xx))
    return np.where(ax < 8.0, small, large)


def _j1(x):
    """J1 likewise (src/ALPS_fns_rel.f90:1695-1735; one constant in single precision)."""
    ax = np.abs(x)
    y = x * x
    small = x * (np.polynomial.polynomial.polyval(y, [72362614232.0, -7895059235.0, 242396853.1, -2972611.439,
                                                      15704.48260, -30.16036606]) /
                 np.polynomial.polynomial.polyval(y, [144725228442.0, 2300535178.0, 18583304.74, 99447.43394,
                                                      376.9991397, 1.0]))
    z = 8.0 / np.maximum(ax, 8.0)
    y = z * z
    p = np.polynomial.polynomial.polyval(y, [1.0, .183105e-2, -.3516396496e-4, .2457520174e-5, -.240337019e-6])
    q = np.polynomial.polynomial.polyval(y, [.04687499995, -.2002690873e-3, .8449199096e-5, -.88228987e-6,
                                             .105787412e-6])
    xx = ax - float(np.float32(2.35619491))
    large = np.sqrt(.636619772 / np.maximum(ax, 8.0)) * (p * np.cos(xx) - z * q * np.sin(xx))
    return np.where(ax < 8.0, small, np.where(x < 0.0, -large, large))


def _jn(n, x):
    """J_n: upward recurrence for x > n, Miller's downward one otherwise
    (src/ALPS_fns_rel.f90:1575-1646)."""
    if n < 2:
        return _j0(x) if n == 0 else _j1(x)
    out = np.zeros_like(x)
    up = x > n
    if up.any():
        t = 2.0 / x[up]
        a, b = _j0(x[up]), _j1(x[up])
        for j in range(1, n):
            a, b = b, j * t * b - a
        out[up] = b
    down = ~up & (x != 0.0)
    if down.any():
        t = 2.0 / x[down]
        m = 2 * ((n + int(math.sqrt(float(np.float32(40 * n))))) // 2)
        above, here, res, total = np.zeros_like(t), np.ones_like(t), np.zeros_like(t), np.zeros_like(t)
        odd = False
        for j in range(m, 0, -1):
            above, here = here, j * t * here - above
            f = np.where(np.abs(here) > 1e10, 1e-10, 1.0)
            above, here, res, total = above * f, here * f, res * f, total * f
            if odd:
                total = total + here
            odd = not odd
            if j == n:
                res = above
        out[down] = res / (2.0 * total - here)
    return out


class _Numpy:
    """chi and det D of species dicts at one k, in plain numpy."""

    def __init__(self, species, kperp, kpar, bessel_zero):
        self.species, self.kperp, self.kpar = species, kperp, kpar
        self.tabs = [self._table(s, bessel_zero) for s in species]
        self.cost = sum((2 * t["nmax"] + 1) * len(s["pz"]) for s, t in zip(species, self.tabs))

    def _table(self, s, bessel_zero):
        pp, pz, f0 = s["pp"], s["pz"], s["f0"]
        z = self.kperp * pp / s["qs"]
        J = [_jn(0, z), _jn(1, z)]
        nmax = 1
        while np.abs(J[nmax]).max() > bessel_zero:
            nmax += 1
            J.append(_jn(nmax, z))
        J.append(_jn(nmax + 1, z))
        J = np.array(J)
        d = np.zeros_like(J[:-1])
        d[0] = -J[1]
        d[1:] = 0.5 * (J[:-2] - J[2:])
        J = J[:-1]
        R = np.array([J * J, (pp * pp) * d * d, pp * J * d])
        w = np.full(len(pp) - 2, 2.0)
        w[-1] = 1.0
        g1 = (f0[2:, 1:-1] - f0[:-2, 1:-1]) / (pp[2:] - pp[:-2])[:, None]
        g2 = (pp[1:-1, None] * (f0[1:-1, 2:] - f0[1:-1, :-2]) / (pz[2:] - pz[:-2]) - pz[1:-1] * g1)
        wp = np.full(len(pz) - 2, 2.0)
        wp[0] = wp[-1] = 1.0
        dpp, dpz = pp[2] - pp[1], pz[2] - pz[1]
        ee = 2.0 * math.pi * s["qs"] / s["ms"] * dpp * dpz * 0.25 * float(w @ (g2 * pz[1:-1]) @ wp)
        A = 2.0 * np.einsum("fni,gij->nfgj", R[:, :, 1:-1] * w, np.array([g1, g2]))
        p = pz[1:-1]
        # entries' families and p_par powers; V[n, entry, g, node 1..M-1]
        V = np.stack([A[:, 0], A[:, 1], A[:, 0] * p * p, A[:, 2], A[:, 0] * p, A[:, 2] * p], axis=1)
        return dict(nmax=nmax, R=R, V=V, ee=ee, dpp=dpp, dpz=dpz)

    def _fit(self, s, p):
        """The analytic continuation at complex p, every p_perp row."""
        a, b, drift, power, scale = s["fit"]
        pp2 = s["pc"] * s["pp"] ** 2
        if s["ftype"] == 2:
            return a * np.exp(power * np.log(1.0 + b * (p - drift) ** 2 + scale * pp2))
        return a * np.exp(-pp2) * np.exp(-b * (p - drift) ** 2)

    def _landau(self, s, t, n, om, p):
        pp, dpp, dpz = s["pp"], t["dpp"], t["dpz"]
        f, fp, fm = self._fit(s, p), self._fit(s, p + dpz), self._fit(s, p - dpz)
        if np.any((np.abs(fp[1:-1]) == 0.0) | (np.abs(fm[1:-1]) == 0.0) | (np.abs(f[2:]) == 0.0)):
            return np.zeros(6, complex)
        dperp = np.empty_like(f)
        dperp[1:-1] = (f[2:] - f[:-2]) / (2.0 * dpp)
        dperp[0], dperp[-1] = (f[1] - f[0]) / dpp, (f[-1] - f[-2]) / dpp
        h = np.ones(len(pp))
        h[[0, -2, -1]] = 0.5
        L = s["qs"] / abs(self.kpar) * ((pp * (fp - fm) / (2.0 * dpz) - p * dperp) * self.kpar / s["ms"] + om * dperp)
        S = t["R"][:, abs(n)] @ (h * L)
        return np.array([S[0], S[1], S[0] * p * p, S[2], S[0] * p, S[2] * p]) * (-2j * math.pi ** 2 * dpp)

    def _window(self, pz, x, dpz):
        """Resonance of one order: (resonant, first range, second range,
        principal-value window) in node indices."""
        m = len(pz) - 1
        if not (pz[1] - M_I * dpz <= x < pz[m - 1] + M_I * dpz or pz[1] <= x < pz[m]):
            return False, (1, m - 1), None, None
        ires = 0
        if pz[1] <= x < pz[m - 1]:
            ires = min(max(int(np.searchsorted(pz, x, "right")) - 1, 1), m - 2)
        for i in range(M_I + 1):
            if pz[0] - dpz * i <= x < pz[0] - dpz * (i - 1):
                ires = -i
            if pz[m - 1] + dpz * i <= x < pz[m - 1] + dpz * (i + 1):
                ires = m - 1 + i
        if ires - M_I <= 2:
            return True, (ires + M_I, m - 1), None, None
        if ires + M_I >= m - 2:
            return True, (1, ires - M_I), None, None
        lower = ires - M_I
        upper = ires + M_I + (1 if abs(x - pz[ires]) < 0.5 * dpz else 2)
        return True, (1, lower), (upper, m - 1), (lower, upper)

    def _principal(self, s, t, n, om, pr, pim, window):
        pz, dpz = s["pz"], t["dpz"]
        m = len(pz) - 1
        V = t["V"][abs(n)]
        h = om * V[:, 0] + (self.kpar / s["ms"]) * V[:, 1]
        lower, upper = window

        def at(p):
            # the last node within half a spacing, kept off the ends
            p = np.atleast_1d(p)
            near = np.floor((p - pz[0]) / dpz + 0.5).astype(int)
            jc = np.zeros(len(p), int)
            for off in (-2, -1, 0, 1, 2):
                j = near + off
                ok = (j >= 1) & (j <= m - 1)
                ok[ok] = np.abs(pz[j[ok]] - p[ok]) <= 0.5 * dpz
                jc[ok] = j[ok]
            jc = np.where(jc >= m - 1, m - 2, np.where(jc <= 1, 2, jc))
            return h[:, jc - 1] + (h[:, jc] - h[:, jc - 2]) * (0.5 / dpz) * (p - pz[jc])

        cap = pr - pz[lower]
        sm = cap / M_P
        T = np.zeros(6, complex)
        k = np.arange(M_P + 1)
        p = pr + sm * k
        p[-1] = pr + cap
        w = np.where((k == 0) | (k == M_P), 1.0, 2.0)
        d = p - pr
        if abs(pim) > T_LIM:
            T += at(p) @ (w / (d - 1j * pim)) - at(2.0 * pr - p) @ (w / (d + 1j * pim))
        else:
            fr = float(np.sum(w[1:] * d[1:] ** 2 / (d[1:] ** 2 + pim * pim)))
            T += (at(pr + dpz) - at(pr - dpz))[:, 0] / (2.0 * dpz) * 2.0 * fr
            T += 2j * math.pi / sm * np.sign(pim) * at(pr)[:, 0]
        ntiny = int((pz[upper] - pr - cap) / sm)
        if ntiny > 0:
            corr = ((pz[upper] - pr - cap) / ntiny) / sm
            k = np.arange(ntiny + 1)
            p = pr + cap + corr * sm * k
            w = np.where((k == 0) | (k == ntiny), 1.0, 2.0) * corr
            T += at(p) @ (w / (p - pr - 1j * pim))
        return T * (2.0 * math.pi * sm * t["dpp"] * 0.25 * (-s["qs"] / self.kpar * 0.5))

    def _chi_species(self, s, t, om):
        """chi (six entries) and its n = -1, 0, 1 parts for every frequency."""
        nom = len(om)
        chi = np.zeros((nom, 6), complex)
        low = np.zeros((3, nom, 6), complex)
        pz, dpz = s["pz"], t["dpz"]
        z = self.kperp / s["qs"]
        C0 = 2.0 * math.pi * t["dpp"] * dpz * 0.25 * s["qs"]
        for n in range(-t["nmax"], t["nmax"] + 1):
            pref = np.array([n * n / (z * z), 1.0, 1.0, 1j * n / z, n / z, -1j])
            keep = np.array([n != 0, True, True, n != 0, n != 0, True])
            x = (s["ms"] * om.real - n * s["qs"]) / self.kpar
            pim = s["ms"] * om.imag / self.kpar
            W = np.ones((nom, len(pz) - 2))
            W[:, 0] = W[:, -1] = 0.5
            res = np.nonzero((x > pz[1] - (M_I + 1) * dpz) & (x < pz[-1] + (M_I + 1) * dpz))[0]
            extra = np.zeros((nom, 6), complex)
            for i in res:
                resonant, a, b, window = self._window(pz, x[i], dpz)
                if not resonant:
                    continue
                W[i] = 0.0
                for r in (a, b):
                    if r is not None and r[0] <= r[1]:
                        W[i, r[0] - 1:r[1]] = 1.0
                        if r[0] < r[1]:
                            W[i, r[0] - 1] = W[i, r[1] - 1] = 0.5
                if window is not None:
                    extra[i] += self._principal(s, t, n, om[i], x[i], pim[i], window)
                if om[i].imag <= 0.0:
                    lf = 2.0 if om[i].imag < 0.0 else 1.0
                    extra[i] += lf * self._landau(s, t, n, om[i], x[i] + 1j * pim[i])
            den = (s["ms"] * om - n * s["qs"])[:, None] - self.kpar * pz[1:-1]
            S = (W / den) @ t["V"][abs(n)].reshape(12, -1).T
            X = om[:, None] * S[:, 0::2] + (self.kpar / s["ms"]) * S[:, 1::2]
            val = keep * pref * (C0 * X + extra)
            chi += val
            if abs(n) <= 1:
                low[n + 1] = val
        chi[:, 2] += t["ee"]
        low[1][:, 2] += t["ee"]
        f = s["ns"] * s["qs"]
        return chi * f, low * f

    def evaluate(self, om, tensors=False):
        om = np.atleast_1d(np.asarray(om, complex))
        parts = [self._chi_species(s, t, om) for s, t in zip(self.species, self.tabs)]
        eps = sum(p[0] for p in parts)
        unit = (om * V_A) ** 2
        kp, kz = self.kperp, self.kpar
        w11, w22 = eps[:, 0] + unit - kz * kz, eps[:, 1] + unit - kz * kz - kp * kp
        w33, w12, w13, w23 = eps[:, 2] + unit - kp * kp, eps[:, 3], eps[:, 4] + kz * kp, eps[:, 5]
        D = w11 * (w22 * w33 + w23 * w23) + 2.0 * w12 * w23 * w13 - w13 * w13 * w22 + w12 * w12 * w33
        if not tensors:
            return D

        def full(c):
            t = np.empty(c.shape[:-1] + (3, 3), complex)
            t[..., ROWS, COLS] = c
            t[..., 1, 0], t[..., 2, 0], t[..., 2, 1] = -c[..., 3], c[..., 4], -c[..., 5]
            return t

        chi0 = np.stack([full(p[0][0] / unit[0]) for p in parts])
        low = np.stack([full(p[1][:, 0] / unit[0]) for p in parts])
        return D, chi0, low, full(np.stack([w11, w22, w33, w12, w13, w23], axis=-1))[0]

    def root(self, guess):
        """The root a secant iteration from the guess runs into."""
        a, b = guess * (1.0 - 1e-5), guess
        fa, fb = self.evaluate([a, b])
        for _ in range(40):
            if fb == fa:
                break
            step = fb * (b - a) / (fb - fa)
            a, fa, b = b, fb, b - step
            if abs(step) <= 1e-13 * abs(b):
                break
            fb = self.evaluate([b])[0]
        return b


def _kscan_points(case):
    """(k_perp, k_par) of a logarithmic scan in k_par (type 4) or |k| (type 2)."""
    kp, kz = case["kperp"], case["kpar"]
    k0 = kz if case["type_s"] == 4 else math.hypot(kp, kz)
    f = [(case["end"] / k0) ** (i / case["steps"]) for i in range(case["steps"] + 1)]
    return [(kp if case["type_s"] == 4 else kp * x, kz * x) for x in f]


def _exact_scan(species, points, guess, bessel_zero):
    rows, w, N = [], guess, None
    for kp, kz in points:
        if N is not None and N.kperp == kp:
            N.kpar = kz
        else:
            N = _Numpy(species, kp, kz, bessel_zero)
        w = N.root(w)
        rows.append([kp, kz, w.real, w.imag])
    return np.array(rows)[:, None, :]


MOST = 3.0e8  # node terms that numpy sums in some ten seconds


def exact(case, seed):
    kind = case["kind"]
    if kind == "relativistic":
        return None  # its f0_rel is a dense spline system of its own
    if kind in ("solves", "served"):
        plasmas = _uneven(case, seed, case["plasmas"] if kind == "solves" else case["polishes"] + 2)
        tabs = [(s, c, g, _Numpy(s, c["kperp"], c["kpar"], c["bessel_zero"])) for c, s, g in plasmas]
        if kind == "solves":
            return {"roots": np.array([N.root(g) for _, _, g, N in tabs])}
        mp = _map(case["nr"], case["ni"], np.random.default_rng(seed + 1), plasmas[-1][0]["kpar"])
        D = tabs[-1][3].evaluate(_lattice(mp)) if tabs[-1][3].cost * mp.nr * mp.ni < MOST else None
        s, c, g, _ = tabs[-2]
        f, n = SERVED_SCAN["kpar_factor"], SERVED_SCAN["steps"]
        rows = _exact_scan(s, [(c["kperp"], c["kpar"] * f ** (i / n)) for i in range(n + 1)], g, c["bessel_zero"])
        return {"roots": np.array([N.root(g) for _, _, g, N in tabs[:-2]]), "rows": rows[1:],
                "cal": D, "val": None if D is None else np.log10(np.abs(D))}
    species, rng = _plasma_of(case, seed)
    if kind == "scan":
        return {"rows": _exact_scan(species, _kscan_points(case),
                                    _alfven_guess(species, case["kperp"], case["kpar"]), case["bessel_zero"])}
    N = _Numpy(species, case["kperp"], case["kpar"], case["bessel_zero"])
    if kind == "tensor":
        D, chi0, low, wave = N.evaluate(_frequencies(rng, 1, case["kpar"]), tensors=True)
        return {"D": D, "chi0": chi0, "chi0_low": low, "wave": wave}
    if kind == "batch":
        return {"D": N.evaluate(_frequencies(rng, case["n"], case["kpar"]))} if N.cost * case["n"] < MOST else None
    if kind == "map":
        om = _lattice(_map(case["nr"], case["ni"], rng, case["kpar"]))
        if N.cost * len(om) >= MOST:
            return {"om": om, "cal": None, "val": None}
        D = N.evaluate(om)
        return {"om": om, "cal": D, "val": np.log10(np.abs(D))}
    # setup: the tables are the continuation's own function, so the fit of
    # every row is the table's parameters
    rng.uniform(0.02, 0.03)
    fits = [np.tile(s["fit"], (len(s["pp"]), 1)).ravel() if s["ftype"] == 2 else
            np.tile(np.array(s["fit"][:3] + [0.0, 0.0]), (len(s["pp"]), 1)).ravel() for s in species]
    return {"fits": fits, "nmax": np.array([t["nmax"] for t in N.tabs]),
            "D": N.evaluate(_frequencies(rng, 3, case["kpar"]))}
