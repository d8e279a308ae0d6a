"""Mixed batches of 2560 frequencies and more whose resonant orders the
item-per-lane form does not take: 128 principal-value samples and more, or as
many in the window's tiny rest.  They are summed as in a smaller batch, in
double-float by warps: a frequency's det D is the same bit for bit at 2559 and
2560 frequencies.  (Growing frequencies: the Landau terms stay out of it.)
"""
import numpy as np
import pytest

from alps_gb300 import workloads

pytestmark = pytest.mark.gpu


def _plasma(M_I, M_P, kpar):
    from alps_gb300 import api
    w = workloads.proton_electron(24, 48, 1.0, kpar, 1e-14)
    w["system"].positions_principal = M_I
    w["system"].n_resonance_interval = M_P
    w["system"].nspec = 1
    w["dists"], w["species"] = w["dists"][:1], w["species"][:1]
    system, species = workloads.build(w, api.generate_f0)
    G = api.Plasma(system, species, precision="mixed")
    G.set_k(1.0, kpar)
    return G


@pytest.mark.parametrize("M_P", [128, 1000])
def test_many_samples(M_P):
    G = _plasma(3, M_P, 0.3)
    rng = np.random.default_rng(5)
    om = rng.uniform(-2.5, 2.5, 2560) + 1j * rng.uniform(1e-4, 0.2, 2560)
    small = G.disp_batch(om[:2559])
    launched = G.stats().kernels_launched
    assert np.array_equal(G.disp_batch(om)[:2559], small)
    assert G.stats().kernels_launched == launched  # no pass that leaves everything


def test_many_samples_in_the_tiny_rest():
    """A window of the one interval around the pole, the pole between 0.06 and
    0.29 of a spacing above its node: the rest of the interval takes (1 - 2 f)/f
    times the 127 samples, 184 and more.  Every order of a frequency lies at
    the same place between nodes (16 spacings apart)."""
    G = _plasma(0, 127, 0.25)
    rng = np.random.default_rng(6)
    om = (rng.integers(3, 14, 2560) + rng.uniform(0.06, 0.29, 2560)) / 16.0
    om = om + 1j * rng.choice([1e-3, 0.01, 0.05], 2560)
    assert np.array_equal(G.disp_batch(om)[:2559], G.disp_batch(om[:2559]))
