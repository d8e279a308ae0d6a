"""The Gamma-row integrals of a relativistic species at the sizes where their
device form changes: numbers of principal-value samples below, at and above a
warp's chunk of 128, windows whose pieces fill more than one round of 32
lanes, odd grids, more Gamma rows per block than a warp decides at once; each
against the oracle at the relativistic gate (1e-8 of the entry's scale).
"""
import pytest

from test_gpu_relativistic import _check_disp, _limit_case, _pair

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M_I,M_P,ngamma,npparbar", [(3, 7, 60, 84), (3, 127, 60, 80), (3, 128, 60, 80), (3, 300, 64, 90),
                                                     (1, 100, 150, 64), (17, 100, 60, 240)])
def test_rows_against_oracle(M_I, M_P, ngamma, npparbar):
    from alps_gb300 import api
    sysd, species = _limit_case()
    sysd.positions_principal, sysd.n_resonance_interval = M_I, M_P
    sysd.ngamma, sysd.npparbar = ngamma, npparbar
    O, G = _pair(api, sysd, species)
    assert G.nmax() == O.nmax()
    for om in [0.5 + 0.1j, 1.2 + 0.05j, 0.9 - 0.05j, 1.1 + 0.001j, 2.5 - 0.3j]:
        _check_disp(O, G, om)
