"""determine_nmax's decisions are the oracle's, from answers of 1 to several
hundred (past the first chunk of 128 orders) and cutoffs from 0.1 to 1e-300,
on both sides of the estimate's range."""
import numpy as np
import pytest

from alps_gb300 import workloads
from test_gpu_parity import _oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bz", [1e-1, 1e-3, 1e-14, 1e-50, 1e-300])
def test_nmax_decisions(bz):
    from alps_gb300 import api
    po = _oracle()
    w = workloads.proton_electron(40, 24, 1.0, 0.3, bz)
    system, species = workloads.build(w, po.generate_f0)
    O = po.OraclePlasma(system, species)
    G = api.Plasma(system, species, precision="fp64")
    for kperp in np.concatenate([np.geomspace(1e-3, 12.0, 24), [30.0]]):
        O.set_k(kperp, 0.3)
        G.set_k(kperp, 0.3)
        assert O.nmax() == G.nmax(), kperp
