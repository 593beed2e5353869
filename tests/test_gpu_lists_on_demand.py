"""The work lists of the sliced contractions are built with the first contraction
of a crystal of ordinary size: a handle that only solves Dyson and W~ holds none."""
import numpy as np
import pytest

from _helpers import crystal

pytestmark = pytest.mark.gpu


def test_dyson_and_screening_hold_no_lists():
    from mbsymmetry_gb300.solver import GWSolver
    cr, tr = crystal("C2")
    s = GWSolver(cr.layout, cr.ns, tr)
    before = s.stats()["device_bytes"]
    s.set_shared_Coulomb(cr.V)
    s.set_fock(cr.F, cr.S)
    s.set_Selfenergy(np.zeros(s.g_size, np.complex128))
    s.dyson(cr.mu)
    s.set_P0(np.zeros(s.p_size, np.complex128))
    s.compute_Pq_from_P0q()
    assert s.stats()["device_bytes"] == before and not s.launch_stats()
    s.solve()
    assert s.stats()["device_bytes"] > before and s.launch_stats()
    s.close()
