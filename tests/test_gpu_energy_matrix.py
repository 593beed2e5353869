"""The Galitskii-Migdal matrix may be set again between self-consistent loops:
the loop's captured graph is kept, so the matrix's device copies (values,
slice images and their scales) must be replaced in place.  C2's sizes, where
the M G product runs on slice images; the column scales of the second matrix
differ from the first one's.  The records equal, bit for bit, those of a handle
that only ever saw the matrix."""
import numpy as np
import pytest

from _helpers import crystal
from mbsymmetry_gb300 import _abi
from mbsymmetry_gb300.transformer import gm_matrix

pytestmark = pytest.mark.gpu


def _solver(cr, tr):
    from mbsymmetry_gb300.solver import GWSolver
    s = GWSolver(cr.layout, 1, tr)
    s.set_shared_Coulomb(cr.V)
    s.set_fock(cr.F, cr.S)
    return s


def _set_matrix(s, M):
    _abi.check(s.lib.gwgb_set_energy_matrix(s.h, M.ctypes.data, M.shape[0]))


def _loop(s, cr, G0):
    s.set_G(G0)
    s.set_Selfenergy(np.zeros(s.g_size, np.complex128))
    return s.sc_loop(2, 0.5, float(cr.layout.nao), cr.mu, tol=1e-10, max_evals=24)


def test_energy_matrix_set_again_keeps_the_graph_valid():
    cr, tr = crystal("C2")
    M1 = np.ascontiguousarray(gm_matrix(tr))
    M2 = np.ascontiguousarray(M1 * 2.0 ** (np.arange(M1.shape[0]) % 9 - 4.0))
    s = _solver(cr, tr)
    s.set_Selfenergy(np.zeros(s.g_size, np.complex128))
    s.dyson(cr.mu)
    G0 = s.G_tau()
    got = []
    for M in (M1, M2, M1):
        _set_matrix(s, M)
        other = _solver(cr, tr)  # takes device memory that a call may have given back
        got.append(_loop(s, cr, G0))
        other.close()
    s.close()
    ref = []
    for M in (M1, M2):
        f = _solver(cr, tr)
        _set_matrix(f, M)
        ref.append(_loop(f, cr, G0))
        f.close()
    assert got[0] == ref[0] and got[1] == ref[1] and got[2] == ref[0]
    assert ref[0][0]["e_corr"] != ref[1][0]["e_corr"]
