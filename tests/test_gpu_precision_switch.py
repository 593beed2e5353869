"""One handle that changes precision shares its work buffers between the plans of three
and six slices: whatever ran before, each precision gives the bits of a handle of
its own, also in the loop whose last iteration is FP64."""
import numpy as np
import pytest

from _helpers import crystal

pytestmark = pytest.mark.gpu


def _solver(precision):
    from mbsymmetry_gb300.solver import GWSolver
    cr, tr = crystal("C2")
    s = GWSolver(cr.layout, cr.ns, tr, precision=precision)
    s.set_shared_Coulomb(cr.V)
    s.set_fock(cr.F, cr.S)
    return cr, s


def _iterate(cr, s):
    s.set_Selfenergy(np.zeros(s.g_size, np.complex128))
    s.dyson(cr.mu)
    s.iteration(cr.mu)
    return s.Selfenergy(), s.G_tau()


def _loop(cr, s, final):
    s.set_Selfenergy(np.zeros(s.g_size, np.complex128))
    s.dyson(cr.mu)
    recs = s.sc_loop(3, 0.5, float(cr.layout.nao), cr.mu, tol=1e-10, max_evals=24, final_fp64=final)
    return recs, s.Selfenergy()


def test_precisions_in_turn_on_one_handle():
    ref = {}
    for p in ("fp64", "ozaki"):
        cr, s = _solver(p)
        ref[p] = _iterate(cr, s)
        if p == "ozaki":
            loop = _loop(cr, s, True)
        s.close()
    cr, s = _solver("fp64")
    for p in ("fp64", "ozaki", "fp64", "ozaki"):
        s.single_prec_run(p == "ozaki")
        assert all(np.array_equal(a, b) for a, b in zip(ref[p], _iterate(cr, s))), p
    recs, sig = _loop(cr, s, True)
    assert recs == loop[0] and np.array_equal(sig, loop[1])
    assert [r["precision"] for r in recs] == [3, 3, 0]
    assert all(np.array_equal(a, b) for a, b in zip(ref["ozaki"], _iterate(cr, s)))
    s.close()
