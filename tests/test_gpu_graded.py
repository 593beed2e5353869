"""What the FP64 contractions guarantee on graded data.  In one AO block of two, V is
zero for the first orbital on one side, where G is one, and G is 2^-40 / 3 where V is
not: every term of P0 and Sigma is then 2^-40 below the product of its rows' largest
elements.

In FMAs (GWGB_FLAG_FP64_FMA) each element keeps its own bits: at most 12 additions and
products in a chain, 24 units of 1.1e-16 of the (here equal-signed) sum, taken as 1e-14.
In slices an operand is held to 2^-57 of its row, which leaves 17 bits of the small
one: the error stays below 2^-53 of the row scales' product, that is 2^-53 / (2^-40 / 3)
times a few (taken as 8) of the result, 3e-3."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fma,slices,tol", [(True, "1", 1e-14), (False, "0", 1e-14), (False, "1", 3e-3)])
def test_sums_far_below_their_rows_scales(fma, slices, tol, monkeypatch):
    from mbsymmetry_gb300.crystal import CrystalSpec, load_ir, make_crystal
    from mbsymmetry_gb300.solver import GWSolver
    from mbsymmetry_gb300.transformer import build_transforms
    monkeypatch.setenv("GWGB_FP64_SLICES", slices)
    cr = make_crystal(CrystalSpec("graded", "fcc", (1, 1, 1), 2, 2, 62, 50.0, ao_block=(2, 2), aux_block=(2, 2),
                                  seed=2))
    tr = build_transforms(load_ir(62), 50.0)
    nts, small = tr.nts, 2.0 ** -40 / 3
    v = np.zeros((2, 2, 2))
    v[:, :, 1] = [[1 / 7, 1 / 3], [1 / 5, 1 / 9]]
    g = np.array([[1.0, 1.0], [1.0, small]])
    P = np.ones((2, 2)) * [[1 / 3, 1 / 11], [1 / 13, 1 / 17]]
    s = GWSolver(cr.layout, 1, tr, fp64_fma=fma)
    s.set_shared_Coulomb(v.ravel().astype(np.complex128))
    s.set_fock(cr.F, cr.S)
    s.set_G(np.tile(g.ravel(), nts).astype(np.complex128))
    s.solve_P0()
    P0 = s.P0_q_t_QP().reshape(nts, 2, 2)[: nts // 2]
    s.set_P0(np.tile(P.ravel(), nts).astype(np.complex128))
    s.solve_sigma_from_P()
    S = s.Selfenergy().reshape(nts, 2, 2)
    s.close()
    L = np.longdouble
    G, V = g.astype(L), v.astype(L)
    # P0[Q][P] = -2 sum G[t][p] V[Q][p][m] G[m][n] V[P][t][n]; Sigma[i][j] = -sum V[Q][i][m] G[m][n] P[Q][P] V[P][j][n]
    p0 = -2 * np.einsum("tp,Qpm,mn,Ptn->QP", G, V, G, V)
    sg = -np.einsum("Qim,mn,QP,Pjn->ij", V, G, P.astype(L), V)
    assert np.abs(p0).max() < 8 * small and np.abs(sg).max() < 8 * small
    assert (np.abs(P0 - p0) < tol * np.abs(p0)).all()
    assert (np.abs(S - sg) < tol * np.abs(sg)).all()


def test_flag_keeps_the_transforms_in_fp64():
    """C2's sizes, where contractions and transforms run in slices without the flag: the
    same iteration to rounding, without lists or images."""
    from _helpers import crystal
    from mbsymmetry_gb300.solver import GWSolver
    cr, tr = crystal("C2")
    out, held = [], []
    for fma in (False, True):
        s = GWSolver(cr.layout, cr.ns, tr, fp64_fma=fma)
        s.set_shared_Coulomb(cr.V)
        s.set_fock(cr.F, cr.S)
        s.set_Selfenergy(np.zeros(s.g_size, np.complex128))
        s.dyson(cr.mu)
        before = s.stats()["device_bytes"]
        s.iteration(cr.mu)
        held.append(s.stats()["device_bytes"] - before)
        assert bool(s.launch_stats()) != fma
        out.append((s.Selfenergy(), s.G_tau()))
        s.close()
    assert held[0] > held[1] == 0
    for a, b in zip(*out):
        assert np.abs(a - b).max() < 1e-10 * np.abs(b).max()
