"""The sliced contractions at the block sizes where their tiles can go wrong:
octets of 8 columns (7, 8, 9), the pairs and quadruples of row tiles that share
an accumulator set (1, 16, 17), rounds of 32 complex K (31, 32, 33) and the
largest blocks (AO 40, aux 64), no contribution at all (1 x 1), for AO and aux blocks alike, with time-reversal partners and
both spins.  Reference: the FP64 oracle.  A slice leaves at most 2^-32 of its
row's scale and a chain has three of them, so Sigma agrees to 1e-8 of its
largest element (2^-32 times the ratio of row scale to element, times the square
root of a few hundred terms)."""
import numpy as np
import pytest

from oracle import Oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lattice,mesh,nao,naux,ao,aux,ns,seed", [
    ("fcc", (1, 1, 1), 1, 1, (1, 1), (1, 1), 1, 7),
    ("fcc", (2, 2, 2), 3, 7, (1, 1), (1, 7), 2, 7),
    ("fcc", (1, 1, 1), 24, 34, (7, 9), (16, 17), 1, 7),
    ("hex", (2, 2, 1), 17, 33, (1, 9), (2, 33), 2, 7),
    ("fcc", (1, 1, 1), 33, 64, (16, 17), (31, 33), 1, 7),
    ("hex", (1, 1, 2), 33, 96, (31, 33), (31, 33), 1, 7),
    ("fcc", (1, 1, 1), 40, 64, (40, 40), (64, 64), 1, 2),
    ("fcc", (1, 1, 1), 5, 128, (2, 3), (64, 64), 2, 7),
])
def test_sliced_sigma_at_tile_edges(lattice, mesh, nao, naux, ao, aux, ns, seed):
    from mbsymmetry_gb300.crystal import CrystalSpec, load_ir, make_crystal
    from mbsymmetry_gb300.solver import GWSolver
    from mbsymmetry_gb300.transformer import build_transforms
    cr = make_crystal(CrystalSpec("edge", lattice, mesh, nao, naux, 62, 50.0, ns=ns, ao_block=ao, aux_block=aux,
                                  seed=seed))
    tr = build_transforms(load_ir(62), 50.0)
    orc = Oracle(cr.layout, ns, tr.nts)
    zero = np.zeros(tr.nts * ns * cr.layout.flat_ao_size, np.complex128)
    G0, _ = orc.dyson(zero, cr.F, cr.S, tr, cr.mu)
    ref, P0, _ = orc.gw_sigma(G0, cr.V, tr)
    s = GWSolver(cr.layout, ns, tr, precision="ozaki")
    s.set_shared_Coulomb(cr.V)
    s.set_fock(cr.F, cr.S)
    s.set_G(G0)
    s.solve_P0()
    P = s.P0_q_t_QP()
    s.solve()
    S = s.Selfenergy()
    s.close()
    assert np.abs(P - P0).max() < 1e-8 * max(1.0, np.abs(P0).max())
    assert np.abs(S - ref).max() < 1e-8 * max(1.0, np.abs(ref).max())
