"""Column tiles of one to four octets next to one another in a CTA's task list,
one row tile each: the drain warps exchange row maxima for three and four octets
only, so tiles with and without an exchange alternate.  Both contractions in three
slices, six runs, bitwise the same and within 1e-8 of the largest element of the
FP64 oracle's result (operands to 2^-32 of a row's scale, three of them in a chain)."""
import numpy as np
import pytest

from oracle import Oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lattice,mesh,nao,naux,ao,aux", [
    ("fcc", (2, 2, 2), 12, 150, (1, 2), (2, 33)),    # Sigma, stage 1: 2 rows of L, aux octets 1 to 5
    ("hex", (2, 2, 1), 60, 40, (2, 33), (1, 4)),     # P0, stage 1: AO octets 1 to 5
])
def test_mixed_widths_are_reproducible(lattice, mesh, nao, naux, ao, aux):
    from mbsymmetry_gb300.crystal import CrystalSpec, load_ir, make_crystal
    from mbsymmetry_gb300.solver import GWSolver
    from mbsymmetry_gb300.transformer import build_transforms
    cr = make_crystal(CrystalSpec("mixed", lattice, mesh, nao, naux, 62, 50.0, ao_block=ao, aux_block=aux, seed=3))
    widths = {-(-int(n) // 8) for x in (cr.layout.ao_sizes if ao[1] > aux[1] else cr.layout.aux_sizes) for n in x}
    assert min(widths) <= 2 < max(widths)
    tr = build_transforms(load_ir(62), 50.0)
    orc = Oracle(cr.layout, 1, tr.nts)
    G0, _ = orc.dyson(np.zeros(tr.nts * cr.layout.flat_ao_size, np.complex128), cr.F, cr.S, tr, cr.mu)
    ref, P0, _ = orc.gw_sigma(G0, cr.V, tr)
    s = GWSolver(cr.layout, 1, tr, precision="ozaki")
    s.set_shared_Coulomb(cr.V)
    s.set_fock(cr.F, cr.S)
    out = []
    for _ in range(6):
        s.set_G(G0)
        s.solve_P0()
        P = s.P0_q_t_QP()
        s.solve()
        out.append((P, s.Selfenergy()))
    s.close()
    assert all(np.array_equal(p, out[0][0]) and np.array_equal(x, out[0][1]) for p, x in out)
    assert np.abs(out[0][0] - P0).max() < 1e-8 * np.abs(P0).max()
    assert np.abs(out[0][1] - ref).max() < 1e-8 * np.abs(ref).max()
