"""The sliced contractions (three slices: precision "ozaki"; six: precision
"fp64") at the block sizes where their tiles can go wrong: octets of 8 columns
(7, 8, 9), the pairs and quadruples of row tiles that share an accumulator set
(1, 16, 17), rounds of 32 complex K (31, 32, 33) and the largest blocks (AO 40,
aux 64), no contribution at all (1 x 1), for AO and aux blocks alike, with
time-reversal partners and both spins; and on graded data (every V element by
its own power of ten down to 10^-8, a third of them
zero), where sums lie in the low slices alone.  Reference: the FP64 oracle.

A three-slice operand is held to 2^-32 of its row's scale and a chain has
three of them, so Sigma agrees to 1e-8 of its largest element (2^-32 times the
ratio of row scale to element, times the square root of a few hundred terms);
six slices are held to 2^-56, FP64 itself to 2^-53 per operation: 1e-12."""
import numpy as np
import pytest

from oracle import Oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["ozaki", "fp64"])
@pytest.mark.parametrize("lattice,mesh,nao,naux,ao,aux,ns,seed,graded", [
    ("fcc", (1, 1, 1), 1, 1, (1, 1), (1, 1), 1, 7, False),
    ("fcc", (2, 2, 2), 3, 7, (1, 1), (1, 7), 2, 7, False),
    ("fcc", (1, 1, 1), 24, 34, (7, 9), (16, 17), 1, 7, False),
    ("hex", (2, 2, 1), 17, 33, (1, 9), (2, 33), 2, 7, False),
    ("fcc", (1, 1, 1), 33, 64, (16, 17), (31, 33), 1, 7, False),
    ("hex", (1, 1, 2), 33, 96, (31, 33), (31, 33), 1, 7, False),
    ("fcc", (1, 1, 1), 40, 64, (40, 40), (64, 64), 1, 2, False),
    ("fcc", (1, 1, 1), 5, 128, (2, 3), (64, 64), 2, 7, False),
    ("hex", (2, 2, 1), 17, 60, (1, 9), (2, 40), 1, 7, True),
])
def test_sliced_sigma_at_tile_edges(precision, lattice, mesh, nao, naux, ao, aux, ns, seed, graded, monkeypatch):
    from mbsymmetry_gb300.crystal import CrystalSpec, load_ir, make_crystal
    from mbsymmetry_gb300.solver import GWSolver
    from mbsymmetry_gb300.transformer import build_transforms
    monkeypatch.setenv("GWGB_FP64_SLICES", "1")  # also where the FP64 kernels would be the faster ones
    cr = make_crystal(CrystalSpec("edge", lattice, mesh, nao, naux, 62, 50.0, ns=ns, ao_block=ao, aux_block=aux,
                                  seed=seed))
    if graded:
        rng = np.random.default_rng(seed)
        cr.V *= np.where(rng.random(cr.V.size) < 1 / 3, 0.0, 10.0 ** -rng.uniform(0, 8, size=cr.V.size))
    tr = build_transforms(load_ir(62), 50.0)
    orc = Oracle(cr.layout, ns, tr.nts)
    zero = np.zeros(tr.nts * ns * cr.layout.flat_ao_size, np.complex128)
    G0, _ = orc.dyson(zero, cr.F, cr.S, tr, cr.mu)
    ref, P0, _ = orc.gw_sigma(G0, cr.V, tr)
    s = GWSolver(cr.layout, ns, tr, precision=precision)
    s.set_shared_Coulomb(cr.V)
    s.set_fock(cr.F, cr.S)
    s.set_G(G0)
    s.solve_P0()
    P = s.P0_q_t_QP()
    s.solve()
    S = s.Selfenergy()
    s.close()
    tol = 1e-8 if precision == "ozaki" else 1e-12
    assert np.abs(P - P0).max() < tol * max(1.0, np.abs(P0).max())
    assert np.abs(S - ref).max() < tol * max(1.0, np.abs(ref).max())
