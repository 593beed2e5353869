"""The batched block inverses at the block sizes where they can go wrong (1, one
warp per block up to 16, one CTA above, odd and even, the largest), on both
paths of the W~ solve (positive definite blocks: symmetric sweeps; indefinite
ones: the pivoted elimination) and on Dyson blocks without a dominant diagonal.
Reference: the FP64 oracle.

An inverse carries n eps kappa of its largest element, a transform multiplies
that by its row sums (below 100 on these grids): 64 * 100 * 1.1e-16 kappa, taken
as 1e-12 kappa."""
import numpy as np
import pytest

from oracle import Oracle

pytestmark = pytest.mark.gpu

SIZES = [(1, 1), (2, 3), (15, 16), (16, 17), (31, 33), (40, 40), (63, 64)]


def _crystal(ao, aux):
    from mbsymmetry_gb300.crystal import CrystalSpec, load_ir, make_crystal
    from mbsymmetry_gb300.transformer import build_transforms
    nao, naux = max(2, sum(ao)), 2 * aux[1]
    cr = make_crystal(CrystalSpec("inv", "fcc", (1, 1, 1), nao, naux, 62, 50.0, ao_block=ao, aux_block=aux, seed=5))
    return cr, build_transforms(load_ir(62), 50.0)


@pytest.mark.parametrize("definite", [True, False])
@pytest.mark.parametrize("aux", SIZES)
def test_screened_blocks(aux, definite):
    from mbsymmetry_gb300.solver import GWSolver
    cr, tr = _crystal((1, 2), aux)
    L, nts, rng = cr.layout, tr.nts, np.random.default_rng(11)
    P0 = np.zeros(nts * L.flat_aux_size, np.complex128)
    w = np.exp(-np.abs(np.arange(nts) - (nts - 1) / 2) / 8.0)  # even in tau
    kappa = 1.0
    for iq in range(L.ink):
        o, sz = L.qaux_slice_offsets_irre[iq], L.qaux_slice_sizes_irre[iq]
        blk = P0[nts * o: nts * (o + sz)].reshape(nts, sz)
        at = 0
        for n in L.aux_sizes[L.irre_list[iq]]:
            q, _ = np.linalg.qr(rng.normal(size=(n, n)) + 1j * rng.normal(size=(n, n)))
            ev = rng.uniform(0.1, 1.0, n) * (-0.2 if definite else rng.choice([-0.2, 0.2], n))
            blk[:, at: at + n * n] = w[:, None] * ((q * ev) @ q.conj().T).ravel()
            # 1 - P(i Omega) has the eigenvalues 1 - c(Omega) ev
            lam = 1.0 - np.real(tr.Tnt_BF @ w[1: 1 + tr.Tnt_BF.shape[1]])[:, None] * ev
            kappa = max(kappa, np.abs(lam).max() / np.abs(lam).min())
            at += n * n
    ref = Oracle(L, 1, nts).p_tilde(P0, tr)
    s = GWSolver(L, 1, tr)
    s.set_shared_Coulomb(cr.V)
    s.set_fock(cr.F, cr.S)
    s.set_P0(P0)
    s.compute_Pq_from_P0q()
    got = s.P0_q_t_QP()
    s.close()
    assert np.abs(got - ref).max() < 1e-12 * kappa * np.abs(ref).max()


@pytest.mark.parametrize("ao", [a for a in SIZES if a[1] <= 40])
def test_dyson_blocks(ao):
    from mbsymmetry_gb300.solver import GWSolver
    cr, tr = _crystal(ao, (1, 2))
    L, nts, rng = cr.layout, tr.nts, np.random.default_rng(12)
    sig = (rng.normal(size=nts * L.flat_ao_size) + 1j * rng.normal(size=nts * L.flat_ao_size)) * 0.5
    ref, _ = Oracle(L, 1, nts).dyson(sig, cr.F, cr.S, tr, cr.mu)
    s = GWSolver(L, 1, tr)
    s.set_shared_Coulomb(cr.V)
    s.set_fock(cr.F, cr.S)
    s.set_Selfenergy(sig)
    s.dyson(cr.mu)
    got = s.G_tau()
    s.close()
    assert np.abs(got - ref).max() < 1e-9 * np.abs(ref).max()  # kappa up to 10^3
