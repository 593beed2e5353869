"""The sliced contractions against the FP64 oracle, relative to the results.

Meshes: within 1e-8 (three slices: 2^-32 of a row's scale, three operands in a chain,
sums of a few hundred terms) and 1e-12 (six) of the largest element, however small that
is; nothing but zeros where no V block couples.

One k point, V graded (every element by its own power of ten down to 10^-8, a third of
them zero): element by element, within the bound that the arithmetic has.  A component
is held to e = 1.13 x 2^-32 (2^-56 at worst) of the power of two above its row's largest one, so a
complex operand to sqrt(2) 2 e of that, a product to 5.7 e and a chain of three to 18 e of
the largest elements' product: a V block with largest element v and G blocks with g1, g2 adds to
an element of P0[Q][P] no more than 2 x 18 e b1^2 b2^2 g1 g2 v^2, and to one of Sigma
18 e qb^2 b2^2 g p v^2.  The oracle's own rounding, 2^-53 a product, is covered by 2^-53 in
e.  Three slices in the place of six would exceed the bound of six."""
import numpy as np
import pytest

from oracle import Oracle

pytestmark = pytest.mark.gpu
EPS = {"ozaki": 1.13 * 2.0 ** -32 + 2.0 ** -53, "fp64": 2.0 ** -56 + 2.0 ** -53}


def _run(precision, monkeypatch, lattice, mesh, nao, naux, ao, aux, ns, seed, graded=False):
    from mbsymmetry_gb300.crystal import CrystalSpec, load_ir, make_crystal
    from mbsymmetry_gb300.solver import GWSolver
    from mbsymmetry_gb300.transformer import build_transforms
    monkeypatch.setenv("GWGB_FP64_SLICES", "1")
    cr = make_crystal(CrystalSpec("bound", lattice, mesh, nao, naux, 62, 50.0, ns=ns, ao_block=ao, aux_block=aux,
                                  seed=seed))
    if graded:
        rng = np.random.default_rng(seed)
        cr.V *= np.where(rng.random(cr.V.size) < 1 / 3, 0.0, 10.0 ** -rng.uniform(0, 8, size=cr.V.size))
    tr = build_transforms(load_ir(62), 50.0)
    orc = Oracle(cr.layout, ns, tr.nts)
    G0, _ = orc.dyson(np.zeros(tr.nts * ns * cr.layout.flat_ao_size, np.complex128), cr.F, cr.S, tr, cr.mu)
    ref, P0, Pt = orc.gw_sigma(G0, cr.V, tr)
    s = GWSolver(cr.layout, ns, tr, precision=precision)
    s.set_shared_Coulomb(cr.V)
    s.set_fock(cr.F, cr.S)
    s.set_G(G0)
    s.solve_P0()
    P = s.P0_q_t_QP()
    s.set_P0(Pt)
    s.solve_sigma_from_P()
    S = s.Selfenergy()
    s.close()
    return cr, tr, G0, Pt, (P0, P), (ref, S)


@pytest.mark.parametrize("precision,tol", [("ozaki", 1e-8), ("fp64", 1e-12)])
@pytest.mark.parametrize("lattice,mesh,nao,naux,ao,aux,ns", [
    ("fcc", (1, 1, 1), 1, 1, (1, 1), (1, 1), 1),
    ("fcc", (2, 2, 2), 3, 7, (1, 1), (1, 7), 2),
    ("hex", (2, 2, 1), 17, 33, (1, 9), (2, 33), 2),
    ("hex", (1, 1, 2), 33, 96, (31, 33), (31, 33), 1),
])
def test_relative_to_the_largest_element(precision, tol, lattice, mesh, nao, naux, ao, aux, ns, monkeypatch):
    *_, p, s = _run(precision, monkeypatch, lattice, mesh, nao, naux, ao, aux, ns, 7)
    for ref, got in (p, s):
        m = np.abs(ref).max()
        assert np.abs(got - ref).max() <= tol * m


@pytest.mark.parametrize("precision", ["ozaki", "fp64"])
@pytest.mark.parametrize("nao,naux,ao,aux,seed", [(17, 60, (1, 9), (2, 40), 1), (24, 34, (7, 9), (16, 17), 7),
                                                  (40, 64, (3, 8), (2, 9), 4)])
def test_graded_data_element_by_element(precision, nao, naux, ao, aux, seed, monkeypatch):
    cr, tr, G0, Pt, (P0, P), (ref, S) = _run(precision, monkeypatch, "fcc", (1, 1, 1), nao, naux, ao, aux, 1, seed, True)
    L, nts, e = cr.layout, tr.nts, EPS[precision]
    half = nts // 2
    g = [np.abs(G0.reshape(nts, -1)[:, o:o + n * n]).max(1) for n, o in zip(L.ao_sizes[0], L.ao_offsets[0])]
    p = [np.abs(Pt.reshape(nts, -1)[:, o:o + n * n]).max(1) for n, o in zip(L.aux_sizes[0], L.aux_offsets[0])]
    bp, bs = np.zeros((half, P0.size // nts)), np.zeros((nts, ref.size // nts))
    for b, (iq, i1, i2) in enumerate(L.tensor_irreps[0]):
        qb, b1, b2 = (int(x) for x in (L.aux_sizes[0][iq], L.ao_sizes[0][i1], L.ao_sizes[0][i2]))
        o = int(L.kpair_slice_offsets[0] + L.tensor_offsets[0][b])
        v = np.abs(cr.V[o:o + qb * b1 * b2]).max()
        at, to = int(L.aux_offsets[0][iq]), int(L.ao_offsets[0][i1])
        bp[:, at:at + qb * qb] += (36 * e * (b1 * b2 * v) ** 2 * g[i1][::-1][:half] * g[i2][:half])[:, None]
        bs[:, to:to + b1 * b1] += (18 * e * (qb * b2 * v) ** 2 * g[i2] * p[iq])[:, None]
    assert L.tensor_irreps[0].size and bp.max() > 0
    for got, want, bound in ((P.reshape(nts, -1)[:half], P0.reshape(nts, -1)[:half], bp),
                             (S.reshape(nts, -1), ref.reshape(nts, -1), bs)):
        off = np.abs(got - want)
        print(f"{precision}: largest error / bound {(off[bound > 0] / bound[bound > 0]).max():.1e}")
        assert (off <= bound).all()
