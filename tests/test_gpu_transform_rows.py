"""The tau <-> omega transforms in slices against those in FP64 FMAs (a handle with
fp64_fma), both against extended precision, tau by tau: towards the middle of the axis
G and P~ fall by many orders of magnitude, and an error relative to the largest row
would be all there is.  W~ with |P0| of 10^-20, so that the solve is the identity and
the two transforms remain, and Dyson, whose inverses are the same on both sides.
Slices are to be no further off: 2-norm and the worst row, with a margin of 1.5 for the
scatter of single roundings."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
CL = np.clongdouble


def _crystal():
    from mbsymmetry_gb300.crystal import CrystalSpec, load_ir, make_crystal
    from mbsymmetry_gb300.transformer import build_transforms
    cr = make_crystal(CrystalSpec("rows", "fcc", (1, 1, 1), 48, 50, 120, 100.0, ao_block=(14, 18), aux_block=(16, 17),
                                  seed=7))
    return cr, build_transforms(load_ir(120), 100.0)


def _measures(got, ref):
    e = np.abs(got.reshape(ref.shape) - ref)
    rows = (e.max(1) / np.abs(ref).max(1)).astype(float)
    return float(np.sqrt((e ** 2).sum() / (np.abs(ref) ** 2).sum())), float(rows.max())


def _compare(run, ref):
    from mbsymmetry_gb300.solver import GWSolver
    cr, tr = _crystal()
    m = []
    for fma in (False, True):
        s = GWSolver(cr.layout, 1, tr, fp64_fma=fma)
        s.set_shared_Coulomb(cr.V)
        s.set_fock(cr.F, cr.S)
        m.append(_measures(run(s, cr), ref))
        s.close()
    (n6, r6), (n64, r64) = m
    print(f"2-norm {n6:.2e} (FMAs {n64:.2e}), worst row {r6:.2e} ({r64:.2e})")
    assert n6 < 1.5 * n64 and r6 < 1.5 * r64


def test_screening_rows():
    cr, tr = _crystal()
    L, nts, rng = cr.layout, tr.nts, np.random.default_rng(1)
    tau = np.asarray(tr.tau_fermi)
    assert 8.0 * (nts - 2) * tr.nw_b * L.flat_aux_size > 4e7
    P0 = np.zeros((nts, L.flat_aux_size), np.complex128)
    for n, o in zip(L.aux_sizes[0], L.aux_offsets[0]):
        for w in rng.uniform(0.3, 3.0, size=3):
            x = rng.normal(size=(n, n)) + 1j * rng.normal(size=(n, n))
            shape = (np.exp(-tau * w) + np.exp(-(tr.beta - tau) * w)) / (1.0 - np.exp(-tr.beta * w))
            P0[:, o:o + n * n] -= 1e-20 * shape[:, None] * (x @ x.conj().T).reshape(1, n * n)
    P0[nts // 2:] = P0[:nts // 2][::-1]

    def run(s, cr):
        s.set_P0(P0.ravel())
        s.compute_Pq_from_P0q()
        return s.P0_q_t_QP()

    _compare(run, tr.Ttn_FB.astype(CL) @ (tr.Tnt_BF.astype(CL) @ P0[1:-1]))


def test_dyson_rows():
    cr, tr = _crystal()
    L, nts, rng = cr.layout, tr.nts, np.random.default_rng(2)
    assert 8.0 * (nts - 2) * tr.nw * L.flat_ao_size > 4e7
    tau = np.asarray(tr.tau_fermi)
    sig = np.zeros((nts, L.flat_ao_size), np.complex128)
    for n, o in zip(L.ao_sizes[0], L.ao_offsets[0]):
        for e in (-1.2, 0.7):
            x = rng.normal(size=(n, n)) + 1j * rng.normal(size=(n, n))
            f = np.exp(-tau * e if e > 0 else (tr.beta - tau) * e) / (1 + np.exp(-tr.beta * abs(e)))
            sig[:, o:o + n * n] -= 0.02 * f[:, None] * (x @ x.conj().T).reshape(1, n * n)
    mu = float(cr.mu)
    w = tr.Tnt.astype(CL) @ sig[1:-1]
    wn = np.array([(2.0 * float(n) + 1.0) * 3.14159265358979323846 / tr.beta for n in tr.wsample_fermi])
    g = np.zeros_like(w)
    F, S = cr.F.reshape(-1), cr.S.reshape(-1)
    for n, o in zip(L.ao_sizes[0], L.ao_offsets[0]):
        n, o = int(n), int(o)
        a = (1j * wn + mu).astype(CL)[:, None, None] * S[o:o + n * n].reshape(n, n) \
            - F[o:o + n * n].reshape(n, n) - w[:, o:o + n * n].reshape(-1, n, n)
        x = np.linalg.inv(a.astype(np.complex128)).astype(CL)
        for _ in range(2):
            x = x @ (2 * np.eye(n) - a @ x)
        g[:, o:o + n * n] = x.reshape(-1, n * n)

    def run(s, cr):
        s.set_Selfenergy(sig.ravel())
        s.dyson(mu)
        return s.G_tau()

    _compare(run, tr.Ttn.astype(CL) @ g)


def test_zero_rows_do_not_set_the_scale():
    """Frequencies at which W~ vanishes, beside others at 10^-25: both handles agree to
    rounding (120 terms, row by row)."""
    from mbsymmetry_gb300 import _abi
    from mbsymmetry_gb300.solver import GWSolver
    cr, tr = _crystal()
    L, nts, rng = cr.layout, tr.nts, np.random.default_rng(3)
    T = np.array(tr.Tnt_BF)
    T[3::4] = 0.0
    P0 = np.zeros((nts, L.flat_aux_size), np.complex128)
    for n, o in zip(L.aux_sizes[0], L.aux_offsets[0]):
        x = rng.normal(size=(n, n)) + 1j * rng.normal(size=(n, n))
        P0[:, o:o + n * n] = -1e-25 * np.cosh(np.linspace(-3, 3, nts))[:, None] * (x @ x.conj().T).reshape(1, n * n)
    out = []
    for fma in (False, True):
        s = GWSolver(L, 1, tr, fp64_fma=fma)
        _abi.check(s.lib.gwgb_set_transforms(s.h, *(a.ctypes.data for a in (tr.Tnt, tr.Ttn, T, tr.Ttn_FB,
                                                                            tr.wsample_fermi)), None, None))
        s.set_shared_Coulomb(cr.V)
        s.set_P0(P0.ravel())
        s.compute_Pq_from_P0q()
        out.append(s.P0_q_t_QP().reshape(nts, -1))
        s.close()
    scale = np.abs(tr.Ttn_FB) @ np.abs(T @ P0[1:-1]).max(1)
    assert np.abs(out[1]).max() > 0
    assert (np.abs(out[0] - out[1]).max(1) < 120 * 2.0 ** -52 * scale).all()
