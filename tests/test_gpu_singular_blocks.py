"""Singular and tiny Dyson blocks.  A block of equal elements m leaves an exact
zero after one elimination step whenever m times its rounded reciprocal m / (m m)
rounds to one, and must then be reported; the inverse of a block at 1e-155, whose
squared pivot is subnormal, is finite."""
import numpy as np
import pytest

from mbsymmetry_gb300 import _abi

pytestmark = pytest.mark.gpu


def _solver(n):
    from mbsymmetry_gb300.crystal import CrystalSpec, load_ir, make_crystal
    from mbsymmetry_gb300.solver import GWSolver
    from mbsymmetry_gb300.transformer import build_transforms
    cr = make_crystal(CrystalSpec("sing", "fcc", (1, 1, 1), n, 2 * n, 62, 50.0, ao_block=(n, n), aux_block=(2, 2),
                                  seed=5))
    tr = build_transforms(load_ir(62), 50.0)
    s = GWSolver(cr.layout, 1, tr)
    s.set_Selfenergy(np.zeros(s.g_size, np.complex128))
    return cr, tr, s


@pytest.mark.parametrize("n", [2, 17, 33])  # one warp, a CTA of 128 and of 256 threads per block
def test_equal_elements_are_singular(n):
    cr, _, s = _solver(n)
    zero = np.zeros_like(cr.F)
    m = np.arange(1.0, 400.0)
    for v in m[m / (m * m) * m == 1.0][:: 1 if n == 2 else 9]:
        s.set_fock(np.full_like(cr.F, v), zero)
        with pytest.raises(_abi.GwgbError) as e:
            s.dyson(0.0)
        assert e.value.code == _abi.GWGB_E_NUMERIC, v
    s.close()


@pytest.mark.parametrize("n", [2, 17, 33])
def test_tiny_blocks_are_finite(n):
    cr, tr, s = _solver(n)
    s.set_fock(np.tile(np.eye(n).ravel() * 1e-155, cr.F.size // (n * n)).reshape(cr.F.shape).astype(cr.F.dtype),
               np.zeros_like(cr.F))
    s.dyson(0.0)
    G = s.G_tau().reshape(tr.nts, -1, n, n)
    s.close()
    ref = -1e155 * tr.Ttn.sum(axis=1)[:, None, None, None] * np.eye(n)
    # the squared pivot 1e-310 is held to 5e-324 / 1e-310 = 5e-14; sums of about 60 terms cancel by up to 1e3
    assert np.abs(G - ref).max() < 1e-9 * np.abs(1e155 * tr.Ttn).sum(axis=1).max()
