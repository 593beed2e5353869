"""V's slice images, kept from one V upload to the next or, above the limit that
GWGB_TC_CHUNK_MB sets, built per chunk inside the solve: the same bits, and a new
V is seen by both.  Hexagonal with time-reversal partners, both spins."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "ozaki"])
def test_images_kept_or_built_per_chunk(precision, monkeypatch):
    from mbsymmetry_gb300.crystal import CrystalSpec, load_ir, make_crystal
    from mbsymmetry_gb300.solver import GWSolver
    from mbsymmetry_gb300.transformer import build_transforms
    monkeypatch.setenv("GWGB_FP64_SLICES", "1")
    cr = make_crystal(CrystalSpec("v", "hex", (2, 2, 1), 17, 60, 62, 50.0, ns=2, ao_block=(1, 9), aux_block=(2, 33),
                                  seed=9))
    tr = build_transforms(load_ir(62), 50.0)
    out = []
    for mb in (None, "1"):
        if mb:
            monkeypatch.setenv("GWGB_TC_CHUNK_MB", mb)
        else:
            monkeypatch.delenv("GWGB_TC_CHUNK_MB", raising=False)
        s = GWSolver(cr.layout, 2, tr, precision=precision)
        s.set_fock(cr.F, cr.S)
        res = []
        for V in (cr.V, 0.75 * cr.V, cr.V):
            s.set_shared_Coulomb(V)
            s.set_Selfenergy(np.zeros(s.g_size, np.complex128))
            s.dyson(cr.mu)
            s.iteration(cr.mu)
            res.append((s.P0_q_t_QP(), s.Selfenergy(), s.G_tau()))
        launches = _builds(s)
        s.close()
        assert all(np.array_equal(a, b) for a, b in zip(res[0], res[2]))
        assert not np.array_equal(res[0][1], res[1][1])
        out.append((launches, res))
    kept, built = out
    assert len(built[0]) > len(kept[0])
    for a, b in zip(kept[1], built[1]):
        assert all(np.array_equal(x, y) for x, y in zip(a, b))


def _builds(s):
    """The image builds inside a solve: those of G and P~, and V's where they are not kept."""
    return [x for x in s.launch_stats() if x["kernel"] == "oz_build_kernel" and x["stage"] in ("Z1", "W")]
