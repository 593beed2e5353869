"""Device allocations that fail (injected on the host): lists, operand images and
work buffers of the sliced contractions.  FP64, which has kernels that need none
of them, still answers; the split precision reports the failure or answers, and the
same handle answers once memory is there again."""
import numpy as np
import pytest

from _helpers import crystal
from mbsymmetry_gb300 import _abi

pytestmark = pytest.mark.gpu


@pytest.fixture
def fail_alloc():
    lib = _abi.load()
    yield lambda first, count: _abi.check(lib.gwgb_test_fail_alloc(first, count))
    lib.gwgb_test_fail_alloc(1, 0)


def _solver(precision):
    from mbsymmetry_gb300.solver import GWSolver
    cr, tr = crystal("C1")
    return cr, tr, GWSolver(cr.layout, cr.ns, tr, precision=precision)


def _inputs(cr, s):
    s.set_shared_Coulomb(cr.V)
    s.set_fock(cr.F, cr.S)


def _solve(cr, s):
    s.set_Selfenergy(np.zeros(s.g_size, np.complex128))
    s.dyson(cr.mu)
    s.solve()
    return s.P0_q_t_QP(), s.Selfenergy()


def _reference(precision):
    cr, _, s = _solver(precision)
    _inputs(cr, s)
    out = _solve(cr, s)
    s.close()
    return out


@pytest.mark.parametrize("first,count", [(n, 1) for n in range(1, 7)] + [(1, 1000), (3, 1000), (5, 1000)])
def test_fp64_answers_without_the_buffers(first, count, fail_alloc, monkeypatch):
    monkeypatch.setenv("GWGB_FP64_SLICES", "1")
    ref = _reference("fp64")
    cr, _, s = _solver("fp64")
    fail_alloc(first, count)
    _inputs(cr, s)
    got = _solve(cr, s)
    again = _solve(cr, s)
    fail_alloc(1, 0)
    s.close()
    for a, b, c in zip(ref, got, again):
        assert np.abs(a - b).max() < 1e-12 * np.abs(a).max()
        assert np.array_equal(b, c)


@pytest.mark.parametrize("first,count", [(n, 1) for n in range(1, 4)] + [(1, 1000), (3, 1000)])
def test_split_precision_recovers(first, count, fail_alloc):
    ref = _reference("ozaki")
    cr, _, s = _solver("ozaki")
    _inputs(cr, s)
    fail_alloc(first, count)
    try:
        got = _solve(cr, s)
    except _abi.GwgbError as e:
        assert e.code in (_abi.GWGB_E_NOMEM, _abi.GWGB_E_UNSUPPORTED)
        got = None
    assert got is None or count == 1
    fail_alloc(1, 0)
    for out in (got, _solve(cr, s)):
        assert out is None or all(np.array_equal(a, b) for a, b in zip(ref, out))
    s.close()


def test_split_precision_lists_fail(fail_alloc):
    """Switching the precision fails with the lists; switching it again works."""
    ref = _reference("ozaki")
    cr, _, s = _solver("fp64")
    _inputs(cr, s)
    fail_alloc(2, 1000)
    try:
        s.single_prec_run(True)
        with pytest.raises(_abi.GwgbError) as e:
            _solve(cr, s)
        assert e.value.code in (_abi.GWGB_E_NOMEM, _abi.GWGB_E_UNSUPPORTED)
    except _abi.GwgbError as e:
        assert e.code in (_abi.GWGB_E_NOMEM, _abi.GWGB_E_UNSUPPORTED)
    fail_alloc(1, 0)
    s.single_prec_run(True)
    assert all(np.array_equal(a, b) for a, b in zip(ref, _solve(cr, s)))
    s.close()


@pytest.mark.parametrize("precision", ["fp64", "ozaki"])
@pytest.mark.parametrize("ns", [1, 2])
def test_less_memory_means_smaller_chunks(precision, ns, fail_alloc, monkeypatch):
    """An allocation that fails makes the engine plan again with smaller chunks, the
    images of G and P~ by ranges of tau and none of V kept: more launches, the same bits."""
    from mbsymmetry_gb300.solver import GWSolver
    monkeypatch.setenv("GWGB_FP64_SLICES", "1")
    cr, tr = crystal("C1", ns=ns)
    out = []
    for chunk, fails in ((None, 0), (None, 1), ("1", 1), (None, 5)):
        if chunk:
            monkeypatch.setenv("GWGB_TC_CHUNK_MB", chunk)
        else:
            monkeypatch.delenv("GWGB_TC_CHUNK_MB", raising=False)
        s = GWSolver(cr.layout, ns, tr, precision=precision)
        _inputs(cr, s)
        s.set_Selfenergy(np.zeros(s.g_size, np.complex128))
        s.dyson(cr.mu)
        G0 = s.G_tau()
        fail_alloc(1, fails)
        s.solve()
        fail_alloc(1, 0)
        n = s.stats()["kernel_launches"]
        first = (s.P0_q_t_QP(), s.Selfenergy())
        s.set_G(G0)
        s.iteration(cr.mu)  # the same plan in a captured graph
        assert np.array_equal(first[1], s.Selfenergy())
        out.append((n, *first))
        s.close()
    assert out[2][0] > 5 * out[0][0]  # one tau range after the other
    for n, P, S in out[1:]:
        assert np.array_equal(P, out[0][1]) and np.array_equal(S, out[0][2])


def test_transforms_run_without_their_images(fail_alloc):
    """Every single allocation of a handle's creation in turn: either the creation
    fails with GWGB_E_NOMEM, or a transform goes on with the FP64 kernel and the W~
    solve and Dyson agree with the undisturbed handle's (60 to 150 terms a transform,
    a solve in between: 1e-12 of the largest element)."""
    from mbsymmetry_gb300.crystal import CrystalSpec, load_ir, make_crystal
    from mbsymmetry_gb300.solver import GWSolver
    from mbsymmetry_gb300.transformer import build_transforms
    cr = make_crystal(CrystalSpec("xf", "fcc", (1, 1, 1), 48, 50, 150, 50.0, ao_block=(14, 18), aux_block=(16, 17),
                                  seed=7))
    tr = build_transforms(load_ir(150), 50.0)
    assert 8.0 * (tr.nts - 2) * tr.nw * cr.layout.flat_ao_size > 4e7 < 8.0 * (tr.nts - 2) * tr.nw_b * cr.layout.flat_aux_size
    rng = np.random.default_rng(4)
    tau = np.asarray(tr.tau_fermi)
    P0 = np.zeros((tr.nts, cr.layout.flat_aux_size), np.complex128)
    for n, o in zip(cr.layout.aux_sizes[0], cr.layout.aux_offsets[0]):  # negative definite, one bosonic pole a block
        x = rng.normal(size=(n, n)) + 1j * rng.normal(size=(n, n))
        w = rng.uniform(0.5, 2.0)
        P0[:, o:o + n * n] = (-0.02 * (np.exp(-tau * w) + np.exp(-(tr.beta - tau) * w)))[:, None] * (x @ x.conj().T).ravel()

    def run(s):
        s.set_shared_Coulomb(cr.V)
        s.set_fock(cr.F, cr.S)
        s.set_Selfenergy(np.zeros(s.g_size, np.complex128))
        s.dyson(cr.mu)
        s.set_P0(P0.ravel())
        s.compute_Pq_from_P0q()
        return s.G_tau(), s.P0_q_t_QP()

    first = GWSolver(cr.layout, 1, tr)
    ref, fell_back = run(first), 0
    b0 = first.stats()["device_bytes"]
    second = GWSolver(cr.layout, 1, tr)
    size = second.stats()["device_bytes"] - b0 if run(second) else 0
    second.close()
    for n in range(1, 121):
        run(first)
        b0 = first.stats()["device_bytes"]
        fail_alloc(n, 1)
        try:
            s = GWSolver(cr.layout, 1, tr)
        except _abi.GwgbError as e:
            assert e.code == _abi.GWGB_E_NOMEM
            continue
        finally:
            fail_alloc(1, 0)
        got = run(s)
        fell_back += s.stats()["device_bytes"] - b0 < size
        s.close()
        for a, b in zip(ref, got):
            assert np.abs(a - b).max() < 1e-12 * np.abs(a).max()
    first.close()
    assert fell_back >= 4
