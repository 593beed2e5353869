"""Rounding of the block inverses of the W~ solve, R = sym((1 - sym(P))^-1) and R P,
against a NumPy restatement of the same elimination in FP64 (products formed first,
then subtracted; R P in FMAs), both against extended precision.  gwgb_wsolve_noalloc
with unit transforms gives R P of each block alone.  Mean relative error over 60
blocks: the restatement's within 1.06, the two rounding alike on the same data.  (With two
FMAs at the size of the element instead the restatement is at 1.12 to 1.26.)"""
import ctypes

import numpy as np
import pytest

from mbsymmetry_gb300 import _abi

pytestmark = pytest.mark.gpu
LD = np.longdouble


def fma(a, b, c):
    return (a.astype(LD) * b + c).astype(np.float64)


def csub(c, a, b):  # c - a b
    a, b = np.broadcast_arrays(a, b)
    return (c.real - fma(a.real, b.real, -(a.imag * b.imag))) + 1j * (c.imag - fma(a.real, b.imag, a.imag * b.real))


def herm(x):
    return 0.5 * (x + x.conj().transpose(0, 2, 1))


def sweeps(A):
    """-A^-1 from the lower triangle, symmetric sweeps without pivoting."""
    n = A.shape[1]
    low = np.tril(np.ones((n, n), bool))
    for k in range(n):
        d = 1.0 / A[:, k, k].real
        c = np.where(np.arange(n) >= k, A[:, :, k], A[:, k, :].conj())
        w = (c.real * d[:, None]) - 1j * (c.imag * d[:, None])
        w[:, k] = -d
        B = csub(A, c[:, :, None], w[:, None, :])
        B[:, k, :], B[:, :, k] = w, w.conj()
        A = np.where(low, B, A)
    R = -np.tril(A, -1)
    R = R + R.conj().transpose(0, 2, 1)
    i = np.arange(n)
    R[:, i, i] = -A[:, i, i].real
    return R


def gauss_jordan(A):
    """A^-1, full pivoting by the larger component."""
    A = A.copy()
    m, n, _ = A.shape
    at, used, swaps = np.arange(m), np.zeros(A.shape[:2], bool), []
    for _ in range(n):
        key = np.maximum(np.abs(A.real), np.abs(A.imag))
        key[used[:, :, None] | used[:, None, :]] = -1.0
        b = key.reshape(m, -1).argmax(1)
        r, c = b // n, b % n
        A[at, r], A[at, c] = A[at, c].copy(), A[at, r].copy()
        used[at, c] = True
        p = A[at, c, c]
        den = p.real * p.real + p.imag * p.imag
        inv = (p.real / den) - 1j * (p.imag / den)
        row = A[at, c].copy()
        row[at, c] = 1.0
        row = row * inv[:, None]
        f = A[at, :, c].copy()
        f[at, c] = 0.0
        A[at, :, c] = 0.0
        A = csub(A, row[:, None, :], f[:, :, None])
        A[at, c] = row
        swaps.append((r, c))
    for r, c in reversed(swaps):
        x, y = A[at, :, r].copy(), A[at, :, c].copy()
        A[at, :, r], A[at, :, c] = y, x
    return A


def product(R, P):
    re, im = np.zeros(P.shape), np.zeros(P.shape)
    for l in range(P.shape[1]):
        a, b = np.broadcast_arrays(R[:, :, l, None], P[:, None, l, :])
        re = fma(-a.imag, b.imag, fma(a.real, b.real, re))
        im = fma(a.imag, b.real, fma(a.real, b.imag, im))
    return re + 1j * im


@pytest.mark.parametrize("definite", [True, False])
@pytest.mark.parametrize("n", [12, 24, 40])
def test_rounding_of_the_solve(n, definite):
    import torch
    nts, m = 62, 60
    rng = np.random.default_rng(n)
    q, _ = np.linalg.qr(rng.normal(size=(m, n, n)) + 1j * rng.normal(size=(m, n, n)))
    ev = -rng.uniform(0.05, 3.0, (m, n)) if definite else rng.choice([-1.0, 3.0], (m, n)) * rng.uniform(0.5, 1.5, (m, n))
    P = herm((q * ev[:, None, :]) @ q.conj().transpose(0, 2, 1))
    A = np.eye(n) - herm(P)
    X = np.linalg.inv(A).astype(np.clongdouble)
    for _ in range(2):
        X = X @ (2 * np.eye(n) - A @ X)
    exact = herm(X) @ P
    model = product(sweeps(A) if definite else herm(gauss_jordan(A)), P)
    # unit transforms: W[w] = P0[w + 1], P[w + 1] = (R W)[w]
    dev = torch.device("cuda:0")
    src = np.zeros((nts, n * n), np.complex128)
    src[1:-1] = P.reshape(m, -1)
    t1 = torch.from_numpy(np.eye(m, dtype=np.complex128)).to(dev)
    t2 = torch.from_numpy(np.eye(nts, m, -1, dtype=np.complex128)).to(dev)
    x = torch.from_numpy(src).to(dev)
    out = torch.zeros_like(x)
    sizes = np.array([n], np.int32)
    torch.cuda.synchronize()
    lib = _abi.load()
    _abi.check(lib.gwgb_wsolve_noalloc(0, *(ctypes.c_void_p(y.data_ptr()) for y in (x, out, t1, t2)), nts, m,
                                       sizes.ctypes.data, 1, None))
    got = out.cpu().numpy()[1:-1].reshape(m, n, n)

    def err(y):
        return float(np.mean(np.sqrt((np.abs(y - exact) ** 2).sum((1, 2)) / (np.abs(exact) ** 2).sum((1, 2)))))

    print(f"n {n} definite {definite}: GPU {err(got):.3e}, restated {err(model):.3e}")
    assert err(got) < 1.06 * err(model)
