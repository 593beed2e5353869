"""Performance cases of the GW engine: what a program that owns a crystal asks
of :class:`mbsymmetry_gb300.solver.GWSolver`.

A case names a crystal (lattice, k mesh, orbital and auxiliary basis sizes,
irrep block ranges, imaginary-time grid, spins), the contraction precision
("fp64", the drop-in, or "ozaki", the sliced path a caller selects with
``single_prec_run(True)``) and one operation:

* ``iteration``: G(tau) from the host, one GW iteration
  (P0 -> P~ -> Sigma -> Dyson), Sigma(tau) and the new G(tau) back: the call a
  host code with its own mixing makes once per cycle;
* ``loop``: three iterations of the device-resident self-consistent loop
  (mu search, mixing, energies), from a given G and Sigma;
* ``dyson``: Sigma(tau) from the host, the Dyson equation, G(tau) back;
* ``screening``: P0(tau) from the host, the W~ solve, P~(tau) back;
* ``exchange``: Hartree-Fock exchange of a density matrix.

The solver (layout, V, F, S, transforms: what a program sets up once per
crystal) is made by :func:`prepare`; G, Sigma and P0 come from the host in
every pass and the results go back, as the reference's solver interface has it.
The FP32-class "tf32x3" and "bf16x3" precisions are kept in the engine for
comparison only and are not timed here.
"""
import functools
import math

import numpy as np
import torch

from mbsymmetry_gb300.crystal import CONFIGS, CrystalSpec, half_filling_mu, load_ir, make_crystal
from mbsymmetry_gb300.solver import GWSolver
from mbsymmetry_gb300.transformer import build_transforms

NE_TOL = 1e-10   # electrons, the loop's mu search
ALPHA = 0.5      # linear mixing
LOOP = 3         # iterations of a "loop" pass


def _case(name, config, op, precision, mesh=None, ns=1, **other):
    """A case with the orbitals, grid and block ranges of one of the repository's crystals."""
    s = CONFIGS[config]
    m = mesh or s.mesh
    c = {"name": name, "op": op, "precision": precision, "lattice": s.lattice, "n1": m[0], "n2": m[1], "n3": m[2],
         "nao": s.nao, "naux": s.naux, "nts": s.nts, "beta": s.beta, "ns": ns, "ao_lo": s.ao_block[0],
         "ao_hi": s.ao_block[1], "aux_lo": s.aux_block[0], "aux_hi": s.aux_block[1], "layout": s.seed}
    c.update(other)
    return c


def listed():
    return [
        # an s+p model on a 3x3x3 mesh: method development and unit tests, where launches and latency count
        _case("sp_fp64", "C1", "iteration", "fp64"),
        _case("sp_sliced", "C1", "iteration", "ozaki"),
        # the same model, both spins, in the self-consistent loop
        _case("sp_spin_loop_fp64", "C1", "loop", "fp64", ns=2),
        # s+p+d, 2 atoms, 3x3x3: the configuration the benchmark quotes, as the drop-in and sliced
        _case("spd_fp64", "C2", "iteration", "fp64"),
        _case("spd_sliced", "C2", "iteration", "ozaki"),
        # 4 atoms, larger irrep blocks on a coarse mesh: a supercell-like run
        _case("spd4_8k_fp64", "C3", "iteration", "fp64", mesh=(2, 2, 2)),
        # the production-size run of the set: 4 atoms on 3x3x3, sliced
        _case("spd4_27k_sliced", "C3m", "iteration", "ozaki"),
        # hexagonal cell without inversion (time-reversal partners in the stars), uneven blocks up to 30
        _case("hex_8k_sliced", "C4", "iteration", "ozaki", mesh=(2, 2, 2)),
        _case("hex_4k_fp64", "C4", "iteration", "fp64", mesh=(2, 2, 1)),
        # single steps that host codes call on their own
        _case("hex_dyson", "C4", "dyson", "fp64", mesh=(2, 2, 2)),
        _case("spd4_screening", "C3", "screening", "fp64", mesh=(2, 2, 2)),
        _case("spd_exchange_fp64", "C2", "exchange", "fp64", mesh=(2, 2, 2)),
    ]


#: contraction FLOPs a drawn case may need, by precision (below the largest listed case of that precision)
_MOST = {"fp64": 1.2e11, "ozaki": 1.2e12}


def draw(rng):
    """One more case of the same ranges: both lattices, meshes of 1 to 27 points, 5 to 80 orbitals with 3.5 to 5
    auxiliary functions each, every committed time grid, one or two spins, both precisions, every operation."""
    while True:
        op = rng.choice(["iteration"] * 6 + ["loop", "dyson", "screening", "exchange"])
        precision = rng.choice(["fp64", "ozaki"]) if op in ("iteration", "exchange") else "fp64"
        lattice = rng.choice(["fcc", "hex"])
        m = rng.choice([(1, 1, 1), (2, 2, 2), (3, 3, 3)] if lattice == "fcc" else
                       [(1, 1, 1), (2, 2, 1), (2, 2, 2), (2, 2, 3), (3, 3, 1), (3, 3, 2)])
        nao = int(round(math.exp(rng.uniform(math.log(5), math.log(80)))))
        naux = int(round(nao * rng.uniform(3.5, 5.0)))
        nts = rng.choice([62, 100, 120, 150])
        c = {"op": op, "precision": precision, "lattice": lattice, "n1": m[0], "n2": m[1], "n3": m[2], "nao": nao,
             "naux": naux, "nts": nts, "beta": rng.choice([50.0, 100.0, 200.0]) if nts > 62 else 50.0,
             "ns": rng.choice([1, 1, 2]), "ao_lo": 1 if nao < 30 else 2, "ao_hi": min(40, max(4, nao // 3)),
             "aux_lo": 2, "aux_hi": min(64, max(12, naux // 4)), "layout": rng.randrange(1, 1 << 20)}
        w = work(c)
        if w["flops"] > _MOST[precision] / (LOOP if op == "loop" else 1) or w["bytes"] > 2.4e9:
            continue
        return c


# --------------------------------------------------------------------------- inputs
@functools.lru_cache(maxsize=64)
def _layout_of(key):
    c = dict(key)
    spec = CrystalSpec("case", c["lattice"], (c["n1"], c["n2"], c["n3"]), c["nao"], c["naux"], c["nts"], c["beta"],
                       ns=c["ns"], ao_block=(c["ao_lo"], c["ao_hi"]), aux_block=(c["aux_lo"], c["aux_hi"]),
                       seed=c["layout"])
    return make_crystal(spec, with_V=False)


def _crystal(case):
    """The layout, rotations and selection rule of the case (no V)."""
    keys = ("lattice", "n1", "n2", "n3", "nao", "naux", "nts", "beta", "ns", "ao_lo", "ao_hi", "aux_lo", "aux_hi",
            "layout")
    return _layout_of(tuple((k, case[k]) for k in keys))


@functools.lru_cache(maxsize=8)
def _transforms(nts, beta):
    return build_transforms(load_ir(nts), beta)


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _make_V(case, L, seed):
    """Complex Gaussian V blocks of the crystal generator's width, with V(k2, k1) = V(k1, k2)^H per aux function."""
    g = torch.Generator(device=_device())
    g.manual_seed(seed)
    x = torch.randn(2 * L.flat_V_size, dtype=torch.float64, device=_device(), generator=g)
    x *= 0.5 / math.sqrt(2.0 * case["nao"])
    V = x.cpu().numpy().view(np.complex128)
    nk = L.nk
    for k1 in range(nk):
        for k2 in range(k1, nk):
            p, pr = k1 * nk + k2, k2 * nk + k1
            q = L.pair_q(k1, k2)
            rev = {(int(a), int(b), int(c)): i for i, (a, b, c) in enumerate(L.tensor_irreps[pr])}
            for b, (iq, i1, i2) in enumerate(L.tensor_irreps[p]):
                iq, i1, i2 = int(iq), int(i1), int(i2)
                if p == pr and i1 > i2:
                    continue
                qb, b1, b2 = int(L.aux_sizes[q][iq]), int(L.ao_sizes[k1][i1]), int(L.ao_sizes[k2][i2])
                o = L.kpair_slice_offsets[p] + L.tensor_offsets[p][b]
                r = L.kpair_slice_offsets[pr] + L.tensor_offsets[pr][rev[(iq, i2, i1)]]
                n = qb * b1 * b2
                blk = V[o:o + n].reshape(qb, b1, b2)
                if o == r:
                    blk = 0.5 * (blk + blk.transpose(0, 2, 1).conj())
                    V[o:o + n] = blk.ravel()
                else:
                    V[r:r + n] = blk.transpose(0, 2, 1).conj().ravel()
    return V


def _make_onebody(case, L, tr, seed):
    """F and S [ns][flat_ao], mu at half filling, and the non-interacting G(tau) [nts][ns][flat_ao]."""
    rng = np.random.default_rng((seed, 11))
    ns, fa = case["ns"], L.flat_ao_size
    F = np.zeros((ns, fa), np.complex128)
    S = np.zeros((ns, fa), np.complex128)
    weight = np.bincount(L.irre_index, minlength=L.ink)
    parts, eigs = [], []
    for s in range(ns):
        for ik, k in enumerate(L.irre_list):
            for b, n in enumerate(L.ao_sizes[k]):
                n = int(n)
                o = int(L.kao_slice_offsets_irre[ik] + L.ao_offsets[k][b])
                x = rng.uniform(-1, 1, size=(n, n)) + 1j * rng.uniform(-1, 1, size=(n, n))
                h = 0.3 * (x + x.conj().T) + np.diag(rng.normal(0.0, 0.5, size=n))
                F[s, o:o + n * n] = h.ravel()
                S[s, o:o + n * n] = np.eye(n).ravel()
                e, u = np.linalg.eigh(h)
                parts.append((s, o, n, e, u))
                eigs.extend((float(v), float(weight[ik]) / ns) for v in e)
    mu = half_filling_mu(eigs, case["nao"], L.nk)
    G = np.zeros((tr.nts, ns, fa), np.complex128)
    tau = np.asarray(tr.tau_fermi)[:, None]
    for s, o, n, e, u in parts:
        x = (e - mu)[None, :]
        f = -np.exp(np.where(x > 0, -tau * x, (tr.beta - tau) * x) - np.log1p(np.exp(-tr.beta * np.abs(x))))
        G[:, s, o:o + n * n] = np.einsum("ia,ta,ja->tij", u, f, u.conj()).reshape(tr.nts, n * n)
    return F, S, mu, G


def _make_P0(L, tr, seed):
    """A polarization with the physical shape: three bosonic poles with negative semidefinite weights per block."""
    rng = np.random.default_rng((seed, 13))
    tau, beta = np.asarray(tr.tau_fermi), tr.beta
    P = np.zeros(tr.nts * L.flat_aux_size, np.complex128)
    for iq, q in enumerate(L.irre_list):
        size = int(L.qaux_slice_sizes[q])
        base = tr.nts * int(L.qaux_slice_offsets_irre[iq])
        view = P[base:base + tr.nts * size].reshape(tr.nts, size)
        for b, n in enumerate(L.aux_sizes[q]):
            n, o = int(n), int(L.aux_offsets[q][b])
            for w in rng.uniform(0.3, 3.0, size=3):
                x = (rng.normal(size=(n, n)) + 1j * rng.normal(size=(n, n))) / math.sqrt(2.0 * n)
                shape = (np.exp(-tau * w) + np.exp(-(beta - tau) * w)) / (1.0 - math.exp(-beta * w))
                view[:, o:o + n * n] -= 0.3 * shape[:, None] * (x @ x.conj().T).reshape(1, n * n)
    return P


def _inputs(case, seed):
    """Everything the seed decides, on the host."""
    L, tr = _crystal(case).layout, _transforms(case["nts"], case["beta"])
    op = case["op"]
    d = {"V": _make_V(case, L, seed)}
    d["F"], d["S"], d["mu"], d["G"] = _make_onebody(case, L, tr, seed)
    if op == "dyson":  # a self-energy of the GW shape: a few fermionic poles per block, a fraction of F
        _, _, _, other = _make_onebody(case, L, tr, seed + 1000003)
        d["Sigma"] = 0.3 * other
    if op == "screening":
        d["P0"] = _make_P0(L, tr, seed)
    if op == "exchange":
        d["rho"] = np.ascontiguousarray(-d["G"][-1])
    return L, tr, d


def prepare(case, seed):
    L, tr, d = _inputs(case, seed)
    s = GWSolver(L, case["ns"], tr, precision=case["precision"], device=0)
    s.set_shared_Coulomb(d.pop("V"))
    s.set_fock(d["F"], d["S"])
    zero = np.zeros(s.g_size, np.complex128)
    return {"op": case["op"], "solver": s, "n_electrons": float(case["nao"]), "zero": zero, **d}


def run(state):
    s, op = state["solver"], state["op"]
    if op == "iteration":
        s.set_G(state["G"])
        s.iteration(state["mu"])
        return {"Sigma": s.Selfenergy(), "G": s.G_tau()}
    if op == "loop":
        s.set_G(state["G"])
        s.set_Selfenergy(state["zero"])
        rec = s.sc_loop(LOOP, ALPHA, state["n_electrons"], state["mu"], tol=NE_TOL)
        return {"Sigma": s.Selfenergy(), "G": s.G_tau(),
                "records": np.array([[r["mu"], r["n_electrons"], r["e_corr"]] for r in rec])}
    if op == "dyson":
        s.set_Selfenergy(state["Sigma"])
        s.dyson(state["mu"])
        return {"G": s.G_tau()}
    if op == "screening":
        s.set_P0(state["P0"])
        s.compute_Pq_from_P0q()
        return {"P": s.P0_q_t_QP()}
    return {"K": s.hf_exchange(state["rho"])}


# --------------------------------------------------------------------------- work
@functools.lru_cache(maxsize=256)
def _work_of(key, op, nts, ns):
    L = _layout_of(key).layout
    irre = set(int(k) for k in L.irre_list)
    p0 = sig = 0.0
    vused = 0
    for k1 in range(L.nk):
        for k2 in range(L.nk):
            q, mq = L.pair_q(k1, k2), L.pair_q(k2, k1)
            for iq, i1, i2 in L.tensor_irreps[k1 * L.nk + k2]:
                n, a, b = int(L.aux_sizes[q][iq]), int(L.ao_sizes[k1][i1]), int(L.ao_sizes[k2][i2])
                f = 8.0 * n * a * b * (a + b + n)
                p0 += f if q in irre else 0.0
                sig += f if k1 in irre else 0.0
                vused += n * a * b if q in irre or mq in irre or k1 in irre else 0
    g, p = 16.0 * nts * ns * L.flat_ao_size, 16.0 * nts * L.flat_aux_size
    cube = sum(float(x) ** 3 for k in L.irre_list for x in L.aux_sizes[k])
    cubeg = ns * sum(float(x) ** 3 for k in L.irre_list for x in L.ao_sizes[k])
    solve = 16.0 * nts * cube + 16.0 * nts * nts * L.flat_aux_size
    dyson = 8.0 * nts * cubeg + 16.0 * nts * nts * ns * L.flat_ao_size
    if op == "dyson":
        return {"bytes": 2 * g, "flops": dyson}
    if op == "screening":
        return {"bytes": 2 * p, "flops": solve}
    if op == "exchange":  # one density matrix: the two V contractions at a single time
        rho = 16.0 * ns * L.flat_ao_size
        return {"bytes": 16.0 * vused + 2 * rho, "flops": ns * sig}
    once = p0 * ns * (nts // 2) + sig * ns * nts + solve + dyson
    n = LOOP if op == "loop" else 1
    return {"bytes": n * (16.0 * vused + 3 * g), "flops": n * once}


def work(case):
    keys = ("lattice", "n1", "n2", "n3", "nao", "naux", "nts", "beta", "ns", "ao_lo", "ao_hi", "aux_lo", "aux_hi",
            "layout")
    return dict(_work_of(tuple((k, case[k]) for k in keys), case["op"], case["nts"], case["ns"]))


# --------------------------------------------------------------------------- exact
class _Exact:
    """The same quantities with torch complex128 matrix products, block by block."""

    def __init__(self, case, seed):
        self.L, self.tr, self.d = _inputs(case, seed)
        self.ns = case["ns"]
        self.dev = _device()
        self.V = self._t(self.d["V"])

    def _t(self, a):
        return torch.from_numpy(np.ascontiguousarray(a)).to(self.dev)

    def _rotate(self, blocks, rep, k, kk, ck, irreps, offsets, base, sizes):
        """O X O^H (conjugated for a time-reversal partner) of every block of k from its representative's."""
        L = self.L
        out = {}
        if int(L.index[ck]) == ck:
            out = dict(blocks[kk])
        else:
            for b, (i1, i2) in enumerate(irreps[ck]):
                m, n = int(sizes[ck][i1]), int(sizes[kk][i2])
                o = int(base[ck] + offsets[ck][b])
                O = self._t(rep[o:o + m * n].reshape(m, n))
                out[int(i1)] = O @ blocks[kk][int(i2)] @ O.conj().T
        return {i: x.conj() if k != ck else x for i, x in out.items()}

    def G_blocks(self, G):
        """{k: {block: [t, s, b, b]}} over the full zone."""
        L = self.L
        G = self._t(G)
        nt = G.shape[0]
        irr = {}
        for ik, k in enumerate(L.irre_list):
            irr[int(k)] = {b: G[:, :, int(L.kao_slice_offsets_irre[ik] + L.ao_offsets[k][b]):][:, :, :int(n) ** 2]
                           .reshape(nt, self.ns, int(n), int(n)) for b, n in enumerate(L.ao_sizes[k])}
        out = {}
        for k in range(L.nk):
            ck = int(L.conj_index[k])
            kk = int(L.irre_list[L.irre_index[ck]])
            out[k] = self._rotate(irr, L.orep, k, kk, ck, L.orep_irreps, L.orep_offsets, L.korep_slice_offsets,
                                  L.ao_sizes)
        return out

    def P_blocks(self, P):
        """{q: {block: [t, n, n]}} over the full zone from {q_irr: {block: ...}}."""
        L = self.L
        out = {}
        for q in range(L.nk):
            cq = int(L.conj_index[q])
            qq = int(L.irre_list[L.irre_index[q]])
            out[q] = self._rotate(P, L.auxrep, q, qq, cq, L.auxrep_irreps, L.auxrep_offsets,
                                  L.kauxrep_slice_offsets, L.aux_sizes)
        return out

    def V_block(self, p, b, n, b1, b2):
        o = int(self.L.kpair_slice_offsets[p] + self.L.tensor_offsets[p][b])
        return self.V[o:o + n * b1 * b2].reshape(n, b1, b2)

    def polarization(self, G):
        """P0 of the irreducible q at every tau: {q: {block: [t, n, n]}}."""
        L, nts = self.L, self.tr.nts
        half = nts // 2
        pref = -1.0 / L.nk * (2.0 if self.ns == 1 else 1.0)
        out = {}
        for q in (int(q) for q in L.irre_list):
            acc = {b: torch.zeros(half, int(n), int(n), dtype=torch.complex128, device=self.dev)
                   for b, n in enumerate(L.aux_sizes[q])}
            for k1 in range(L.nk):
                k2 = L.mom_cons(k1, 0, q)
                p = k1 * L.nk + k2
                for b, (iq, i1, i2) in enumerate(L.tensor_irreps[p]):
                    n, b1, b2 = int(L.aux_sizes[q][iq]), int(L.ao_sizes[k1][i1]), int(L.ao_sizes[k2][i2])
                    v = self.V_block(p, b, n, b1, b2)
                    for s in range(self.ns):
                        g1 = G[k1][int(i1)].flip(0)[:half, s]                          # G(beta - tau)[t', p]
                        g2 = G[k2][int(i2)][:half, s]                                  # G(tau)[m, n]
                        x1 = g1 @ v.permute(1, 0, 2).reshape(b1, n * b2)               # [t][t'][(Q, m)]
                        x2 = v.conj().reshape(n * b1, b2) @ g2.transpose(1, 2)         # [t][(P, t')][m]
                        x1 = x1.reshape(half, b1, n, b2).permute(0, 2, 1, 3).reshape(half, n, b1 * b2)
                        acc[int(iq)] += pref * (x1 @ x2.reshape(half, n, b1 * b2).transpose(1, 2))
            out[q] = {b: torch.cat([x, x.flip(0)]) for b, x in acc.items()}
        return out

    def screened(self, P0):
        """P~ = (1 - P~0)^-1 P~0 through the Matsubara grid."""
        fwd, bwd = self._t(self.tr.Tnt_BF), self._t(self.tr.Ttn_FB)
        out = {}
        for q, blocks in P0.items():
            out[q] = {}
            for b, x in blocks.items():
                n = x.shape[-1]
                w = (fwd @ x[1:-1].reshape(-1, n * n)).reshape(-1, n, n)
                a = torch.eye(n, dtype=w.dtype, device=self.dev) - 0.5 * (w + w.conj().transpose(1, 2))
                r = torch.linalg.inv(a)
                r = 0.5 * (r + r.conj().transpose(1, 2))
                out[q][b] = (bwd @ (r @ w).reshape(-1, n * n)).reshape(-1, n, n)
        return out

    def self_energy(self, G, P, nt):
        """Sigma (or the exchange, with P = None) of the stored k: [t][s][flat_ao]."""
        L = self.L
        out = torch.zeros(nt, self.ns, L.flat_ao_size, dtype=torch.complex128, device=self.dev)
        for ik, k1 in enumerate(int(k) for k in L.irre_list):
            for k2 in range(L.nk):
                q = int(L.mom_cons(k1, k2, 0))   # k1 - k2 = q
                p = k1 * L.nk + k2
                for b, (iq, i1, i2) in enumerate(L.tensor_irreps[p]):
                    n, b1, b2 = int(L.aux_sizes[q][iq]), int(L.ao_sizes[k1][i1]), int(L.ao_sizes[k2][i2])
                    v = self.V_block(p, b, n, b1, b2)
                    o = int(L.kao_slice_offsets_irre[ik] + L.ao_offsets[k1][int(i1)])
                    vh = v.conj().permute(2, 0, 1).reshape(b2 * n, b1)                  # [(n, P)][j]
                    for s in range(self.ns):
                        g = G[k2][int(i2)][:, s]                                        # [t][m][n]
                        y = (v.reshape(n * b1, b2) @ g).reshape(nt, n, b1, b2)          # [t][Q][i][n]
                        y = y.permute(0, 2, 3, 1).reshape(nt, b1 * b2, n)
                        if P is not None:
                            y = y @ P[q][int(iq)]                                       # [t][(i, n)][P]
                        y = y.reshape(nt, b1, b2 * n) @ vh
                        out[:, s, o:o + b1 * b1] -= y.reshape(nt, b1 * b1) / L.nk
        return out

    def dyson(self, sigma):
        L, tr = self.L, self.tr
        w = torch.einsum("wt,tsx->wsx", self._t(tr.Tnt), sigma[1:-1])
        iw = self._t(1j * (2.0 * tr.wsample_fermi + 1.0) * np.pi / tr.beta) + self.d["mu"]
        a = iw[:, None, None] * self._t(self.d["S"])[None] - self._t(self.d["F"])[None] - w
        out = torch.zeros_like(a)
        for ik, k in enumerate(L.irre_list):
            for b, n in enumerate(L.ao_sizes[k]):
                n, o = int(n), int(L.kao_slice_offsets_irre[ik] + L.ao_offsets[k][b])
                x = a[:, :, o:o + n * n].reshape(-1, self.ns, n, n)
                out[:, :, o:o + n * n] = torch.linalg.inv(x).reshape(-1, self.ns, n * n)
        return torch.einsum("tw,wsx->tsx", self._t(tr.Ttn), out)


def exact(case, seed):
    op = case["op"]
    if op == "loop" or work(case)["flops"] > 1e12:  # mu is fixed only to the search's tolerance; or too long
        return None
    e = _Exact(case, seed)
    if op == "dyson":
        return {"G": e.dyson(e._t(e.d["Sigma"])).reshape(-1)}
    if op == "screening":
        L, nts = e.L, e.tr.nts
        P0 = {}
        for iq, q in enumerate(int(q) for q in L.irre_list):
            size, base = int(L.qaux_slice_sizes[q]), nts * int(L.qaux_slice_offsets_irre[iq])
            x = e._t(e.d["P0"])[base:base + nts * size].reshape(nts, size)
            x = torch.cat([x[:nts // 2], x[:nts // 2].flip(0)])
            P0[q] = {b: x[:, int(L.aux_offsets[q][b]):int(L.aux_offsets[q][b]) + int(n) ** 2]
                     .reshape(nts, int(n), int(n)) for b, n in enumerate(L.aux_sizes[q])}
        P = e.screened(P0)
        return {"P": torch.cat([torch.cat([x.reshape(nts, -1) for x in P[int(q)].values()], 1).reshape(-1)
                                for q in L.irre_list])}
    if op == "exchange":
        G = e.G_blocks(e.d["rho"][None])
        return {"K": e.self_energy(G, None, 1).reshape(case["ns"], -1)}
    G = e.G_blocks(e.d["G"])
    P = e.P_blocks(e.screened(e.polarization(G)))
    sigma = e.self_energy(G, P, case["nts"])
    return {"Sigma": sigma.reshape(-1), "G": e.dyson(sigma).reshape(-1)}
