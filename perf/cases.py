"""Performance cases: the calls that a CI program makes of this framework, over the sizes it makes them at.

Every case goes through the package's public classes and functions with the buffers and handles a program keeps:

* ``sigma``     sigma = H C of one species (``POLYQUANT_DETSET.sigma``): the step of every Davidson iteration
* ``sigma2``    the same for an electron-positron product space
* ``batch``     ``CIBatch.sigma`` over independent problems of uneven size
* ``ham``       ``create_ham`` (the reference's default ``build_matrix`` route) and one sigma with the matrix
* ``ao2mo``     the AO->MO two-electron transform that feeds a CI
* ``props``     <S^2> of the states and the 1-RDMs of the first one, after a solve
* ``davidson``  a whole solve: energies and vectors

CI vectors have normal entries whose magnitudes spread over four decades, as the entries of Davidson's vectors do.
``exact`` evaluates the same operators in 64 bits from the second-quantised form on product-space arrays.
"""
from __future__ import annotations

import itertools
from math import comb

import numpy as np
import torch

from polyquant_gb300 import synthetic
from polyquant_gb300._lib import (PQ_AO_PACKED8, PQ_AO_PAIRS, PQ_FP32, PQ_FP64, PQ_XFORM_BF16X3, PQ_XFORM_FP64,
                                  PQ_XFORM_TF32X3)
from polyquant_gb300.batch import CIBatch
from polyquant_gb300.detset import INT_MAX, POLYQUANT_DETSET
from polyquant_gb300.integral import ao2mo

PREC = {"fp64": PQ_FP64, "fp32": PQ_FP32}
MODE = {"fp64": PQ_XFORM_FP64, "bf16x3": PQ_XFORM_BF16X3, "tf32x3": PQ_XFORM_TF32X3}


# ---- the cases ---------------------------------------------------------------------------------------------------
def listed():
    return [
        # full CI of water in the STO-3G basis (7 orbitals, 441 determinants): the smallest call, one vector
        dict(name="sigma_water_fci", kind="sigma", n=7, na=5, nb=5, level=0, nvec=1, prec="fp64"),
        # CISD of ten electrons in 24 orbitals (water in a double-zeta basis): a truncated, ragged space
        dict(name="sigma_water_cisd", kind="sigma", n=24, na=5, nb=5, level=2, nvec=3, prec="fp64"),
        # one root of an open-shell full CI, unequal spin lists: a single-state solve
        dict(name="sigma_fci13_1root", kind="sigma", n=13, na=6, nb=5, level=0, nvec=1, prec="fp64"),
        # block Davidson's sigma of four roots in double precision
        dict(name="sigma_fci14_4roots", kind="sigma", n=14, na=7, nb=7, level=0, nvec=4, prec="fp64"),
        # the benchmark's 16-orbital full CI, four roots, in the precision that a mixed solve spends its time in
        dict(name="sigma_fci16_fp32", kind="sigma", n=16, na=8, nb=8, level=0, nvec=4, prec="fp32"),
        # positronium hydride in the benchmark's 60 + 40 orbitals, three roots
        dict(name="sigma_psh", kind="sigma2", ne=60, ea=1, eb=1, np=40, pa=1, pb=0, level=0, nvec=3, prec="fp64"),
        # sixteen uneven full-CI problems (with and without positrons) advanced together, two roots each
        dict(name="batch_16_problems", kind="batch", count=16, pick=3, nvec=2, prec="fp64"),
        # the same CISD through the explicit sparse H: the matrix and one product with it
        dict(name="ham_water_cisd", kind="ham", n=24, na=5, nb=5, level=2, nvec=1),
        # AO->MO in double precision, a basis that fills no tile, with deleted virtuals
        dict(name="ao2mo_fp64_150", kind="ao2mo", n=150, nmo=141, mode="fp64"),
        # the benchmark's 256-function transform in split BF16
        dict(name="ao2mo_bf16x3_256", kind="ao2mo", n=256, nmo=256, mode="bf16x3"),
        # properties of four states of a 12-orbital full CI
        dict(name="props_fci12", kind="props", n=12, na=6, nb=6, level=0, nvec=4),
        # a whole double-precision solve for four states
        dict(name="davidson_fci10", kind="davidson", n=10, na=5, nb=5, level=0, nvec=4),
    ]


def draw(rng):
    kind = rng.choice(["fci", "fci", "trunc", "trunc", "sigma2", "batch", "ham", "ao2mo", "ao2mo", "props", "davidson"])
    prec = "fp32" if rng.random() < 0.25 else "fp64"
    if kind == "fci":
        while True:
            n = rng.randint(5, 14)
            na = rng.randint(1, min(8, n - 1))
            nb = rng.randint(max(0, na - 2), na)
            if 30 <= comb(n, na) * comb(n, nb) <= 12_000_000:
                return dict(kind="sigma", n=n, na=na, nb=nb, level=0, nvec=rng.randint(1, 5), prec=prec)
    if kind == "trunc":
        n = rng.randint(9, 34)
        na = rng.randint(2, 6 if n <= 24 else 4)
        nb = rng.randint(max(1, na - 1), na)
        level = 3 if n <= 13 and rng.random() < 0.5 else 2
        level = min(level, n - na)
        return dict(kind="sigma", n=n, na=na, nb=nb, level=level, nvec=rng.randint(1, 4), prec=prec)
    if kind == "sigma2":
        ne, npos = rng.randint(12, 60), rng.randint(6, 40)
        if rng.random() < 0.4:
            ne, npos = rng.randint(6, 9), rng.randint(4, 8)
            return dict(kind="sigma2", ne=ne, ea=2, eb=rng.randint(1, 2), np=npos, pa=1, pb=rng.randint(0, 1),
                        level=rng.choice([0, 2, 3]), nvec=rng.randint(1, 4), prec=prec)
        return dict(kind="sigma2", ne=ne, ea=1, eb=1, np=npos, pa=1, pb=0, level=0, nvec=rng.randint(1, 4), prec=prec)
    if kind == "batch":
        return dict(kind="batch", count=rng.randint(3, 16), pick=rng.randint(4, 100000), nvec=rng.randint(1, 3), prec=prec)
    if kind == "ham":
        n = rng.randint(6, 24)
        na = rng.randint(2, min(5, n - 2))
        return dict(kind="ham", n=n, na=na, nb=rng.randint(max(1, na - 1), na), level=2, nvec=rng.randint(1, 4))
    if kind == "ao2mo":
        mode = rng.choice(["fp64", "fp64", "bf16x3", "tf32x3"])
        n = int(round(10 ** rng.uniform(1.0, 2.17 if mode == "fp64" else 2.4)))
        if mode == "fp64" and rng.random() < 0.3:
            nb = rng.randint(5, n)
            return dict(kind="ao2mo", n=n, nmo=max(2, n - rng.randint(0, 4)), n2=nb, nmo2=max(2, nb - rng.randint(0, 3)),
                        mode=mode)
        return dict(kind="ao2mo", n=n, nmo=max(2, n - rng.randint(0, n // 8)), mode=mode)
    if kind == "props":
        n = rng.randint(6, 12)
        na = rng.randint(2, n // 2)
        return dict(kind="props", n=n, na=na, nb=rng.randint(max(1, na - 1), na), level=rng.choice([0, 0, 2]),
                    nvec=rng.randint(1, 5))
    n = rng.randint(7, 10)
    na = rng.randint(3, n // 2)
    return dict(kind="davidson", n=n, na=na, nb=na, level=0, nvec=rng.randint(1, 4))


# ---- inputs ------------------------------------------------------------------------------------------------------
def _levels(n, na, nb, level):
    """Excitation limits: 0 is full CI."""
    fa, fb = min(na, n - na), min(nb, n - nb)
    return [fa, fb, fa + fb] if level == 0 else [min(level, fa), min(level, fb), level]


def _problem(c, seed):
    """Keyword arguments of POLYQUANT_DETSET."""
    if c["kind"] == "sigma2":
        he, hp, ee, pp, ep = synthetic.ep_integrals(c["ne"], c["np"], seed)
        return dict(n_orb=[c["ne"], c["np"]], n_alpha=[c["ea"], c["pa"]], n_beta=[c["eb"], c["pb"]],
                    h1=[[he, he], [hp, hp]], eri={(0, 0, 0, 0): ee, (1, 0, 1, 0): pp, (0, 0, 1, 0): ep},
                    excitation_level=[_levels(c["ne"], c["ea"], c["eb"], 0), _levels(c["np"], c["pa"], c["pb"], 0)],
                    restricted=[1, 1], charge=[-1.0, 1.0],
                    max_collective_excitation_level=c["level"] if c["level"] else INT_MAX)
    h, eri = synthetic.fci_integrals(c["n"], seed)
    return dict(n_orb=[c["n"]], n_alpha=[c["na"]], n_beta=[c["nb"]], h1=[[h, h]], eri={(0, 0, 0, 0): eri},
                excitation_level=[_levels(c["n"], c["na"], c["nb"], c["level"])], restricted=[1], charge=[-1.0])


def _batch_problems(c, seed):
    specs = [s for s in synthetic.batch_specs(4 * c["count"], seed=c["pick"]) if synthetic.batch_spec_dets(s) <= 400_000]
    return [synthetic.batch_problem(dict(s, seed=(seed * 1009 + i) % (1 << 31))) for i, s in enumerate(specs[:c["count"]])]


def _vectors(n_dets, nvec, seed):
    """nvec CI vectors as a program holds them: one contiguous column each."""
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    x = torch.randn(nvec, n_dets, device="cuda", dtype=torch.float64, generator=g)
    x *= torch.pow(10.0, torch.rand(nvec, n_dets, device="cuda", dtype=torch.float64, generator=g).mul_(-4.0))
    return x.div_(x.norm(dim=1, keepdim=True)).t()


def _ao_inputs(c, seed):
    """AO integrals on the device (8-fold packed for one basis, a pair matrix for two) and the MO coefficients."""
    g = torch.Generator(device="cuda").manual_seed(int(seed))

    def factor(n):
        i, j = torch.tril_indices(n, n, device="cuda")
        b = torch.randn(min(1024, 4 * n), i.numel(), device="cuda", dtype=torch.float64, generator=g)
        return b.mul_(torch.exp(-(i - j).abs().double() / 16.0))

    def coefficients(n, m):
        q, _ = torch.linalg.qr(torch.randn(n, n, device="cuda", dtype=torch.float64, generator=g))
        return q[:, :m].t().contiguous().t()

    B = factor(c["n"])
    C = coefficients(c["n"], c["nmo"])
    if "n2" in c:
        P = factor(c["n2"])
        L = min(B.shape[0], P.shape[0])
        return (P[:L].t() @ B[:L]).contiguous(), C, coefficients(c["n2"], c["nmo2"])
    M = torch.mm(B.t().float(), B.float()).double() if c["n"] > 160 else torch.mm(B.t(), B)
    del B
    return M[torch.ones(M.shape, dtype=torch.bool, device="cuda").tril_()], C, None


def prepare(case, seed):
    c, k = case, case["kind"]
    if k == "ao2mo":
        eri, C, C2 = _ao_inputs(c, seed)
        return dict(case=c, eri=eri, C=C, C2=C2)
    if k == "batch":
        b = CIBatch(_batch_problems(c, seed))
        return dict(case=c, op=b, C=[_vectors(n, c["nvec"], seed + 17 * i) for i, n in enumerate(b.n_dets)])
    op = POLYQUANT_DETSET(**_problem(c, seed))
    return dict(case=c, op=op, C=None if k == "davidson" else _vectors(op.N_dets, c["nvec"], seed))


def run(state):
    c, k = state["case"], state["case"]["kind"]
    if k in ("sigma", "sigma2", "batch"):
        return state["op"].sigma(state["C"], precision=PREC[c["prec"]])
    if k == "ham":
        nnz = state["op"].create_ham()
        return nnz, state["op"].sigma(state["C"])
    if k == "ao2mo":
        return ao2mo(state["eri"], state["C"], state["C2"], layout=PQ_AO_PACKED8 if state["C2"] is None else PQ_AO_PAIRS,
                     mode=MODE[c["mode"]])
    if k == "props":
        return (state["op"].s2(state["C"]), state["op"].rdm1(state["C"][:, 0], spin=0),
                state["op"].rdm1(state["C"][:, 0], spin=1))
    e, v, _ = state["op"].davidson(num_states=c["nvec"], num_subspace_vec=2 * c["nvec"], convergence_E=1e-8,
                                   return_vectors=True)
    return e, v


# ---- the operators in 64 bits ------------------------------------------------------------------------------------
def _strings(n, ne, kmax):
    """Occupation masks and their levels: the Fermi string, then by level, holes outer, particles inner."""
    masks, lev = [(1 << ne) - 1], [0]
    for k in range(1, min(kmax, ne) + 1):
        for o in itertools.combinations(range(ne), k):
            for v in itertools.combinations(range(ne, n), k):
                masks.append(((1 << ne) - 1) ^ sum(1 << x for x in o) ^ sum(1 << x for x in v))
                lev.append(k)
    return np.array(masks, dtype=np.int64), np.array(lev)


def _between(m, a, b):
    lo, hi = np.minimum(a, b), np.maximum(a, b)
    return np.bitwise_count(m & ((np.int64(1) << hi) - 1) & ~((np.int64(2) << lo) - 1)) & 1


def _bit(x):
    return np.round(np.log2(np.maximum(x, 1).astype(np.float64))).astype(np.int64)


def _pair(i, j):
    hi, lo = np.maximum(i, j), np.minimum(i, j)
    return hi * (hi + 1) // 2 + lo


class _Axis:
    """One spin list: its one-particle operators (from, to, pair, sign) and its own Hamiltonian, dense."""

    def __init__(self, n, ne, kmax, h, eri):
        self.m, self.lev = _strings(n, ne, kmax)
        self.n, self.ns, self.npair = n, len(self.m), n * (n + 1) // 2
        occ = ((self.m[:, None] >> np.arange(n)) & 1).astype(np.float32)
        diff = ne - occ @ occ.T
        H = np.zeros((self.ns, self.ns))
        d = _pair(np.arange(n), np.arange(n))
        ob = occ.astype(np.float64)
        J = eri[np.ix_(d, d)]
        i, j = np.meshgrid(np.arange(n), np.arange(n), indexing="ij")
        K = eri[_pair(i, j), _pair(i, j)]
        H[np.arange(self.ns), np.arange(self.ns)] = ob @ np.diag(h) + 0.5 * np.einsum("si,ij,sj->s", ob, J - K, ob)
        self.I1, self.J1 = np.nonzero(diff == 1)
        a, b = self.m[self.I1], self.m[self.J1]
        hole, part = _bit(a & ~b), _bit(b & ~a)
        self.pair1, self.sign1 = _pair(hole, part), 1.0 - 2.0 * _between(a, hole, part)
        for k in range(0, len(a), 1 << 18):
            s = slice(k, k + (1 << 18))
            f = h[hole[s], part[s]].copy()
            for o in range(n):
                g = eri[self.pair1[s], d[o]] - eri[_pair(hole[s], o), _pair(np.full_like(hole[s], o), part[s])]
                f += ob[self.I1[s], o] * g
            H[self.I1[s], self.J1[s]] = self.sign1[s] * f
        I2, J2 = np.nonzero(diff == 2)
        a, b = self.m[I2], self.m[J2]
        x, y = a & ~b, b & ~a
        h0, p0 = x & -x, y & -y
        h1, p1 = _bit(x ^ h0), _bit(y ^ p0)
        mid = a ^ h0 ^ p0
        h0, p0 = _bit(h0), _bit(p0)
        sg = 1.0 - 2.0 * (_between(a, h0, p0) ^ _between(mid, h1, p1))
        H[I2, J2] = sg * (eri[_pair(h0, p0), _pair(h1, p1)] - eri[_pair(h0, p1), _pair(h1, p0)])
        self.n1, self.n2 = len(self.I1), len(I2)
        self.H = torch.from_numpy(H).cuda()
        st, o = np.nonzero(occ)
        I = np.concatenate([self.I1, st])
        Jn = np.concatenate([self.J1, st])
        P = np.concatenate([self.pair1, d[o]])
        S = np.concatenate([self.sign1, np.ones(len(st))])
        order = np.argsort(P, kind="stable")
        cut = np.searchsorted(P[order], np.arange(self.npair + 1))
        dev = [torch.from_numpy(v[order]).cuda() for v in (I, Jn, S)]
        self.ops = [tuple(v[cut[p]:cut[p + 1]] for v in dev) for p in range(self.npair)]


def _axes_of(pb):
    axes, coupling = [], []
    ns = len(pb["n_orb"])
    for s in range(ns):
        for sp, ne in enumerate((pb["n_alpha"][s], pb["n_beta"][s])):
            lev = pb["excitation_level"][s]
            axes.append(_Axis(pb["n_orb"][s], ne, min(lev[sp], lev[2]), pb["h1"][s][0], pb["eri"][(s, 0, s, 0)]))
    for x in range(2 * ns):
        for y in range(x + 1, 2 * ns):
            s, t = x // 2, y // 2
            f = 1.0 if s == t else pb["charge"][0] * pb["charge"][1]
            coupling.append((x, y, f * pb["eri"][(s, 0, t, 0)]))
    lv = [a.lev.reshape([-1 if i == k else 1 for i in range(2 * ns)]) for k, a in enumerate(axes)]
    mask = np.ones([a.ns for a in axes], dtype=bool)
    tot = np.zeros(mask.shape, dtype=np.int64)
    for s in range(ns):
        e = lv[2 * s] + lv[2 * s + 1]
        mask &= e <= pb["excitation_level"][s][2]
        tot = tot + e
    mask &= tot <= pb.get("max_collective_excitation_level", INT_MAX)
    return axes, coupling, torch.from_numpy(mask).cuda()


def _apply(axis, x, k):
    """e_P x along axis k for every pair P (a new leading axis)."""
    y = x.movedim(k, 0)
    t = torch.zeros((axis.npair,) + tuple(y.shape), dtype=torch.float64, device=x.device)
    for p, (I, J, s) in enumerate(axis.ops):
        if len(I):
            t[p].index_add_(0, I, y[J] * s.reshape([-1] + [1] * (y.dim() - 1)))
    return t


def _exact_sigma(pb, C):
    axes, coupling, mask = _axes_of(pb)
    out = torch.zeros_like(C)
    for v in range(C.shape[1]):
        x = torch.zeros(mask.shape, dtype=torch.float64, device="cuda")
        x[mask] = C[:, v]
        y = torch.zeros_like(x)
        for k, a in enumerate(axes):
            y += torch.tensordot(a.H, x, dims=([1], [k])).movedim(0, k)
        for kx, ky, M in coupling:
            t = _apply(axes[ky], x, ky)
            g = (torch.from_numpy(np.ascontiguousarray(M)).cuda() @ t.reshape(t.shape[0], -1)).reshape((-1,) + t.shape[1:])
            del t
            for p, (I, J, s) in enumerate(axes[kx].ops):
                if len(I):
                    z = g[p].movedim(0, ky).movedim(kx, 0)
                    y.movedim(kx, 0).index_add_(0, I, z[J] * s.reshape([-1] + [1] * (z.dim() - 1)))
            del g
        out[:, v] = y[mask]
    return out


def _exact_ao2mo(eri, c, C, C2):
    """(ij|kl) from the full pair matrix, one index after the other."""
    n, n2 = c["n"], c.get("n2", c["n"])
    C2 = C if C2 is None else C2
    np1, np2 = n * (n + 1) // 2, n2 * (n2 + 1) // 2
    if "n2" in c:
        M = eri
    else:
        M = torch.zeros(np1, np1, dtype=torch.float64, device="cuda")
        M[torch.ones(M.shape, dtype=torch.bool, device="cuda").tril_()] = eri
        M = M + M.tril(-1).t()

    def half(R, n, C):
        """rows of pairs of an n-function basis -> pairs of C's columns."""
        i, j = torch.tril_indices(n, n, device="cuda")
        a, b = torch.tril_indices(C.shape[1], C.shape[1], device="cuda")
        out = torch.empty(R.shape[0], len(a), dtype=torch.float64, device="cuda")
        step = max(1, (1 << 27) // (n * n))
        for r in range(0, R.shape[0], step):
            s = torch.empty(R[r:r + step].shape[0], n, n, dtype=torch.float64, device="cuda")
            s[:, i, j] = R[r:r + step]
            s[:, j, i] = R[r:r + step]
            out[r:r + step] = (C.t() @ (s @ C))[:, a, b]
        return out

    h = half(M, n, C)              # rows: pairs of the second basis
    del M
    return half(h.t().contiguous(), n2, C2)


def _exact_props(pb, C):
    axes, _, mask = _axes_of(pb)
    a, b = axes
    na, nb = pb["n_alpha"][0], pb["n_beta"][0]
    n, s2, rdm = a.n, [], []
    off = _pair(*np.meshgrid(np.arange(n), np.arange(n), indexing="ij"))
    for v in range(C.shape[1]):
        x = torch.zeros(mask.shape, dtype=torch.float64, device="cuda")
        x[mask] = C[:, v]
        if v == 0:
            for k, ax in enumerate(axes):
                d = (_apply(ax, x, k) * x.movedim(k, 0)).reshape(ax.npair, -1).sum(1).cpu().numpy()
                rdm.append(np.where(np.eye(n, dtype=bool), d[off], 0.5 * d[off]))
        w = float((x * x).sum()) * ((na - nb) ** 2 / 4.0 + (na + nb) / 2.0)
        # minus the sum over ordered (p, q) of <E^alpha_pq E^beta_qp>: the two spins move in opposite directions
        xs = x.cpu().numpy()
        for oa, ob in zip(a.ops, b.ops):
            if not len(oa[0]) or not len(ob[0]):
                continue
            (Ia, Ja, sa), (Ib, Jb, sb) = ([t.cpu().numpy() for t in o] for o in (oa, ob))
            da, db = np.sign(a.m[Ia] - a.m[Ja]), np.sign(b.m[Ib] - b.m[Jb])
            for way in (-1, 0, 1):
                ka, kb = da == way, db == -way
                w -= float(np.einsum("ij,ij,i,j->", xs[np.ix_(Ia[ka], Ib[kb])], xs[np.ix_(Ja[ka], Jb[kb])], sa[ka], sb[kb]))
        s2.append(w)
    return np.array(s2), rdm[0], rdm[1]


def exact(case, seed):
    c, k = case, case["kind"]
    if k == "ao2mo":
        eri, C, C2 = _ao_inputs(c, seed)
        return _exact_ao2mo(eri, c, C, C2)
    if k == "batch":
        pbs = _batch_problems(c, seed)
        return [_exact_sigma(pb, _vectors(_count(pb), c["nvec"], seed + 17 * i)) for i, pb in enumerate(pbs)]
    if k == "sigma" and comb(c["n"], c["na"]) * comb(c["n"], c["nb"]) > 2e7 and c["level"] == 0:
        return None
    pb = _problem(c, seed)
    if k == "davidson":
        nd = _count(pb)
        if nd > 5000:
            return None
        H = _exact_sigma(pb, torch.eye(nd, dtype=torch.float64, device="cuda"))
        w = torch.linalg.eigvalsh(H).cpu().numpy()
        return w[:c["nvec"]], None
    C = _vectors(_count(pb), c["nvec"], seed)
    if k == "props":
        return _exact_props(pb, C)
    s = _exact_sigma(pb, C)
    return (None, s) if k == "ham" else s


# ---- the work of one pass ----------------------------------------------------------------------------------------
def _list_counts(n, ne, kmax):
    return [comb(ne, k) * comb(n - ne, k) for k in range(min(kmax, ne, n - ne) + 1)]


def _count(pb):
    from itertools import product

    per = []
    for s in range(len(pb["n_orb"])):
        lev = pb["excitation_level"][s]
        a = _list_counts(pb["n_orb"][s], pb["n_alpha"][s], lev[0])
        b = _list_counts(pb["n_orb"][s], pb["n_beta"][s], lev[1])
        per.append([(i + j, x * y) for (i, x), (j, y) in product(enumerate(a), enumerate(b)) if i + j <= lev[2]])
    mc = pb.get("max_collective_excitation_level", INT_MAX)
    return sum(int(np.prod([t[1] for t in combo])) for combo in product(*per) if sum(t[0] for t in combo) <= mc)


def _adjacency(n, ne, kmax):
    """Singles and doubles that lead from a string of level x (x holes, x particles) to level y, as [x, y] counts."""
    m, v = min(kmax, ne, n - ne), n - ne
    s, d = np.zeros((m + 1, m + 1)), np.zeros((m + 1, m + 1))
    for x in range(m + 1):
        for y in range(m + 1):
            s[x, y] = {1: (ne - x) * (v - x), 0: x * (ne - x) + x * (v - x), -1: x * x}.get(y - x, 0)
            # u of the two orbitals emptied are particles, w of the two filled are holes
            d[x, y] = sum(comb(x, u) * comb(ne - x, 2 - u) * comb(x, w) * comb(v - x, 2 - w) for u in range(3)
                          for w in range(3) if y - x == 2 - u - w)
    return s, d


def _connections(pb):
    """Nonzero elements of H in the determinant list (the diagonal included), from the level structure."""
    from itertools import product

    ns = len(pb["n_orb"])
    lists, adj = [], []
    for s in range(ns):
        for sp, ne in enumerate((pb["n_alpha"][s], pb["n_beta"][s])):
            kmax = pb["excitation_level"][s][sp]
            lists.append(_list_counts(pb["n_orb"][s], ne, kmax))
            adj.append(_adjacency(pb["n_orb"][s], ne, kmax))
    mc = pb.get("max_collective_excitation_level", INT_MAX)

    def kept(t):
        return all(t[2 * s] + t[2 * s + 1] <= pb["excitation_level"][s][2] for s in range(ns)) and sum(t) <= mc

    total = 0.0
    for t in product(*(range(len(x)) for x in lists)):
        if not kept(t):
            continue
        row = 1.0
        for k in range(2 * ns):
            for y in range(len(lists[k])):
                if kept(t[:k] + (y,) + t[k + 1:]):
                    row += adj[k][0][t[k], y] + adj[k][1][t[k], y]
            for j in range(k + 1, 2 * ns):
                for y in range(len(lists[k])):
                    for z in range(len(lists[j])):
                        if adj[k][0][t[k], y] and adj[j][0][t[j], z] and kept(t[:k] + (y,) + t[k + 1:j] + (z,) + t[j + 1:]):
                            row += adj[k][0][t[k], y] * adj[j][0][t[j], z]
        total += row * np.prod([float(lists[k][t[k]]) for k in range(2 * ns)])
    return total


def work(case):
    c, k = case, case["kind"]
    if k == "ao2mo":
        n, m, n2, m2 = c["n"], c["nmo"], c.get("n2", c["n"]), c.get("nmo2", c["nmo"])
        pa, pb_, qa, qb = n * (n + 1) // 2, n2 * (n2 + 1) // 2, m * (m + 1) // 2, m2 * (m2 + 1) // 2
        src = pa * pb_ if "n2" in c else pa * (pa + 1) // 2
        flops = 2.0 * pb_ * (n * n * m + n * m * m) + 2.0 * qa * (n2 * n2 * m2 + n2 * m2 * m2)
        return {"bytes": 8.0 * (src + qa * qb + n * m + n2 * m2), "flops": flops}
    pbs = _batch_problems(c, 0) if k == "batch" else [_problem(c, 0)]
    nd = sum(_count(p) for p in pbs)
    nv = c["nvec"]
    if k == "props":
        p = pbs[0]
        n1 = p["n_alpha"][0] * (c["n"] - p["n_alpha"][0]) + p["n_beta"][0] * (c["n"] - p["n_beta"][0])
        return {"bytes": 8.0 * nd * nv, "flops": 2.0 * nd * (n1 + nv * n1 / 4.0)}
    nnz = sum(_connections(p) for p in pbs)
    if k == "davidson":  # one pass over a basis of that size, a dozen times
        return {"bytes": 12 * 16.0 * nd * nv, "flops": 12 * 2.0 * nnz * nv}
    if k == "ham":
        return {"bytes": 12.0 * nnz + 16.0 * nd * nv, "flops": 2.0 * nnz * (nv + 1)}
    return {"bytes": 16.0 * nd * nv + 8.0 * nd, "flops": 2.0 * nnz * nv}
