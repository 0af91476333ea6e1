"""The work this framework does for a user's program, as timed cases.

A program that solves a selected-CI problem loads integrals and alpha/beta
strings, multiplies vectors with the Hamiltonian (the sigma product, FP64 or
with FP32 storage, on device or on host buffers, on the fly or with the
stored matrix), projects them on its subspace, solves for eigenpairs and
reduces the result to densities and derivatives. Every case goes through the
package's public entry points (sbdx.Context). Integrals and strings follow
the synthetic laws of sbdx.synth; a case's seed draws all of them.

`exact` restates each path in plain torch, FP64: H = sum h_pq E_pq
+ 1/2 sum (pq|rs) (E_pq E_rs - delta_qr E_ps) over the interleaved spin
orbitals (alpha p -> 2p, beta p -> 2p + 1).
"""
import functools
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if os.path.join(ROOT, "sbd-ykt_b200") not in sys.path:
    sys.path.insert(0, os.path.join(ROOT, "sbd-ykt_b200"))

import sbdx  # noqa: E402
from sbdx import synth  # noqa: E402

DEV = "cuda" if torch.cuda.is_available() else "cpu"


# ---- the cases ---------------------------------------------------------------


def listed():
    return [
        # a water-sized product (275 strings per spin, the smallest set of the
        # reference's h2o data): every Davidson step of a small molecule, launch latency
        dict(name="sigma64-275x275", kind="sigma", precision=64, L=24, n=5, na=275, nb=275),
        # one uneven, odd-sized subspace of a batch (200 to 4000 strings per spin, L = 40), FP32 storage
        dict(name="sigma32-613x1187", kind="sigma", precision=32, L=40, n=8, na=613, nb=1187),
        # the differentiation workload's product, FP64
        dict(name="sigma64-2000x2000", kind="sigma", precision=64, L=32, n=6, na=2000, nb=2000),
        # the headline product: 64 M determinants at L = 58, in both storage types
        dict(name="sigma64-8000x8000", kind="sigma", precision=64, L=58, n=7, na=8000, nb=8000),
        dict(name="sigma32-8000x8000", kind="sigma", precision=32, L=58, n=7, na=8000, nb=8000),
        # a host program's product: page-locked C in, S out
        dict(name="host64-4003x3997", kind="host", L=58, n=7, na=4003, nb=3997),
        # the product with the stored Hamiltonian (the reference's method 1)
        dict(name="stored64-1000x1000", kind="stored", L=24, n=5, na=1000, nb=1000),
        # the subspace projection of a Davidson step: a mixed solver's (FP32
        # corrections, two roots) and an FP64 one on an odd vector length
        dict(name="project32-24x2", kind="project", precision=32, D=32000000, m=24, nx=2),
        dict(name="project64-13x1", kind="project", precision=64, D=11998999, m=13, nx=1),
        # the energy's adjoint with respect to the integrals (1- and 2-RDM of the root inside)
        dict(name="backward-2000x2000", kind="backward", L=32, n=6, na=2000, nb=2000),
        # a whole diag call on new strings: connectivity, FP64 Davidson, densities and RDMs
        dict(name="diag64-400x400", kind="diag", L=24, n=5, na=400, nb=400),
        # a two-root mixed-precision solve of one subspace, with both roots' densities
        dict(name="roots32-613x1187", kind="roots", L=40, n=8, na=613, nb=1187),
    ]


SPACES = ((24, 5), (32, 6), (40, 8), (58, 7))  # orbitals, electrons per spin


def draw(rng):
    def log(lo, hi):
        return int(round(lo * (hi / lo) ** rng.random()))

    kind = rng.choice(("sigma", "sigma", "sigma", "sigma", "host", "stored", "project", "project", "backward", "diag",
                       "roots"))
    if kind == "project":
        nx = rng.randint(1, 4)
        m, precision = log(1, 40), rng.choice((32, 64))
        return dict(kind=kind, precision=precision, D=log(100000, min(32000000, 1500000000 // (m + nx) * 32 // precision)),
                    m=m, nx=nx)
    L, n = rng.choice(SPACES)
    lo, hi = dict(sigma=(150, 8000), host=(500, 4000), stored=(150, 1000), backward=(150, 2000), diag=(100, 450),
                  roots=(200, 850))[kind]
    case = dict(kind=kind, L=L, n=n, na=log(lo, hi), nb=log(lo, hi))
    if kind == "sigma":
        case["precision"] = rng.choice((32, 64))
    return case


# ---- inputs ------------------------------------------------------------------


def problem(case, seed):
    """Integrals and strings of the case's law, all drawn from the seed."""
    L, n = case["L"], case["n"]
    I0, h, eri = synth.make_integrals(L, 96, 10 * seed + 1)
    a = synth.sample_strings(L, n, case["na"], 10 * seed + 2)
    b = synth.sample_strings(L, n, case["nb"], 10 * seed + 3)
    return synth.Problem(L=L, nelec=2 * n, I0=I0, h=h, eri=eri, alpha=a, beta=b)


def ci_vector(prob, seed):
    """A normalised CI vector: amplitudes fall with the excitation rank of the
    alpha and of the beta string, as a converged or trial vector's do."""
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    n = prob.nelec // 2

    def fall(s):
        rank = n - np.bitwise_count(s & np.uint64((1 << n) - 1)).astype(np.int64)
        return torch.from_numpy(0.3 ** rank).to(DEV)

    C = torch.randn((prob.na, prob.nb), dtype=torch.float64, device=DEV, generator=g)
    C *= fall(prob.alpha)[:, None]
    C *= fall(prob.beta)[None, :]
    return (C / C.norm()).reshape(-1)


def vectors(case, seed):
    """A projection's operands: m subspace vectors and nx new ones of unit
    length (to the precision of the draw), and room for the dots."""
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    t = torch.float32 if case["precision"] == 32 else torch.float64
    D, m, nx = case["D"], case["m"], case["nx"]
    V = torch.randn((m, D), dtype=t, device=DEV, generator=g).mul_(D ** -0.5)
    X = torch.randn((nx, D), dtype=t, device=DEV, generator=g).mul_(D ** -0.5)
    # new vectors overlap the subspace before they are orthogonalised
    X += V[:nx] if m >= nx else V[:1]
    return V, X, torch.empty((m, nx), dtype=torch.float64, device=DEV)


def prepare(case, seed):
    kind = case["kind"]
    ctx = sbdx.Context(0)
    if kind == "project":
        V, X, P = vectors(case, seed)
        return dict(case=case, ctx=ctx, V=V, X=X, P=P)
    prob = problem(case, seed)
    if kind == "diag":  # the strings are new in every call of diag
        ctx.set_integrals(prob.L, prob.I0, prob.h, prob.eri)
        return dict(case=case, ctx=ctx, alpha=prob.alpha, beta=prob.beta)
    ctx.load(prob)
    if kind != "backward":  # the adjoint rebuilds its lists itself
        ctx.build_connectivity()
    if kind == "roots":
        return dict(case=case, ctx=ctx)
    if kind == "stored":
        ctx.build_hamiltonian()
    X = ci_vector(prob, seed)
    if kind == "sigma" and case["precision"] == 32:
        X = X.float()
    if kind == "host":
        X = X.cpu().pin_memory()
        return dict(case=case, ctx=ctx, X=X, S=torch.empty_like(X).pin_memory())
    return dict(case=case, ctx=ctx, X=X, S=torch.empty_like(X))


# ---- one pass ----------------------------------------------------------------


def run(state):
    case, ctx = state["case"], state["ctx"]
    kind = case["kind"]
    if kind in ("sigma", "stored"):
        precision = sbdx.SBDX_FP32 if case.get("precision") == 32 else sbdx.SBDX_FP64
        ctx.sigma_device(precision, state["X"].data_ptr(), state["S"].data_ptr())
        return state["S"]
    if kind == "host":
        ctx.sigma_host_ptr(state["X"].data_ptr(), state["S"].data_ptr())
        return state["S"]
    if kind == "project":
        V, X, P = state["V"], state["X"], state["P"]
        precision = sbdx.SBDX_FP32 if case["precision"] == 32 else sbdx.SBDX_FP64
        ctx.project_device(precision, V.data_ptr(), V.shape[1], V.shape[0], X.data_ptr(), X.shape[1], X.shape[0],
                           V.shape[1], P.data_ptr())
        return P
    if kind == "backward":
        dh, deri = ctx.energy_backward_device(state["X"].data_ptr())
        return dict(dh=dh, deri=deri)
    if kind == "diag":
        ctx.set_strings(state["alpha"], state["beta"])
        info, _ = ctx.davidson(max_it=10, max_nb=16, eps=1e-8, to_host=False)
        W = ctx.wavefunction_device()
        one, two = ctx.rdm_device(W)
        return dict(energy=info.energy, density=ctx.occupation_device(W), weights=ctx.alpha_weights_device(W), one=one,
                    two=two)
    info, E, res, _ = ctx.davidson_roots(2, max_it=100, max_nb=12, eps=1e-8, precision=sbdx.SBDX_FP32, to_host=False)
    W = [ctx.wavefunction_device(r) for r in range(2)]
    return dict(energies=E, density=[ctx.occupation_device(w) for w in W],
                one=[ctx.rdm_device(w, two=False)[0] for w in W])


# ---- what a pass cannot do without -------------------------------------------


@functools.lru_cache(maxsize=64)
def det_pairs(L, n, na, nb):
    """Pairs of determinants with a non-zero element, the diagonal included."""

    def counts(N, seed):
        s = synth.sample_strings(L, n, N, seed)
        one = two = 0
        for r in range(0, N, 512):
            d = np.bitwise_count(s[r:r + 512, None] ^ s[None, :])
            one += int(np.count_nonzero(d == 2))
            two += int(np.count_nonzero(d == 4))
        return one, two

    (sa, da), (sb, db) = counts(na, 2), counts(nb, 3)
    return na * nb + nb * (sa + da) + na * (sb + db) + sa * sb


def work(case):
    kind = case["kind"]
    if kind == "project":
        D, m, nx = case["D"], case["m"], case["nx"]
        return {"bytes": (m + nx) * D * case["precision"] // 8 + 8 * m * nx, "flops": 2 * m * nx * D}
    L, na, nb = case["L"], case["na"], case["nb"]
    D, pairs = na * nb, det_pairs(L, case["n"], na, nb)
    fixed = 8 * (synth.neri(L) + L * L + na + nb)
    if kind == "stored":  # 12 bytes per stored element, the diagonal, both vectors
        return {"bytes": 12 * (pairs - D) + 8 * D * 4, "flops": 2 * pairs}
    if kind == "backward":
        return {"bytes": 8 * D + fixed + 8 * (synth.neri(L) + L * L), "flops": 2 * pairs}
    if kind in ("diag", "roots"):  # at least a dozen products and vector updates of a converging solve
        steps = 12 * (2 if kind == "roots" else 1)
        word = 4 if kind == "roots" else 8
        return {"bytes": steps * 4 * word * D + fixed, "flops": steps * 2 * pairs}
    return {"bytes": 2 * case.get("precision", 64) // 8 * D + fixed, "flops": 2 * pairs}


def tolerance(case):
    kind = case["kind"]
    if kind in ("sigma", "host", "stored"):
        # FP64 sums of a few hundred terms in another order; FP32 storage of
        # vectors and integrals, short FP32 sums, FP64 row accumulation
        # (measured against 64-bit sums: 2.5e-8 and 0.5 to 1.8e-15)
        return {"rel": 1e-7, "max": 4e-6} if case.get("precision") == 32 else {"rel": 8e-15, "max": 1e-12}
    if kind == "project":  # FP64 products and sums over D (measured 1 to 2e-16)
        return {"rel": 2e-15, "max": 1e-13}
    if kind == "backward":  # FP64 sums over all determinants (measured 4 to 10e-16)
        return {"rel": 4e-15, "max": 1e-12}
    # solves converged to a residual of 1e-8: energies to its square, densities to the residual
    return {"rel": 1e-7, "max": 1e-5}


# ---- the same in plain torch, 64 bits ----------------------------------------


def pair(p, q):
    hi, lo = np.maximum(p, q), np.minimum(p, q)
    return hi * (hi + 1) // 2 + lo


def orb(bit):  # orbital of an isolated bit
    return np.log2(bit.astype(np.float64)).astype(np.int64)


def between(p, q):  # mask of the orbitals strictly between p and q
    lo, hi = np.minimum(p, q).astype(np.uint64), np.maximum(p, q).astype(np.uint64)
    one = np.uint64(1)
    return ((one << hi) - one) & ~((one << (lo + one)) - one)


def excitations(s):
    """Singles (bra, ket, particle a, hole i, sign) and doubles (bra, ket, a, b,
    i, j, sign) among the strings, from E_ai and E_bj E_ai on the ket."""
    rs, rd = [], []
    for r in range(0, len(s), 512):
        d = np.bitwise_count(s[r:r + 512, None] ^ s[None, :])
        for want, out in ((2, rs), (4, rd)):
            x, k = np.nonzero(d == want)
            out.append(np.stack([x + r, k]))
    one = np.uint64(1)

    def lowest(x):
        return x & (~x + one)

    (r1, k1), (r2, k2) = np.concatenate(rs, 1), np.concatenate(rd, 1)
    a, i = orb(s[r1] & ~s[k1]), orb(s[k1] & ~s[r1])
    singles = (r1, k1, a, i, 1.0 - 2.0 * (np.bitwise_count(s[k1] & between(a, i)) & 1))
    part, hole = s[r2] & ~s[k2], s[k2] & ~s[r2]
    pl, hl = lowest(part), lowest(hole)
    a, b, i, j = orb(pl), orb(part ^ pl), orb(hl), orb(hole ^ hl)
    mid = s[k2] ^ hl ^ pl
    par = np.bitwise_count(s[k2] & between(a, i)) + np.bitwise_count(mid & between(b, j))
    return singles, (r2, k2, a, b, i, j, 1.0 - 2.0 * (par & 1))


def put(x):
    return torch.from_numpy(np.ascontiguousarray(x)).to(DEV)


class Exact:
    """H on the product basis in the ordering "all alpha, then all beta"."""

    def __init__(self, prob):
        self.prob, L = prob, prob.L
        P = L * (L + 1) // 2
        x, y = np.tril_indices(P)
        V = np.zeros((P, P))
        V[x, y] = V[y, x] = prob.eri
        self.V, self.h = V, prob.h.reshape(L, L)
        p = np.arange(L)
        self.dd = pair(p, p)
        self.sides = [self.side(s) for s in (prob.alpha, prob.beta)]
        # sign of moving every beta operator behind the alpha ones: one for each
        # alpha orbital above a beta orbital
        occ_a, occ_b = self.sides[0]["occ"], self.sides[1]["occ"]
        above = occ_a.flip(1).cumsum(1).flip(1) - occ_a
        self.phi = 1.0 - 2.0 * ((above @ occ_b.T) % 2)

    def side(self, s):
        L, V, h = self.prob.L, self.V, self.h
        n = len(s)
        occ = ((s[:, None] >> np.arange(L, dtype=np.uint64)) & np.uint64(1)).astype(np.float64)
        singles, doubles = excitations(s)
        r, k, a, i, sg = singles
        q = np.arange(L)
        K = V[pair(a[:, None], q[None, :]), pair(q[None, :], i[:, None])]
        v1 = sg * (h[a, i] + (occ[k] * (V[pair(a, i)][:, self.dd] - K)).sum(1))
        r2, k2, a2, b2, i2, j2, sg2 = doubles
        v2 = sg2 * (V[pair(a2, i2), pair(b2, j2)] - V[pair(a2, j2), pair(b2, i2)])
        X = V[np.ix_(self.dd, self.dd)] - V[pair(q[:, None], q[None, :]), pair(q[:, None], q[None, :])]
        dg = occ @ np.diag(h) + 0.5 * ((occ @ X) * occ).sum(1)
        ar = np.arange(n)
        H = torch.sparse_coo_tensor(put(np.stack([np.concatenate([r, r2, ar]), np.concatenate([k, k2, ar])])),
                                    put(np.concatenate([v1, v2, dg])), (n, n)).coalesce()
        # E_pq entries, the number operators among them, by bra
        rn, qn = np.nonzero(occ)
        er, ek = np.concatenate([r, rn]), np.concatenate([k, rn])
        ep, es = np.concatenate([pair(a, i), self.dd[qn]]), np.concatenate([sg, np.ones(len(rn))])
        o = np.argsort(er, kind="stable")
        return dict(n=n, occ=put(occ), singles=singles, doubles=doubles, H=H, bra=er[o], ket=ek[o], pq=ep[o], sg=es[o])

    def opposite(self, use):
        """For blocks of beta bras of like list length: use(ib, C'-column lists)."""
        B = self.sides[1]
        off = np.searchsorted(B["bra"], np.arange(B["n"] + 1))
        length = np.diff(off)
        order = np.argsort(length, kind="stable")
        at = 0
        while at < len(order):
            m = int(length[order[at]])
            # columns per block: lists of like length, a few GB of workspace
            most = max(1, int(2.5e9 // (8 * len(self.V) * self.sides[0]["n"])))
            end = at + 1
            while end < len(order) and end - at < most and length[order[end]] <= max(1.2 * m, m + 4):
                end += 1
            ib = order[at:end]
            m = int(length[ib].max())
            idx = off[ib][:, None] + np.minimum(np.arange(m)[None, :], length[ib][:, None] - 1)
            sg = np.where(np.arange(m)[None, :] < length[ib][:, None], B["sg"][idx], 0.0)
            use(put(ib), put(B["ket"][idx]), put(B["pq"][idx]), put(sg))
            at = end

    def sigma(self, C):
        A, B = self.sides
        X = C.reshape(A["n"], B["n"]).double() * self.phi
        S = torch.sparse.mm(A["H"], X) + torch.sparse.mm(B["H"], X.T.contiguous()).T + self.prob.I0 * X
        V, Xt = put(self.V), X.T.contiguous()
        P = len(V)
        flat = put(A["pq"] * A["n"] + A["ket"])
        bra, sa = put(A["bra"]), put(A["sg"])

        def use(ib, jb, rs, sg):
            T = torch.bmm(V[rs].transpose(1, 2), Xt[jb] * sg[..., None])  # [column, pq, ja]
            g = T.reshape(len(ib), P * A["n"])[:, flat] * sa
            out = torch.zeros((len(ib), A["n"]), dtype=torch.float64, device=DEV)
            S[:, ib] += out.index_add_(1, bra, g).T

        self.opposite(use)
        return (S * self.phi).reshape(-1)

    def gradient(self, C):
        """dE/dh and dE/d(pq|rs) of <C|H|C>, by packed classes."""
        A, B = self.sides
        L, P = self.prob.L, len(self.V)
        X = C.reshape(A["n"], B["n"]).double() * self.phi
        Gh = torch.zeros((L, L), dtype=torch.float64, device=DEV)
        GV = torch.zeros(P * P, dtype=torch.float64, device=DEV)

        def add(x, y, v):
            GV.index_add_(0, put((x * P + y).reshape(-1)), v.reshape(-1))

        q = np.arange(L)
        for S, M in ((A, X @ X.T), (B, X.T @ X)):
            r, k, a, i, sg = S["singles"]
            v = M[put(r), put(k)] * put(sg)
            Gh.view(-1).index_add_(0, put(a * L + i), v)
            vo = v[:, None] * S["occ"][put(k)]
            add(np.repeat(pair(a, i)[:, None], L, 1), np.repeat(self.dd[None, :], len(a), 0), vo)
            add(pair(a[:, None], q[None, :]), pair(q[None, :], i[:, None]), -vo)
            r, k, a, b, i, j, sg = S["doubles"]
            v = M[put(r), put(k)] * put(sg)
            add(pair(a, i), pair(b, j), v)
            add(pair(a, j), pair(b, i), -v)
            w = M.diagonal()
            Gh.diagonal().add_(w @ S["occ"])
            pp = 0.5 * (S["occ"].T * w) @ S["occ"]
            add(np.repeat(self.dd[:, None], L, 1), np.repeat(self.dd[None, :], L, 0), pp)
            both = pair(q[:, None], q[None, :])
            add(both, both, -pp)
        Xt = X.T.contiguous()
        bra, ket, pq, sa = put(A["bra"]), put(A["ket"]), put(A["pq"]), put(A["sg"])
        g2 = GV.view(P, P)

        def use(ib, jb, rs, sg):
            for c in range(len(ib)):
                left = Xt[ib[c]][bra] * sa                    # [entries]
                T = torch.zeros((jb.shape[1], P), dtype=torch.float64, device=DEV)
                T.index_add_(1, pq, Xt[jb[c]][:, ket] * left)  # [beta entries, pq]
                g2.index_add_(1, rs[c], (T * sg[c][:, None]).T)

        self.opposite(use)
        dh = Gh + Gh.T - torch.diag(Gh.diagonal())
        g2 = g2 + g2.T - torch.diag(g2.diagonal())
        x, y = np.tril_indices(P)
        return dh.reshape(-1), g2[put(x), put(y)]


def exact(case, seed):
    kind = case["kind"]
    if kind == "project":
        V, X, _ = vectors(case, seed)
        return torch.stack([torch.stack([(v.double() * x.double()).sum() for x in X]) for v in V])
    if kind in ("diag", "roots"):  # converged vectors: compared with the start's
        return None
    prob = problem(case, seed)
    C = ci_vector(prob, seed)
    if case.get("precision") == 32:
        C = C.float()
    if kind == "backward":
        dh, deri = Exact(prob).gradient(C)
        return dict(dh=dh, deri=deri)
    return Exact(prob).sigma(C)
