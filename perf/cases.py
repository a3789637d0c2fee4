"""Timed cases of the exact-diagonalisation engine.

Each case is one call (or one short chain of calls) that a program built on
the engine makes, through the public entry points: products H*v of Hubbard
and Heisenberg sectors, Lanczos runs, whole solves, reduced densities,
batched Green's functions and the differentiable step.  ``listed`` gives the
fixed cases, ``draw`` more of the same ranges, ``prepare`` the inputs and
handles a program holds before the call, ``run`` the call, ``work`` the bytes
and operations it cannot do without, and ``exact`` the same outputs in
64-bit torch without the engine.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from pyhub_gb300 import _capi
from pyhub_gb300.core import gradients as GR
from pyhub_gb300.core import greens_batched as GB
from pyhub_gb300.core import lanczos as LZ
from pyhub_gb300.solver import FermiHubbard
from pyhub_gb300.tools import lattices as LT

OMEGA = 512        # frequencies of a Green's-function case
ETA = 0.05


def listed():
    return [
        # the product a small cluster's Lanczos or a dense diagonalisation repeats thousands of times: the
        # 8-site ring of the reference's own example sizes; latency counts
        dict(name="hv_f64_ring8", kind="hv", lattice="ring", lx=8, ly=1, nup=4, ndn=4, dtype="f64", dots=False),
        # the random-bond 14-site cluster of the differentiable workload, FP64 with the fused dots the
        # three-term recurrence uses
        dict(name="hv_f64_random14", kind="hv", lattice="random", lx=14, ly=1, nup=7, ndn=7, dtype="f64", dots=True),
        # the headline product: 4x4 periodic, half filling, FP32 vectors
        dict(name="hv_f32_4x4", kind="hv", lattice="square", lx=4, ly=4, nup=8, ndn=8, dtype="f32", dots=False),
        # Heisenberg products: an FP64 refinement step on 4x6 and the FP32 stage on 4x7
        dict(name="heis_hv_f64_4x6", kind="heis_hv", lattice="square", lx=4, ly=6, dtype="f64", dots=True),
        dict(name="heis_hv_f32_4x7", kind="heis_hv", lattice="square", lx=4, ly=7, dtype="f32", dots=True),
        # a whole small solve as the examples do it: ground state, density matrix, spin correlations
        dict(name="solve_ring8", kind="solve", lattice="ring", lx=8, ly=1, nup=4, ndn=4),
        # the FP64 full-reorthogonalisation Lanczos that kernel() takes for sectors up to 4M states (3x4 cluster)
        dict(name="lanczos_f64_3x4", kind="lanczos", lattice="square", lx=4, ly=3, nup=6, ndn=6, dtype="f64",
             steps=100),
        # the FP32 stage of the mixed solve on the headline cluster
        dict(name="lanczos_f32_4x4", kind="lanczos", lattice="square", lx=4, ly=4, nup=8, ndn=8, dtype="f32",
             steps=40),
        # density matrices, double occupancies and spin correlations of a 14-site state
        dict(name="rdm_random14", kind="rdm", lattice="random", lx=14, ly=1, nup=7, ndn=7),
        # all spin correlations of a 4x6 Heisenberg state
        dict(name="spincor_4x6", kind="heis_rdm", lattice="square", lx=4, ly=6),
        # Green's functions of eight 12-site clusters: every particle and hole start vector at once
        dict(name="greens_8x12", kind="greens", clusters=8, lx=4, ly=3, n=6, dtype="f32", steps=40),
        # the differentiable step: ground state, energy gradient and the adjoint gradient of a 1-RDM loss
        dict(name="gradients_random10", kind="gradients", lx=10, nup=5, ndn=5),
    ]


def _shape(rng, n):
    pick = rng.choice(["ring", "square", "random"])
    if pick == "square":
        for lx in (4, 3, 2):
            if n % lx == 0 and n // lx > 1:
                return "square", lx, n // lx
    return ("random" if pick == "random" else "ring"), n, 1


def draw(rng):
    kind = rng.choice(["hv", "hv", "heis_hv", "heis_hv", "solve", "lanczos", "lanczos", "rdm", "heis_rdm", "greens",
                       "gradients"])
    if kind == "hv":
        n = rng.randint(6, 16)
        lat, lx, ly = _shape(rng, n)
        top = 8 if n < 16 else 7
        nup, ndn = (min(top, max(1, n // 2 - rng.randint(0, 2))) for _ in range(2))
        return dict(kind=kind, lattice=lat, lx=lx, ly=ly, nup=nup, ndn=ndn, dtype=rng.choice(["f32", "f64"]),
                    dots=rng.random() < 0.5)
    if kind in ("heis_hv", "heis_rdm"):
        n = 2 * rng.randint(4, 14 if kind == "heis_hv" else 12)
        lat, lx, ly = _shape(rng, n)
        c = dict(kind=kind, lattice=lat, lx=lx, ly=ly)
        if kind == "heis_hv":
            c.update(dtype=rng.choice(["f32", "f64"]), dots=rng.random() < 0.5)
        return c
    if kind == "solve":
        # random bonds: a unique ground state
        n = rng.randint(6, 11)
        return dict(kind=kind, lattice="random", lx=n, ly=1, nup=n // 2, ndn=n // 2 - rng.randint(0, 1))
    if kind == "lanczos":
        f32 = rng.random() < 0.5
        n = rng.randint(11, 14) if f32 else rng.randint(9, 13)
        lat, lx, ly = _shape(rng, n)
        top = 40 if f32 else (100 if n > 10 else 50)
        return dict(kind=kind, lattice=lat, lx=lx, ly=ly, nup=n // 2, ndn=n // 2 - rng.randint(0, 1),
                    dtype="f32" if f32 else "f64", steps=rng.randint(16, top))
    if kind == "rdm":
        n = rng.randint(6, 14)
        lat, lx, ly = _shape(rng, n)
        return dict(kind=kind, lattice=lat, lx=lx, ly=ly, nup=n // 2, ndn=max(1, n // 2 - rng.randint(0, 2)))
    if kind == "greens":
        lx, ly = rng.choice([(3, 3), (5, 2), (4, 2), (6, 2), (4, 3)])
        return dict(kind=kind, clusters=rng.randint(1, 8), lx=lx, ly=ly, n=lx * ly // 2 - rng.randint(0, 1),
                    dtype=rng.choice(["f32", "f32", "f64"]), steps=rng.randint(12, 32))
    n = rng.randint(6, 10)
    return dict(kind=kind, lx=n, nup=n // 2, ndn=n // 2)


# ------------------------------------------------------------------ inputs

def _dt(case):
    return torch.float64 if case.get("dtype", "f64") == "f64" else torch.float32


def _hubbard(case, seed):
    """Hopping matrix and on-site U of the case (the interaction differs from seed to seed)."""
    n = case["lx"] * case.get("ly", 1)
    rng = np.random.default_rng(1000 + int(seed))
    if case["lattice"] == "random":
        t, U, _ = LT.random_bond_cluster(n, n // 2, int(seed))
        return t, U
    t = LT.ring(n) if case["lattice"] == "ring" else LT.square(case["lx"], case["ly"], -1.0, periodic=True)
    return t, np.full(n, float(rng.uniform(3.0, 9.0)))


def _heis(case):
    n = case["lx"] * case["ly"]
    if case["lattice"] == "square":
        return LT.square(case["lx"], case["ly"], 1.0, periodic=True)
    if case["lattice"] == "ring":
        return LT.ring(n, 1.0)
    t, _, _ = LT.random_bond_cluster(n, n // 2, n)
    np.fill_diagonal(t, 0.0)
    return t


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _randn(n, seed):
    v = torch.randn(n, generator=_gen(seed), dtype=torch.float64, device="cuda")
    return v / torch.linalg.vector_norm(v)


def _state(nsup, nsdn, ustr, dstr, seed):
    """A correlated many-body state: random amplitudes damped by 0.5 per doubly occupied site."""
    v = torch.randn(nsdn, nsup, generator=_gen(seed), dtype=torch.float64, device="cuda")
    both = dstr[:, None] & ustr[None, :]
    occ = torch.zeros_like(both)
    for b in range(32):
        occ += (both >> b) & 1
    v *= torch.pow(torch.tensor(0.5, dtype=torch.float64, device="cuda"), occ.double())
    return (v / torch.linalg.vector_norm(v)).reshape(-1)


def _clusters(case, seed):
    rng = np.random.default_rng(2000 + int(seed))
    out = []
    for _ in range(case["clusters"]):
        t = LT.square(case["lx"], case["ly"], -1.0, periodic=False, tp=float(rng.uniform(-0.3, 0.3)))
        out.append((t, float(rng.uniform(0.5, 8.0))))
    return out


def _gradient_inputs(case, seed):
    """Parameters of the cluster and the target density matrix (that of other parameters)."""
    n = case["lx"]
    t, U, bonds = LT.random_bond_cluster(n, n // 2, 17 + n)
    P = GR.HubbardParams(n, bonds)
    rng = np.random.default_rng(3000 + int(seed))
    theta = P.pack(t, U) * (1.0 + 0.1 * rng.standard_normal(P.nparams))
    a = rng.standard_normal((n, n))
    target = np.diag(np.full(n, case["nup"] / n)) + 0.05 * (a + a.T)
    return P, theta, {"up": target, "down": target}


def _z(case):
    return torch.linspace(-10.0, 10.0, OMEGA, dtype=torch.float64, device="cuda") + 1j * ETA


def _greens_keys(case):
    n = case["n"]
    return [("e_up", (n + 1, n)), ("h_up", (n - 1, n)), ("e_down", (n, n + 1)), ("h_down", (n, n - 1))]


def prepare(case, seed):
    k = case["kind"]
    s = {"case": case}
    n = case["lx"] * case.get("ly", 1)
    if k in ("hv", "lanczos", "rdm"):
        t, U = _hubbard(case, seed)
        sec = _capi.Sector(n, case["nup"], case["ndn"], _capi.ED_HUBBARD, t=t, U=U)
        s["sec"] = sec
        if k == "rdm":
            u, d = sec.strings()
            psi = _state(sec.nsup, sec.nsdn, torch.from_numpy(u.astype(np.int64)).cuda(),
                         torch.from_numpy(d.astype(np.int64)).cuda(), seed)
            s["psi"] = sec.from_ref(psi)
        else:
            s["x"] = sec.from_ref(_randn(sec.dim, seed)).to(_dt(case))
    elif k in ("heis_hv", "heis_rdm"):
        sec = _capi.Sector(n, n // 2, 0, _capi.ED_HEISENBERG, J=_heis(case))
        s["sec"] = sec
        s["x" if k == "heis_hv" else "psi"] = sec.from_ref(_randn(sec.dim, seed)).to(_dt(case))
    if k in ("hv", "heis_hv"):
        s["y"] = torch.zeros_like(s["x"])
        if case["dots"]:
            s["dots"] = torch.zeros(2, dtype=torch.float64, device="cuda")
            s["scratch"] = torch.empty(_capi.scratch_bytes(sec.n, 1) // 8 + 1, dtype=torch.float64, device="cuda")
    if k == "solve":
        s["t"], s["U"] = _hubbard(case, seed)
    if k == "gradients":
        s["P"], s["theta"], s["target"] = _gradient_inputs(case, seed)
    if k == "greens":
        secs, shift, sign, srcs = [], [], [], []
        for t, U in _clusters(case, seed):
            src = _capi.Sector(n, case["n"], case["n"], _capi.ED_HUBBARD, t=t, U=np.full(n, U))
            srcs.append(src)
            for kind, (nu, nd) in _greens_keys(case):
                sec = _capi.Sector(n, nu, nd, _capi.ED_HUBBARD, t=t, U=np.full(n, U))
                sg = 1.0 if kind[0] == "e" else -1.0
                secs += [sec] * n
                sign += [sg] * n
                shift += [-sg * 0.5 * n] * n
        bl = GB.BatchedLanczos(secs, case["steps"], dtype=_dt(case), rows="auto")
        i = 0
        for c, src in enumerate(srcs):
            u, d = src.strings()
            psi = src.from_ref(_state(src.nsup, src.nsdn, torch.from_numpy(u.astype(np.int64)).cuda(),
                                      torch.from_numpy(d.astype(np.int64)).cuda(), 100 * seed + c))
            for kind, _ in _greens_keys(case):
                for site in range(1, n + 1):
                    _capi.gf_start(src, secs[i], kind, site, psi, bl.start(i))
                    i += 1
        s.update(bl=bl, z=_z(case), shift=torch.tensor(shift, dtype=torch.float64, device="cuda"),
                 sign=torch.tensor(sign, dtype=torch.float64, device="cuda"))
    return s


# ------------------------------------------------------------------ the calls

def run(s):
    case = s["case"]
    k = case["kind"]
    n = case["lx"] * case.get("ly", 1)
    if k in ("hv", "heis_hv"):
        if case["dots"]:
            s["sec"].hv(s["x"], s["y"], dots=s["dots"], scratch=s["scratch"])
            return {"y": s["y"], "dots": s["dots"].to(s["y"].dtype)}
        s["sec"].hv(s["x"], s["y"])
        return {"y": s["y"]}
    if k == "lanczos":
        r = LZ.lanczos_full(s["sec"], s["x"], case["steps"], _dt(case), ritz_dtype=_dt(case))
        # a state's sign is free: taken along the start vector
        return {"e0": float(r.ritz[0]), "psi": r.psi.mul_(1.0 if r.ritz_vectors[0, 0] > 0 else -1.0)}
    if k == "solve":
        fh = FermiHubbard(n, case["nup"], case["ndn"], s["t"], s["U"])
        fh.kernel()
        return {"e0": float(fh.e0), "one_rdm": fh.one_rdm["up"], "ni": fh.ni, "spin": fh.spin_cor_matrix,
                "amplitude": np.abs(fh.psi0)}
    if k == "rdm":
        gamma, docc, sisj = s["sec"].rdm1(s["psi"])
        return {"gamma": gamma, "docc": docc, "sisj": sisj}
    if k == "heis_rdm":
        return {"sisj": s["sec"].rdm1(s["psi"])[2]}
    if k == "greens":
        bl = s["bl"]
        bl.run()
        g = _capi.cf_eval(bl.alpha, bl.beta, s["z"], shift=s["shift"], sign=s["sign"])
        return {"G": g if case["dtype"] == "f64" else g.to(torch.complex64)}
    sol = GR.solve(s["P"], s["theta"], case["nup"], case["ndn"])
    hf = GR.hf_gradient(s["P"], sol)
    loss, grad, _ = GR.rdm_loss_gradient(s["P"], sol, s["target"])
    return {"e0": float(sol.e0), "gamma": sol.gamma["up"], "hf": hf, "loss": loss, "grad": grad}


# ------------------------------------------------------------------ what a call cannot do without

def _binom(n, k):
    return math.comb(n, k) if 0 <= k <= n else 0


def _hops(case):
    """Average number of hops per element (both spins)."""
    n = case["lx"] * case.get("ly", 1)
    if case.get("lattice", "random") == "random":
        bonds = n + n // 2
    elif case["lattice"] == "ring":
        bonds = n
    else:
        bonds = np.count_nonzero(LT.square(case["lx"], case["ly"], 1.0, periodic=True)) // 2
    return sum(2.0 * bonds * ne * (n - ne) / (n * (n - 1)) for ne in (case["nup"], case["ndn"]))


def work(case):
    k = case["kind"]
    n = case["lx"] * case.get("ly", 1)
    es = 8 if case.get("dtype", "f64") == "f64" else 4
    if k in ("heis_hv", "heis_rdm"):
        D = _binom(n, n // 2)
        if k == "heis_rdm":
            return {"bytes": 8.0 * D, "flops": 2.0 * D * (n * (n - 1) / 4 + n)}
        bonds = np.count_nonzero(_heis(case)) // 2
        return {"bytes": 2.0 * es * D, "flops": 2.0 * D * (bonds * n / (2.0 * (n - 1)) + 1)}
    if k == "greens":
        tot = sum(_binom(n, nu) * _binom(n, nd) * n for _, (nu, nd) in _greens_keys(case)) * case["clusters"]
        bonds = np.count_nonzero(LT.square(case["lx"], case["ly"], -1.0, periodic=False, tp=0.1)) // 2
        inst = 4 * n * case["clusters"]
        # per step: u_k and u_{k-1} read, u_{k+1} written
        return {"bytes": case["steps"] * tot * 3.0 * es + 16.0 * inst * OMEGA,
                "flops": case["steps"] * tot * (2.0 * bonds + 8.0) + 10.0 * inst * OMEGA * case["steps"]}
    D = _binom(n, case["nup"]) * _binom(n, case["ndn"])
    hv_flops = 2.0 * D * (_hops(case) + 1)
    if k == "hv":
        return {"bytes": 2.0 * es * D, "flops": hv_flops}
    if k == "rdm":
        return {"bytes": 8.0 * D, "flops": 2.0 * D * (n * n / 8.0 + n * n / 32.0 + n)}
    m = case.get("steps", 60 if k == "solve" else 120)
    # a full-reorthogonalisation step k reads the k+1 stored vectors, and forms and removes k+1 projections
    bytes_ = es * D * (m * (m + 1) / 2.0 + 3.0 * m)
    flops = m * hv_flops + 4.0 * D * m * (m + 1) / 2.0
    if k == "gradients":
        bytes_ += 120 * 8.0 * D * 4.0    # the adjoint solve: about 120 short-recurrence iterations
        flops += 120 * (hv_flops + 10.0 * D)
    return {"bytes": bytes_, "flops": flops}


# ------------------------------------------------------------------ the same in 64 bits, without the engine

class _Strings:
    """Strings of ne particles on n sites in the engine's order: ascending empty-site pattern, bit j = site j+1."""

    def __init__(self, n, ne):
        self.n, self.ne = n, ne
        h = np.arange(1 << n, dtype=np.int64)
        pop = np.zeros(1 << n, dtype=np.int8)
        for b in range(n):
            pop += ((h >> b) & 1).astype(np.int8)
        self.holes = h[pop == n - ne]
        self.size = len(self.holes)

    def occ(self, j):
        return 1 - ((self.holes >> j) & 1)

    def hop(self, j, k):
        """Strings with site j occupied and k empty, the string with the particle moved to k, and its sign."""
        at = np.nonzero((self.occ(j) == 1) & (self.occ(k) == 0))[0]
        h = self.holes[at]
        to = np.searchsorted(self.holes, h ^ (1 << j) ^ (1 << k))
        lo, hi = min(j, k), max(j, k)
        par = np.zeros(len(at), dtype=np.int64)
        for b in range(lo + 1, hi):
            par += 1 - ((h >> b) & 1)
        return (torch.from_numpy(at).cuda(), torch.from_numpy(to).cuda(),
                torch.from_numpy(1.0 - 2.0 * (par & 1)).cuda())


class _Hub:
    """H of one Hubbard sector on [..., nsdn, nsup] arrays in 64 bits."""

    def __init__(self, n, nup, ndn, t, U):
        self.up, self.dn = _Strings(n, nup), _Strings(n, ndn)
        self.n = n
        self.hu = [(t[k, j],) + self.up.hop(j, k) for j in range(n) for k in range(n) if j != k and t[j, k] != 0.0]
        self.hd = [(t[k, j],) + self.dn.hop(j, k) for j in range(n) for k in range(n) if j != k and t[j, k] != 0.0]
        ou = torch.from_numpy(np.stack([self.up.occ(j) for j in range(n)]).astype(np.float64)).cuda()
        od = torch.from_numpy(np.stack([self.dn.occ(j) for j in range(n)]).astype(np.float64)).cuda()
        e = torch.from_numpy(np.diag(t).copy()).cuda()
        u = torch.from_numpy(np.broadcast_to(np.asarray(U, dtype=np.float64), (n,)).copy()).cuda()
        self.diag = (od.T * u) @ ou + (e @ ou)[None, :] + (e @ od)[:, None]

    @property
    def shape(self):
        return self.dn.size, self.up.size

    def __call__(self, x):
        y = self.diag * x
        for c, at, to, sg in self.hu:
            y.index_add_(-1, to, x.index_select(-1, at) * (c * sg))
        for c, at, to, sg in self.hd:
            y.index_add_(-2, to, x.index_select(-2, at) * (c * sg)[:, None])
        return y


def _heis_bonds(case):
    n = case["lx"] * case["ly"]
    J = _heis(case)
    h = torch.from_numpy(_Strings(n, n // 2).holes).cuda()
    return n, J, h


def _heis_flip(h, a, b):
    """States with antiparallel sites a and b, and where the two swapped land."""
    at = torch.nonzero(((h >> a) ^ (h >> b)) & 1)[:, 0]
    return at, torch.searchsorted(h, h[at] ^ ((1 << a) | (1 << b)))


def _heis_hv(case, x):
    n, J, h = _heis_bonds(case)
    y = torch.zeros_like(x)
    for a in range(n):
        for b in range(a + 1, n):
            if J[a, b] == 0.0:
                continue
            at, to = _heis_flip(h, a, b)
            y += 0.5 * J[a, b] * x
            y[at] += -J[a, b] * x[at] - (-1.0) ** (a + b) * J[a, b] * x[to]
    return y


def _lanczos(H, v0, m, tol=0.0):
    """Lowest pair after m steps with full (twice applied) reorthogonalisation; tol > 0 stops on the residual."""
    V = [v0 / torch.linalg.vector_norm(v0)]
    a, b = [], []
    for k in range(m):
        w = H(V[k])
        a.append(float(torch.sum(w * V[k])))
        Q = torch.stack([v.reshape(-1) for v in V]) if w.numel() < (1 << 23) else None
        for _ in range(2):
            if Q is not None:
                w = w - (Q.T @ (Q @ w.reshape(-1))).view_as(w)
            else:
                for v in V:
                    w = w - torch.sum(v * w) * v
        b.append(float(torch.linalg.vector_norm(w)))
        e, z = np.linalg.eigh(np.diag(a) + np.diag(b[:-1], 1) + np.diag(b[:-1], -1))
        if b[k] < 1e-12 or (tol and abs(b[k] * z[-1, 0]) < tol):
            break
        V.append(w / b[k])
    psi = torch.zeros_like(V[0])
    for j in range(len(a)):
        psi += math.copysign(1.0, z[0, 0]) * float(z[j, 0]) * V[j]
    return float(e[0]), psi / torch.linalg.vector_norm(psi)


def _rdm(H, psi):
    """gamma (spin up, down), double occupancies and S.S of one Hubbard state, as the reference forms them."""
    n, up, dn = H.n, H.up, H.dn
    p2 = psi * psi
    ou = torch.from_numpy(np.stack([up.occ(j) for j in range(n)]).astype(np.float64)).cuda()
    od = torch.from_numpy(np.stack([dn.occ(j) for j in range(n)]).astype(np.float64)).cuda()
    cu, cd = p2.sum(0), p2.sum(1)
    nu, nd = ou @ cu, od @ cd
    ud = od @ p2 @ ou.T                       # <n_down,j n_up,k>
    uu, dd = (ou * cu) @ ou.T, (od * cd) @ od.T
    zz = 0.25 * (uu - ud.T - ud + dd)
    g = torch.zeros(2, n, n, dtype=torch.float64, device="cuda")
    sm = zz.clone()
    for j in range(n):
        g[0, j, j], g[1, j, j] = nu[j], nd[j]
        sm[j, j] += 0.5 * (nu[j] + nd[j]) - ud[j, j]
        for k in range(j):
            at, to, sg = up.hop(j, k)
            g[0, j, k] = g[0, k, j] = torch.sum(psi[:, at] * psi[:, to] * sg)
            dat, dto, dsg = dn.hop(j, k)
            g[1, j, k] = g[1, k, j] = torch.sum(psi[dat] * psi[dto] * dsg[:, None])
            rat, rto, rsg = dn.hop(k, j)
            s = torch.sum(psi[rat][:, at] * psi[rto][:, to] * sg * rsg[:, None])
            sm[j, k] -= s
            sm[k, j] = sm[j, k]
    return g, torch.diagonal(ud).clone(), sm


def _exact_solve(case, seed):
    n = case["lx"] * case["ly"]
    t, U = _hubbard(case, seed)
    H = _Hub(n, case["nup"], case["ndn"], t, U)
    D = H.shape[0] * H.shape[1]
    v0 = (torch.rand(D, generator=_gen(0), dtype=torch.float64, device="cuda") - 0.5).view(H.shape)
    e, psi = _lanczos(H, v0, min(400, D), tol=1e-12)
    g, docc, sm = _rdm(H, psi)
    return {"e0": e, "one_rdm": g[0], "ni": docc, "spin": sm, "amplitude": psi.abs().reshape(-1)}


def _exact_gradients(case, seed):
    n = case["lx"]
    P, theta, target = _gradient_inputs(case, seed)
    t, U = P.unpack(theta)
    H = _Hub(n, case["nup"], case["ndn"], t, U)
    D = H.shape[0] * H.shape[1]
    v0 = (torch.rand(D, generator=_gen(0), dtype=torch.float64, device="cuda") - 0.5).view(H.shape)
    e, psi = _lanczos(H, v0, min(400, D), tol=1e-12)
    dH = []
    for i, j in P.bonds:
        b = np.zeros((n, n))
        b[i, j] = b[j, i] = 1.0
        dH.append(_Hub(n, case["nup"], case["ndn"], b, 0.0))
    for i in range(n):
        dH.append(_Hub(n, case["nup"], case["ndn"], np.zeros((n, n)), np.eye(n)[i]))
    for i in range(n):
        dH.append(_Hub(n, case["nup"], case["ndn"], np.diag(np.eye(n)[i]), 0.0))
    hf = torch.stack([torch.sum(psi * A(psi)) for A in dH])
    g, _, _ = _rdm(H, psi)
    w = [2.0 * (g[k].cpu().numpy() - target["up"]) for k in (0, 1)]
    loss = float(sum(np.sum((x / 2.0) ** 2) for x in w))
    A = _Hub(n, case["nup"], case["ndn"], 0.25 * sum(x + x.T for x in w), 0.0)
    rhs = -2.0 * A(psi)
    rhs = rhs - torch.sum(psi * rhs) * psi
    x, r = torch.zeros_like(rhs), rhs.clone()
    p, rr = r.clone(), torch.sum(r * r)
    for _ in range(4000):   # conjugate gradients: H - E0 is positive on the complement of psi
        q = H(p) - e * p
        q = q - torch.sum(psi * q) * psi
        al = rr / torch.sum(p * q)
        x = x + al * p
        r = r - al * q
        new = torch.sum(r * r)
        if float(new) < 1e-28 * float(torch.sum(rhs * rhs)):
            break
        p, rr = r + (new / rr) * p, new
    grad = torch.stack([torch.sum(x * B(psi)) for B in dH])
    return {"e0": e, "gamma": g[0], "hf": hf, "loss": loss, "grad": grad}


def _exact_greens(case, seed):
    n, m = case["lx"] * case["ly"], case["steps"]
    z = _z(case)
    out = []
    for c, (t, U) in enumerate(_clusters(case, seed)):
        up, dn = _Strings(n, case["n"]), _Strings(n, case["n"])
        us = torch.from_numpy(_string_bits(up)).cuda()
        ds = torch.from_numpy(_string_bits(dn)).cuda()
        psi = _state(up.size, dn.size, us, ds, 100 * seed + c).view(dn.size, up.size)
        for kind, (nu, nd) in _greens_keys(case):
            H = _Hub(n, nu, nd, t, U)
            X = torch.zeros((n,) + H.shape, dtype=torch.float64, device="cuda")
            spin_up = kind.endswith("up")
            src, dst = (up, H.up) if spin_up else (dn, H.dn)
            for j in range(n):
                want = 0 if kind[0] == "e" else 1
                at = np.nonzero(src.occ(j) == want)[0]
                h = src.holes[at]
                to = torch.from_numpy(np.searchsorted(dst.holes, h ^ (1 << j))).cuda()
                par = np.zeros(len(at), dtype=np.int64)
                for b in range(j):
                    par += 1 - ((h >> b) & 1)
                sg = torch.from_numpy(1.0 - 2.0 * (par & 1)).cuda()
                at = torch.from_numpy(at).cuda()
                if spin_up:   # the overall sign of a start vector does not enter G_jj
                    X[j][:, to] = psi[:, at] * sg
                else:
                    X[j][to] = psi[at] * sg[:, None]
            nrm = torch.sqrt(torch.sum(X * X, dim=(1, 2)))
            a, b = [], [nrm]
            prev, cur = torch.zeros_like(X), X / nrm[:, None, None]
            for _ in range(m):
                w = H(cur)
                al = torch.sum(w * cur, dim=(1, 2))
                w = w - al[:, None, None] * cur - (b[-1] if len(b) > 1 else torch.zeros_like(al))[:, None, None] * prev
                be = torch.sqrt(torch.sum(w * w, dim=(1, 2)))
                a.append(al)
                b.append(be)
                prev, cur = cur, w / be[:, None, None]
            s = 1.0 if kind[0] == "e" else -1.0
            zz = (z - s * 0.5 * n)[None, :]
            f = torch.zeros((n, len(z)), dtype=torch.complex128, device="cuda")
            for k in range(m - 1, -1, -1):
                f = (b[k] ** 2)[:, None] / (zz - s * a[k][:, None] - f)
            out.append(f)
    return {"G": torch.cat(out)}


def _string_bits(st):
    """Occupation words of the strings (site 1 in the highest of n bits)."""
    w = np.zeros(st.size, dtype=np.int64)
    for j in range(st.n):
        w |= st.occ(j).astype(np.int64) << (st.n - 1 - j)
    return w


def exact(case, seed):
    k = case["kind"]
    n = case["lx"] * case.get("ly", 1)
    if k in ("hv", "lanczos", "rdm"):
        t, U = _hubbard(case, seed)
        H = _Hub(n, case["nup"], case["ndn"], t, U)
        nsdn, nsup = H.shape
        if k == "rdm":
            psi = _state(nsup, nsdn, torch.from_numpy(_string_bits(H.up)).cuda(),
                         torch.from_numpy(_string_bits(H.dn)).cuda(), seed).view(nsdn, nsup)
            g, docc, sm = _rdm(H, psi)
            if case["nup"] == case["ndn"]:
                g[1] = g[0]      # the reference copies the up matrix
            return {"gamma": g, "docc": docc, "sisj": sm}
        x = _randn(nsdn * nsup, seed).to(_dt(case)).double().view(nsdn, nsup)
        if k == "lanczos":
            e, psi = _lanczos(H, x, case["steps"])
            out = {"e0": e}
            y = psi
        else:
            out = {}
            y = H(x)
        ld = (nsup + 31) // 32 * 32
        pad = torch.zeros((nsdn, ld), dtype=torch.float64, device="cuda")
        pad[:, :nsup] = y
        out["psi" if k == "lanczos" else "y"] = pad.view(-1)
        if case.get("dots"):
            out["dots"] = torch.stack([torch.sum(x * y), torch.sum(y * y)])
        return out
    if k == "heis_hv":
        D = _binom(n, n // 2)
        x = _randn(D, seed).to(_dt(case)).double()
        y = _heis_hv(case, x)
        pad = torch.zeros((D + 31) // 32 * 32, dtype=torch.float64, device="cuda")
        pad[:D] = y
        out = {"y": pad}
        if case["dots"]:
            out["dots"] = torch.stack([torch.sum(x * y), torch.sum(y * y)])
        return out
    if k == "heis_rdm":
        n, _, h = _heis_bonds(case)
        psi = _randn(h.numel(), seed)
        p2 = psi * psi
        sm = torch.zeros(n, n, dtype=torch.float64, device="cuda")
        for a in range(n):
            sm[a, a] = 0.75 * p2.sum()
            for b in range(a + 1, n):
                at, to = _heis_flip(h, a, b)
                anti = p2[at].sum()
                flip = 0.5 * torch.sum(psi[at] * psi[to])
                sm[a, b] = sm[b, a] = 0.25 * (p2.sum() - 2.0 * anti) + (-1.0) ** (a + b) * flip
        return {"sisj": sm}
    if k == "solve":
        return _exact_solve(case, seed)
    if k == "gradients":
        return _exact_gradients(case, seed)
    return _exact_greens(case, seed)
