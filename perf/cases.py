"""The work that a program has this framework do, as cases that can be timed.

Every case is one pass through the public entry points of `helfem_gb300`: a
Fock build (J and K) of an atomic or a diatomic basis in its plain FP64 or its
split-precision form, an exchange-correlation build on the DFT grid, or a
whole atomic SCF solve. Bases, grids and densities follow the benchmark's and
the tests' configurations (Ne, Kr and N2 among them) and the seeded workloads
of `helfem_gb300.workloads`.

`exact` states the same results in 64 bits from the integrals' definitions
(torch; no table or code of the package): Lagrange polynomials on Gauss-Lobatto
nodes, Gauss-Legendre quadrature, the Laplace and Neumann expansions of 1/r12,
and autograd derivatives of the functionals.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import helfem_gb300 as hg
from helfem_gb300 import workloads as wl

F64 = torch.float64
LDA, PW, PBE = "lda_x-lda_c_vwn", "lda_x-lda_c_pw", "gga_x_pbe-gga_c_pbe"


# ---------------------------------------------------------------------------
# The cases
# ---------------------------------------------------------------------------


def _atom(kind, Z, nelem, lmax, mmax, nnodes=15, rmax=40.0, zexp=2.0, **kw):
    return dict(kind=kind, Z=Z, nelem=nelem, lmax=lmax, mmax=mmax, nnodes=nnodes, rmax=rmax, zexp=zexp, **kw)


def _dia(kind, Z1, Z2, R, nelem, lm, **kw):
    lm = list(lm) + [-1] * (4 - len(lm))
    return dict(kind=kind, Z1=Z1, Z2=Z2, R=R, nelem=nelem, lm0=lm[0], lm1=lm[1], lm2=lm[2], lm3=lm[3], **kw)


def listed():
    return [
        # the smallest Fock build: a helium-sized basis with the entry point's default flags (latency)
        dict(_atom("fock", 2, 5, 0, 0, split=False, symmetric=False, density="bound"), name="he_fock"),
        # the first benchmark configuration: Ne, 10 elements, l <= 1 with m = 0, plain FP64
        dict(_atom("fock", 10, 10, 1, 0, zexp=1.0, split=False, symmetric=True, density="bound"), name="ne_fock"),
        # the Kr configuration (40 elements, l <= 2, dense density) in the plain drop-in form ...
        dict(_atom("fock", 36, 40, 2, 2, rmax=60.0, zexp=1.0, split=False, symmetric=True, density="dense"),
             name="kr_fock"),
        # ... and in split precision, the framework's headline number
        dict(_atom("fock", 36, 40, 2, 2, rmax=60.0, zexp=1.0, split=True, symmetric=True, density="dense"),
             name="kr_fock_split"),
        # the same through the host-matrix entry point, as a caller of the reference's C++ API has it
        dict(_atom("fock_host", 36, 40, 2, 2, rmax=60.0, zexp=1.0, split=True, symmetric=True, density="dense"),
             name="kr_fock_host_split"),
        # a heavy atom of the batch workload: l <= 3, 13-node elements, an odd element count, m-block density
        dict(_atom("fock", 86, 33, 3, 3, nnodes=13, rmax=57.0, split=True, symmetric=True, density="bound"),
             name="rn_fock_split"),
        # DFT: the exchange-correlation part of a light atom's LDA iteration, restricted, small elements
        dict(_atom("xc", 18, 17, 1, 1, nnodes=10, func=PW, restricted=True), name="ar_xc_lda"),
        # and of a heavy one's PBE iteration, unrestricted
        dict(_atom("xc", 36, 40, 2, 2, rmax=60.0, zexp=1.0, func=PBE, restricted=False), name="kr_xc_pbe"),
        # diatomics: the tests' H2 basis, default flags (latency)
        dict(_dia("dfock", 1, 1, 1.4, 3, [4], split=False, symmetric=False), name="h2_fock"),
        # N2 with the benchmark's geometry and angular pattern, split precision
        dict(_dia("dfock", 7, 7, 2.074, 12, [10, 10, 8, 6], split=True, symmetric=True), name="n2_fock_split"),
        # a heteronuclear molecule's PBE iteration on the pure-m grid
        dict(_dia("dxc", 7, 8, 2.17, 14, [9, 8, 6], func=PBE, restricted=True), name="no_xc_pbe"),
        # a whole request of the serving workload: one atomic HF solve to convergence
        dict(_atom("scf", 18, 20, 1, 1, method="hf", split=True), name="ar_scf"),
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["fock", "fock", "fock", "fock_host", "xc", "xc", "dfock", "dfock", "dxc", "scf"])
    if kind in ("fock", "fock_host", "xc"):
        lmax = rng.choice([0, 1, 1, 2, 2, 3])
        mmax = lmax if rng.random() < 0.8 else 0
        nn = rng.choice([10, 13, 15, 15, 15, 17])
        top = {0: 80, 1: 60, 2: 40, 3: 28}[lmax]
        c = _atom(kind, rng.choice([[2, 4], [6, 10, 14], [26, 36, 47], [60, 80, 86]][lmax]),
                  _log_int(rng, 5, top), lmax, mmax, nnodes=nn, rmax=round(rng.uniform(40.0, 80.0), 2),
                  zexp=rng.choice([1.0, 2.0, 2.0]))
        if kind == "xc":
            c.update(func=rng.choice([LDA, PW, PBE, PBE]), restricted=rng.random() < 0.5)
        else:
            c.update(split=kind == "fock_host" or rng.random() < 0.6, symmetric=rng.random() < 0.75,
                     density=rng.choice(["bound", "bound", "dense"]))
        return c
    if kind in ("dfock", "dxc"):
        Z1, Z2, R = rng.choice([(1, 1, 1.4), (7, 7, 2.074), (7, 8, 2.17), (6, 8, 2.13), (10, 0, 1.0)])
        l0 = rng.randint(3, 10)
        lm = [l0]
        for _ in range(rng.randint(0, 3)):
            if lm[-1] - len(lm) >= 2:
                lm.append(max(len(lm), lm[-1] - rng.randint(0, 2)))
        c = _dia(kind, Z1, Z2, R, _log_int(rng, 3, 12 if len(lm) > 2 else 20), lm)
        if kind == "dxc":
            c.update(func=rng.choice([LDA, PW, PBE, PBE]), restricted=rng.random() < 0.5)
        else:
            split = rng.random() < 0.7
            if not split:  # the plain form is some 3 times the work
                c["nelem"] = min(c["nelem"], 9)
            c.update(split=split, symmetric=rng.random() < 0.75)
        return c
    Z = rng.randint(2, 20)
    lmax = wl.occupied_lmax(Z)
    return _atom("scf", Z, _log_int(rng, 10, 24), lmax, lmax, nnodes=rng.choice([10, 13, 15]),
                 method=rng.choice(["hf", "hf", LDA]), split=rng.random() < 0.5)


# ---------------------------------------------------------------------------
# Bases and densities
# ---------------------------------------------------------------------------


def _angular(c):
    lv, mv = hg.angular_basis(c["lmax"], c["mmax"])
    return [int(l) for l in lv], [int(m) for m in mv]


def _lm(c):
    return [c[k] for k in ("lm0", "lm1", "lm2", "lm3") if c[k] >= 0]


def _rng(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _orthonormal(C, S):
    """Loewdin-orthonormal columns in the metric S."""
    w, v = torch.linalg.eigh(C.T @ (S @ C))
    return C @ (v / w.sqrt()) @ v.T


def _atom_density(c, seed):
    """P = C C^T (18 or fewer columns): `dense`, seeded normal columns over the whole basis, Loewdin-orthonormal in
    the overlap; `bound`, Slater-type shells per (l, m), the same for every m, with seeded exponents."""
    lv, mv = _angular(c)
    nn, bval = c["nnodes"], hg.get_grid(c["rmax"], c["nelem"], 4, c["zexp"])
    el = _Elements(nn, bval, drop_first=True)
    S = el.assemble(el.weighted(lambda r: torch.ones_like(r), 64))
    nr, na = S.shape[0], len(lv)
    g = _rng(seed)
    if c.get("density", "bound") == "dense":
        C = torch.randn((na, nr, 18), generator=g, device="cuda", dtype=F64)
        SC = torch.einsum("rs,asc->arc", S, C).reshape(na * nr, 18)
        C = C.reshape(na * nr, 18)
        w, v = torch.linalg.eigh(C.T @ SC)
        C = C @ (v / w.sqrt()) @ v.T
        return C, torch.ones(18, device="cuda", dtype=F64)
    r = el.node_values()
    cols, occ = [], []
    for l in range(c["lmax"] + 1):
        nsh = max(1, min(5 - l, (4 if c["Z"] > 54 else 3 if c["Z"] > 18 else 2 if c["Z"] > 4 else 1) - l // 2))
        zeta = c["Z"] ** (1.0 - 0.35 * torch.arange(nsh, device="cuda", dtype=F64)) / (l + 1)
        zeta = zeta * (0.8 + 0.4 * torch.rand(nsh, generator=g, device="cuda", dtype=F64))
        u = torch.stack([r ** (l + 1 + n) * torch.exp(-zeta[n] * r) for n in range(nsh)], 1)
        u = _orthonormal(u / u.abs().max(0).values, S)
        f = 0.6 + 0.4 * torch.rand(nsh, generator=g, device="cuda", dtype=F64)
        for a in range(na):
            if lv[a] == l:
                for n in range(nsh):
                    col = torch.zeros((na, nr), device="cuda", dtype=F64)
                    col[a] = u[:, n]
                    cols.append(col.reshape(-1))
                    occ.append(f[n])
    return torch.stack(cols, 1), torch.stack(occ)


def _diatomic_density(c, d, seed):
    """Orbitals of sigma, pi and delta type (whichever the basis has), seeded, decaying in mu and in l, orthonormal in
    the overlap; P does not mix m, as in every solve with linear symmetry."""
    g = _rng(seed)
    idx = torch.as_tensor(d.pure_indices().astype(np.int64)).cuda()
    mv = torch.as_tensor(np.asarray(d.mval)).cuda()
    lv = torch.as_tensor(np.asarray(d.lval)).cuda()
    el = _Elements(15, np.asarray(d._bval), drop_first=False)
    mu = el.node_values()
    cols, occ = [], []
    for m in sorted(set(int(x) for x in d.mval)):
        n = {0: 5 if d.Z1 + d.Z2 > 4 else 1, 1: 1, 2: 1}.get(abs(m), 0)
        sel = torch.nonzero(mv[idx // d.nrad] == m)[:, 0]
        if n == 0:
            continue
        S = torch.as_tensor(d.one_electron_block("S", m)).cuda()
        l = lv[idx[sel] // d.nrad].to(F64)
        x = mu[idx[sel] % d.nrad]
        zeta = d.Rhalf * (0.7 + 2.0 * torch.rand(n, generator=g, device="cuda", dtype=F64))
        a = torch.randn((int(lv.max()) + 1, n), generator=g, device="cuda", dtype=F64)
        a = a * 0.6 ** torch.arange(a.shape[0], device="cuda", dtype=F64)[:, None]
        C = a[l.long()] * torch.exp(-zeta * (torch.cosh(x) - 1)[:, None]) * (torch.sinh(x) ** abs(m))[:, None]
        C = _orthonormal(C / C.abs().max(0).values, S)
        full = torch.zeros((d.nbf, n), device="cuda", dtype=F64)
        full[sel] = C
        cols.append(full)
        occ.append(0.6 + 0.4 * torch.rand(n, generator=g, device="cuda", dtype=F64))
    return torch.cat(cols, 1), torch.cat(occ)


def _closed(C, f):
    return (C * f) @ C.T


def _make_atom(c):
    lv, mv = hg.angular_basis(c["lmax"], c["mmax"])
    return hg.Atom(c["Z"], hg.get_grid(c["rmax"], c["nelem"], 4, c["zexp"]), lv, mv, nnodes=c["nnodes"])


def _make_diatomic(c):
    return hg.Diatomic.from_grid(c["Z1"], c["Z2"], c["R"], c["nelem"], _lm(c))


def _spins(c, C, f):
    """The densities of an XC call: the total one, or two spin densities."""
    if c["restricted"]:
        return _closed(C, 2.0 * f), None
    return _closed(C, torch.ones_like(f)), _closed(C, f)


def prepare(case, seed):
    c = case
    s = {"case": c}
    if c["kind"] == "scf":
        g = np.random.default_rng(int(seed))
        lv, mv = hg.angular_basis(c["lmax"], c["mmax"])
        bval = hg.get_grid(float(g.uniform(40.0, 80.0)), c["nelem"], 4, c["zexp"])
        s["h"] = hg.Atom(c["Z"], bval, lv, mv, nnodes=c["nnodes"])
        s["nel"] = ((c["Z"] + 1) // 2, c["Z"] // 2)
        s["l_occ"] = wl.l_occupations(*s["nel"], c["lmax"])
        return s
    if c["kind"] in ("dfock", "dxc"):
        s["h"] = h = _make_diatomic(c)
        C, f = _diatomic_density(c, h, seed)
    else:
        s["h"] = h = _make_atom(c)
        C, f = _atom_density(c, seed)
    if c["kind"] in ("xc", "dxc"):
        s["Pa"], s["Pb"] = _spins(c, C, f)
        s["Ha"] = torch.empty_like(s["Pa"])
        s["Hb"] = None if s["Pb"] is None else torch.empty_like(s["Pb"])
        s["E"] = torch.empty(2, device="cuda", dtype=F64)
        s["func"] = hg.parse_xc(c["func"])
        h.dft_grid()
        return s
    P = _closed(C, f)
    if c["kind"] == "fock_host":
        for k in "PJK":
            t = torch.empty(P.shape, dtype=F64, pin_memory=True)
            if k == "P":
                t.copy_(P)
            s[k] = t.numpy().T
        torch.cuda.synchronize()
    else:
        s["P"], s["J"], s["K"] = P, torch.empty_like(P), torch.empty_like(P)
    return s


def run(state):
    s = state
    c, h = s["case"], s["h"]
    if c["kind"] == "fock":
        h.jk(s["P"], s["J"], s["K"], symmetric=c["symmetric"], split=c["split"], split_j=c["split"])
        return {"J": s["J"], "K": s["K"]}
    if c["kind"] == "fock_host":
        h.jk_host(s["P"], J=s["J"], K=s["K"], symmetric=c["symmetric"], split=c["split"], split_j=c["split"])
        return {"J": s["J"], "K": s["K"]}
    if c["kind"] == "dfock":
        h.coulomb(s["P"], s["J"])
        h.exchange(s["P"], s["K"], symmetric=c["symmetric"], split=c["split"])
        return {"J": s["J"], "K": s["K"]}
    if c["kind"] == "scf":
        r = h.scf(*s["nel"], method=c["method"], symmetry=2, l_occ=s["l_occ"], split=c["split"])
        return {"Etot": r["Etot"], "eps": r["orbital_energies"]}
    h.xc(*s["func"], s["Pa"], s["Ha"], s["Pb"], s["Hb"], energies=s["E"])
    return {"E": s["E"], "Ha": s["Ha"], "Hb": s["Hb"]}


# ---------------------------------------------------------------------------
# What a pass cannot do without
# ---------------------------------------------------------------------------


def work(case):
    """Bytes: every input read once and every output written once. Operations: the multiplications and additions of the
    element-tile products and quadrature sums, one per distinct result (half of them where the result is symmetric)."""
    c = case
    nn, nel = c.get("nnodes", 15), c["nelem"]
    if c["kind"] in ("dfock", "dxc"):
        lm = _lm(c)
        lv, mv = hg.lm_to_l_m(lm)
        nang, nrad = len(lv), nel * (nn - 1)
        nbf = sum(nrad - (m != 0) for m in mv)
        if c["kind"] == "dxc":
            ns = 1 if c["restricted"] else 2
            npair = sum(1 for i in range(nang) for j in range(i + 1) if mv[i] == mv[j])
            na, nq, nc = 4 * int(max(lv)) + 12, 5 * nn, 3 if c["func"] == PBE else 1
            fl = ns * nel * (4.0 * npair * nq * nn * nn + 4.0 * nc * npair * nq * na)
            return {"bytes": 16.0 * ns * nbf * nbf, "flops": fl}
        ent = 0
        for j in range(nang):
            for k in range(nang):
                if mv[j] == mv[k]:
                    ms = {abs(int(mv[j]) - int(m)) for m in mv}
                    ent += sum(max(0, min(int(lv[j]), int(lv[k])) + int(max(lv)) + 2 - m) // 2 + 1 for m in ms)
        pairs = nel * (nel - 1) / 2
        return {"bytes": 24.0 * nbf * nbf, "flops": ent * (12.0 * nn ** 3 * pairs + 4.0 * nn ** 4 * nel)}
    lv, mv = _angular(c)
    na, nrad = len(lv), nel * (nn - 1) - 1
    nbf = na * nrad
    if c["kind"] == "xc":
        ns = 1 if c["restricted"] else 2
        npair = na * (na + 1) / 2
        ang, nq, nc = (4 * c["lmax"] + 12) * (4 * c["mmax"] + 12), 5 * nn, 4 if c["func"] == PBE else 1
        fl = ns * nel * (4.0 * npair * nq * nn * nn + 4.0 * nc * npair * nq * ang)
        return {"bytes": 16.0 * ns * nbf * nbf, "flops": fl}
    ent = 0
    for j in range(na):
        for k in range(na):
            for L in range(2 * c["lmax"] + 1):
                ent += any((lv[j] + lv[i] + L) % 2 == 0 and abs(lv[j] - lv[i]) <= L <= lv[j] + lv[i]
                           and (lv[k] + lv[q] + L) % 2 == 0 and abs(lv[k] - lv[q]) <= L <= lv[k] + lv[q]
                           and mv[j] - mv[i] == mv[k] - mv[q] and abs(mv[j] - mv[i]) <= L
                           for i in range(na) for q in range(na))
    fl = ent * (4.0 * nn ** 3 * nel * (nel - 1) / 2 + nn ** 4 * nel)
    if c["kind"] == "scf":  # some twelve iterations, each a Fock build and the spectra of its blocks
        return {"bytes": 12 * 24.0 * nbf * nbf, "flops": 12 * (fl + 4.0 * (c["lmax"] + 1) * nrad ** 3)}
    return {"bytes": 24.0 * nbf * nbf, "flops": fl}


# ---------------------------------------------------------------------------
# The same in 64 bits, from the definitions
# ---------------------------------------------------------------------------


def _gl(n):
    x, w = np.polynomial.legendre.leggauss(n)
    return torch.as_tensor(x).cuda(), torch.as_tensor(w).cuda()


def _lobatto(n):
    P = np.polynomial.legendre.Legendre.basis(n - 1)
    x = np.sort(P.deriv().roots().real)
    for _ in range(3):
        x = x - P.deriv()(x) / P.deriv(2)(x)
    return np.concatenate([[-1.0], x, [1.0]])


def _lagrange(x, nodes, der=0):
    """Values (or first derivatives) of the Lagrange polynomials, shape x.shape + (n,)."""
    n = len(nodes)
    d = x[..., None] - nodes
    eye = torch.eye(n, device="cuda", dtype=torch.bool)
    q = torch.where(eye, torch.ones_like(nodes), nodes[:, None] - nodes[None, :])
    f = d[..., None, :] / q  # (..., i, p): (x - x_p) / (x_i - x_p)
    f = torch.where(eye, torch.ones_like(f), f)
    if der == 0:
        return f.prod(-1)
    out = 0
    for k in range(n):
        h = f.clone()
        h[..., :, k] = 1.0
        t = h.prod(-1) / q[:, k]
        t[..., k] = 0.0
        out = out + t
    return out


class _Elements:
    """Lagrange elements on [b_e, b_e+1]; neighbours share a function. Element tiles carry all nn functions, `mask`
    marks those of the basis and `g` numbers them."""

    def __init__(self, nn, bval, drop_first):
        self.nn, self.nel = nn, len(bval) - 1
        b = torch.as_tensor(np.asarray(bval, dtype=np.float64)).cuda()
        self.b0, self.h, self.mid = b[:-1], 0.5 * (b[1:] - b[:-1]), 0.5 * (b[1:] + b[:-1])
        self.nodes = torch.as_tensor(_lobatto(nn)).cuda()
        g = torch.arange(self.nel, device="cuda")[:, None] * (nn - 1) + torch.arange(nn, device="cuda")[None, :]
        self.g = g - 1 if drop_first else g
        self.n = self.nel * (nn - 1) - (1 if drop_first else 0)
        self.mask = ((self.g >= 0) & (self.g < self.n)).to(F64)
        self.gc = self.g.clamp(0, self.n - 1)

    def node_values(self):
        r = self.mid[:, None] + self.h[:, None] * self.nodes[None, :]
        out = torch.zeros(self.n, device="cuda", dtype=F64)
        ok = self.mask > 0
        out[self.g[ok]] = r[ok]
        return out

    def B(self, x, der=0):
        return _lagrange(x, self.nodes, der)

    def weighted(self, f, nq):
        """int B_i B_j f(r) dr per element, masked: (nel, nn, nn)."""
        x, w = _gl(nq)
        r = self.mid[:, None] + self.h[:, None] * x
        B = self.B(x)
        t = torch.einsum("eq,qi,qj->eij", f(r) * w * self.h[:, None], B, B)
        return t * self.mask[:, :, None] * self.mask[:, None, :]

    def assemble(self, T):
        M = torch.zeros((self.n, self.n), device="cuda", dtype=F64)
        for e in range(self.nel):
            M.index_put_((self.gc[e][:, None], self.gc[e][None, :]),
                         T[e] * self.mask[e][:, None] * self.mask[e][None, :], accumulate=True)
        return M

    def tiles(self, P):
        """(..., n, n) -> (..., nel*nn, nel*nn), a function that two elements share in both."""
        gi, m = self.gc.reshape(-1), self.mask.reshape(-1)
        return P[..., gi[:, None], gi[None, :]] * m[:, None] * m[None, :]

    def untile(self, T):
        """The transposed map: shared functions receive the sum of their elements' entries."""
        gi, m = self.gc.reshape(-1), self.mask.reshape(-1)
        out = torch.zeros(T.shape[:-2] + (self.n, T.shape[-1]), device="cuda", dtype=F64)
        out.index_add_(-2, gi, T * m[:, None])
        res = torch.zeros(T.shape[:-2] + (self.n, self.n), device="cuda", dtype=F64)
        return res.index_add_(-1, gi, out * m[None, :])


def _theta(l, m, x):
    """Y_l^m(theta, phi) = theta_l^m(cos theta) exp(i m phi), Condon-Shortley phase."""
    a = abs(m)
    if a > l:
        return torch.zeros_like(x)
    s = ((1 - x) * (1 + x)).clamp(min=0).sqrt()
    p = torch.full_like(x, 1.0 / math.sqrt(4 * math.pi))
    for k in range(1, a + 1):
        p = -p * s * math.sqrt((2 * k + 1) / (2 * k))
    q = torch.zeros_like(x)
    for k in range(a + 1, l + 1):
        al = math.sqrt((4 * k * k - 1) / (k * k - a * a))
        be = math.sqrt(((k - 1) ** 2 - a * a) / (4 * (k - 1) ** 2 - 1)) if k > a + 1 else 0.0
        p, q = al * (x * p - be * q), p
    return p if m >= 0 or a % 2 == 0 else -p


def _coupling(lv, mv, L, M, cos2=False):
    """G[j, i] = int Y_j^* (cos^2) Y_L^M Y_i."""
    x, w = _gl(96)
    Y = torch.stack([_theta(l, m, x) for l, m in zip(lv, mv)])
    f = _theta(L, M, x) * w * 2 * math.pi * (x * x if cos2 else 1.0)
    G = torch.einsum("jx,ix,x->ji", Y, Y, f)
    m = torch.as_tensor(mv).cuda()
    G = torch.where(m[:, None] - m[None, :] == M, G, torch.zeros_like(G))
    return torch.where(G.abs() > 1e-13, G, torch.zeros_like(G))


def _side(el, left, X, right, upper):
    """left(a) X(a, b) right(b)^T over the element pairs a < b (or a > b)."""
    n, nn = el.nel, el.nn
    T = X.reshape(X.shape[:-2] + (n, nn, n, nn))
    T = torch.einsum("aip,...apbq->...aibq", left, T)
    T = torch.einsum("bjq,...aibq->...aibj", right, T)
    m = torch.triu(torch.ones(n, n, device="cuda", dtype=F64), 1)
    m = m if upper else m.T
    return (T * m[:, None, :, None]).reshape(X.shape)


def _diag(el, X):
    """The (e, e) tiles: (..., nel, nn, nn)."""
    n, nn = el.nel, el.nn
    T = X.reshape(X.shape[:-2] + (n, nn, n, nn))
    return torch.diagonal(T, dim1=-4, dim2=-2).movedim(-1, -3)


def _put_diag(el, Y):
    n, nn = el.nel, el.nn
    T = torch.zeros(Y.shape[:-3] + (n, nn, n, nn), device="cuda", dtype=F64)
    for e in range(n):
        T[..., e, :, e, :] = Y[..., e, :, :]
    return T.reshape(Y.shape[:-3] + (n * nn, n * nn))


def _inner(el, wfun, n_out, n_in, cubic):
    """Quadrature of an in-element kernel f(r1) g(r2), r2 < r1: outer points and weights, B there, inner points and
    weights, B there. `cubic` smooths an endpoint singularity at the first element's origin."""
    xo, wo = _gl(n_out)
    xi, wi = _gl(n_in)
    t = 0.5 * (xo + 1)
    s = t[None, :].expand(el.nel, -1).clone()
    ds = (0.5 * wo)[None, :].expand(el.nel, -1).clone()
    if cubic:
        s[0], ds[0] = t ** 3, 0.5 * wo * 3 * t * t
    r1 = el.b0[:, None] + 2 * el.h[:, None] * s
    w1 = 2 * el.h[:, None] * ds
    half = 0.5 * (r1 - el.b0[:, None])
    r2 = el.b0[:, None, None] + half[..., None] * (xi + 1)
    w2 = half[..., None] * wi
    B1 = el.B((r1 - el.mid[:, None]) / el.h[:, None]) * el.mask[:, None, :]
    B2 = el.B((r2 - el.mid[:, None, None]) / el.h[:, None, None]) * el.mask[:, None, None, :]
    return r1, w1, B1, r2, w2, B2


def _atom_jk(c, seed):
    lv, mv = _angular(c)
    na = len(lv)
    el = _Elements(c["nnodes"], hg.get_grid(c["rmax"], c["nelem"], 4, c["zexp"]), True)
    C, f = _atom_density(c, seed)
    nr = el.n
    P = el.tiles(_closed(C, f).reshape(na, nr, na, nr).permute(0, 2, 1, 3))  # (i, l, tiles, tiles)
    r1, w1, B1, r2, w2, B2 = _inner(el, None, 128, 48, False)
    J = torch.zeros_like(_diag(el, P))
    K = torch.zeros((na, na, nr, nr), device="cuda", dtype=F64)
    Pd = _diag(el, P)
    for L in range(2 * c["lmax"] + 1):
        G = {M: _coupling(lv, mv, L, M) for M in range(-L, L + 1)}
        G = {M: g for M, g in G.items() if bool((g != 0).any())}
        fac = 4 * math.pi / (2 * L + 1)
        rs = el.weighted(lambda r: r ** L, 128)
        rb = el.weighted(lambda r: r ** (-L - 1.0), 128)
        rb[0] = 0.0
        Gin = torch.einsum("epq,epqk,epql->epkl", w2 * r2 ** L, B2, B2)
        T = torch.einsum("ep,epi,epj,epkl->eijkl", w1 * r1 ** (-L - 1.0), B1, B1, Gin)
        T = T + T.permute(0, 3, 4, 1, 2)
        for M, g in G.items():
            X = torch.einsum("kl,kleij->eij", g, Pd)
            big = torch.einsum("eij,eji->e", rb, X)
            small = torch.einsum("eij,eji->e", rs, X)
            above = big.flip(0).cumsum(0).flip(0) - big
            below = small.cumsum(0) - small
            V = torch.einsum("eijkl,ekl->eij", T, X) + rs * above[:, None, None] + rb * below[:, None, None]
            J += fac * torch.einsum("ji,epq->ijepq", g, V)
        for j in range(na):  # X[k] = sum over M, i, l of G[j, i] G[k, l] P[i, l]
            X = torch.zeros_like(P[0])
            hit = False
            for M, g in G.items():
                on = torch.nonzero(g[j])[:, 0].tolist()
                if on:
                    Y = sum(g[j, i] * P[i] for i in on)
                    X += fac * torch.einsum("kl,lab->kab", g, Y)
                    hit = True
            if not hit:
                continue
            Y = _side(el, rs, X, rb, True) + _side(el, rb, X, rs, False)
            Y += _put_diag(el, torch.einsum("epsqt,kest->kepq", T, _diag(el, X)))
            K[j] -= el.untile(Y)
    Jg = el.untile(_put_diag(el, J))
    back = lambda A: A.permute(0, 2, 1, 3).reshape(na * nr, na * nr)  # noqa: E731
    return {"J": back(Jg), "K": back(K)}


def _legendre_pq(Lmax, Mmax, mu):
    """P_L^M and Q_L^M of cosh(mu) without the Condon-Shortley phase, (M, L, ...): upward recurrences for P; for Q_L^0
    and Q_L^1 Christoffel's form near mu = 0 and Miller's backward recurrence elsewhere, then upward in M."""
    x, w = torch.cosh(mu), torch.sinh(mu)
    P = torch.zeros((Mmax + 1, Lmax + 1) + mu.shape, device="cuda", dtype=F64)
    Q = torch.zeros_like(P)
    d = torch.ones_like(mu)
    for M in range(min(Mmax, Lmax) + 1):
        if M:
            d = d * (2 * M - 1) * w
        P[M, M] = d
        if M < Lmax:
            P[M, M + 1] = (2 * M + 1) * x * d
        for L in range(M + 1, Lmax):
            P[M, L + 1] = ((2 * L + 1) * x * P[M, L] - (L + M) * P[M, L - 1]) / (L + 1 - M)
    q0 = -torch.log(torch.tanh(0.5 * mu))
    near = mu < 1.0 / max(Lmax, 1)
    xs, ws, qs = x[near], w[near], q0[near]
    if xs.numel():
        z, o = torch.zeros_like(xs), torch.ones_like(xs)
        p, v, dp, dv = [o, xs], [z, o], [z, o], [z, z]
        for k in range(1, Lmax):
            rec = lambda a: ((2 * k + 1) * xs * a[k] - k * a[k - 1]) / (k + 1)  # noqa: E731
            dp.append(((2 * k + 1) * (p[k] + xs * dp[k]) - k * dp[k - 1]) / (k + 1))
            dv.append(((2 * k + 1) * (v[k] + xs * dv[k]) - k * dv[k - 1]) / (k + 1))
            p.append(rec(p))
            v.append(rec(v))
        for L in range(Lmax + 1):
            Q[0, L][near] = p[L] * qs - v[L]
            if Mmax:
                Q[1, L][near] = ws * dp[L] * qs - p[L] / ws - ws * dv[L]
    far = ~near
    xs, ws, qs, ms = x[far], w[far], q0[far], mu[far]
    if xs.numel():
        N = Lmax + int(math.ceil(37.0 / float(ms.min()))) + 20
        for M in range(min(Mmax, 1) + 1):
            nxt, cur = torch.zeros_like(xs), torch.full_like(xs, 1e-280)
            val = torch.zeros((Lmax + 1,) + xs.shape, device="cuda", dtype=F64)
            for L in range(N, 0, -1):
                nxt, cur = cur, ((2 * L + 1) * xs * cur - (L - M + 1) * nxt) / (L + M)
                if L - 1 <= Lmax:
                    val[L - 1] = cur
                s = torch.where(cur.abs() > 1e200, torch.full_like(cur, 1e-250), torch.ones_like(cur))
                cur, nxt = cur * s, nxt * s
                if L - 1 <= Lmax:
                    val = val * s
            val = val * ((qs if M == 0 else -1.0 / ws) / val[0])
            for L in range(Lmax + 1):
                Q[M, L][far] = val[L]
    for M in range(1, Mmax):
        for L in range(Lmax + 1):
            Q[M + 1, L] = -2.0 * M * x / w * Q[M, L] + (L + M) * (L - M + 1) * Q[M - 1, L]
    return P, Q


def _diatomic_jk(c, seed):
    h = _make_diatomic(c)
    C, f = _diatomic_density(c, h, seed)
    lv, mv = [int(l) for l in h.lval], [int(m) for m in h.mval]
    bval, idx, Rh = np.asarray(h._bval), torch.as_tensor(h.pure_indices().astype(np.int64)).cuda(), h.Rhalf
    h.close()
    el = _Elements(15, bval, False)
    na, nr, nel = len(lv), el.n, el.nel
    Lmax, mmax = 2 * max(lv) + 2, max(mv)
    x, w = _gl(96)
    mu = el.mid[:, None] + el.h[:, None] * x
    B = el.B(x)
    Pd, Qd = _legendre_pq(Lmax, 2 * mmax, mu)
    wd = w * el.h[:, None] * torch.sinh(mu)
    mm = el.mask[:, :, None] * el.mask[:, None, :]
    tab = lambda F, k: torch.einsum("mleq,eq,qi,qj->mleij", F, wd * torch.cosh(mu) ** k, B, B) * mm  # noqa: E731
    p0, p2, q0, q2 = tab(Pd, 0), tab(Pd, 2), tab(Qd, 0), tab(Qd, 2)
    r1, w1, B1, r2, w2, B2 = _inner(el, None, 64, 64, True)
    P2p, Q1p = _legendre_pq(Lmax, 2 * mmax, r2)[0], _legendre_pq(Lmax, 2 * mmax, r1)[1]
    s1, c1, s2, c2 = torch.sinh(r1), torch.cosh(r1), torch.sinh(r2), torch.cosh(r2)
    ang = torch.as_tensor(mv).cuda()
    Pg = torch.zeros((na * nr, na * nr), device="cuda", dtype=F64)
    Pg[idx[:, None], idx[None, :]] = _closed(C, f)
    Pg = Pg.reshape(na, nr, na, nr).permute(0, 2, 1, 3)
    ms = sorted(set(mv))
    sh = {m: torch.nonzero(ang == m)[:, 0] for m in ms}
    dens = {m: el.tiles(Pg[sh[m]][:, sh[m]]) for m in ms if bool((Pg[sh[m]][:, sh[m]] != 0).any())}
    J = torch.zeros((na, na, nel, 15, 15), device="cuda", dtype=F64)
    K = {m: torch.zeros((len(sh[m]), len(sh[m]), el.nel * 15, el.nel * 15), device="cuda", dtype=F64) for m in ms}
    for Ma in range(2 * mmax + 1):
        for L in range(Ma, Lmax + 1):
            G0 = {M: _coupling(lv, mv, L, M, True) for M in {Ma, -Ma}}
            G2 = {M: _coupling(lv, mv, L, M) for M in {Ma, -Ma}}
            if not any(bool((G0[M] != 0).any()) for M in G0):
                continue
            fac = (-1.0) ** Ma * 4 * math.pi * Rh ** 5 / math.prod(range(L - Ma + 1, L + Ma + 1))
            g = [torch.einsum("epq,epqk,epql->epkl", w2 * s2 * c2 ** k * P2p[Ma, L], B2, B2) for k in (0, 2)]
            o = [w1 * s1 * c1 ** k * Q1p[Ma, L] for k in (0, 2)]
            T = lambda a, b: torch.einsum("ep,epi,epj,epkl->eijkl", o[a], B1, B1, g[b])  # noqa: E731
            tr = lambda t: t.permute(0, 3, 4, 1, 2)  # noqa: E731
            t00, t22 = T(0, 0), T(1, 1)
            t00, t22, t02 = t00 + tr(t00), t22 + tr(t22), T(0, 1) + tr(T(1, 0))
            A0, A2, D0, D2 = p0[Ma, L], p2[Ma, L], q0[Ma, L], q2[Ma, L]
            if Ma == 0:  # a density that does not mix m has M = 0 multipoles only
                X0 = sum(torch.einsum("kl,kleij->eij", G0[0][sh[m]][:, sh[m]], _diag(el, p)) for m, p in dens.items())
                X2 = sum(torch.einsum("kl,kleij->eij", G2[0][sh[m]][:, sh[m]], _diag(el, p)) for m, p in dens.items())
                dot = lambda a, b: torch.einsum("eij,eji->e", a, b)  # noqa: E731
                big, small = dot(D0, X0) - dot(D2, X2), dot(A0, X0) - dot(A2, X2)
                above = (big.flip(0).cumsum(0).flip(0) - big)[:, None, None]
                below = (small.cumsum(0) - small)[:, None, None]
                D0z, D2z = D0.clone(), D2.clone()
                D0z[0], D2z[0] = 0.0, 0.0  # nothing lies inside the first element
                on = lambda t, y: torch.einsum("eijkl,ekl->eij", t, y)  # noqa: E731
                V0 = on(t00, X0) - on(t02, X2) + A0 * above + D0z * below
                V2 = on(t22, X2) - on(tr(t02), X0) - A2 * above - D2z * below
                J += fac * (torch.einsum("ji,epq->ijepq", G0[0], V0) + torch.einsum("ji,epq->ijepq", G2[0], V2))
            for mk in ms:
                R = None
                for M in G0:
                    ml = mk - M
                    if ml not in dens:
                        continue
                    a0, a2 = G0[M][sh[mk]][:, sh[ml]], G2[M][sh[mk]][:, sh[ml]]
                    Y0, Y2 = (torch.einsum("kl,ilab->ikab", a, dens[ml]) for a in (a0, a2))
                    S = [torch.einsum("ji,ikab->jkab", a, y) for a in (a0, a2) for y in (Y0, Y2)]
                    R = S if R is None else [u + v for u, v in zip(R, S)]
                if R is None:
                    continue
                x00, x02, x20, x22 = R
                Y = 0
                for up, (i0, i2, j0, j2) in ((True, (A0, A2, D0, D2)), (False, (D0, D2, A0, A2))):
                    Y = Y + _side(el, i0, x00, j0, up) - _side(el, i0, x02, j2, up)
                    Y = Y - _side(el, i2, x20, j0, up) + _side(el, i2, x22, j2, up)
                on = lambda t, y: torch.einsum("epsqt,jkest->jkepq", t, _diag(el, y))  # noqa: E731
                Y += _put_diag(el, on(t00, x00) - on(t02, x02) - on(tr(t02), x20) + on(t22, x22))
                K[mk] -= fac * Y
    def pure(blocks):
        F = torch.zeros((na, na, nr, nr), device="cuda", dtype=F64)
        for m, b in blocks.items():
            F[sh[m][:, None], sh[m][None, :]] = el.untile(b)
        return F.permute(0, 2, 1, 3).reshape(na * nr, na * nr)[idx[:, None], idx[None, :]]
    Jb = {m: _put_diag(el, J[sh[m]][:, sh[m]]) for m in ms}
    return {"J": pure(Jb), "K": pure(K)}


# ---- functionals (energy per volume; derivatives by autograd) ----


def _f_zeta(z1, z2):
    return (z1 ** (4 / 3) + z2 ** (4 / 3) - 2) / (2 ** (4 / 3) - 2)


def _slater(a, b):
    return -0.75 * (6 / math.pi) ** (1 / 3) * (a ** (4 / 3) + b ** (4 / 3))


def _vwn(a, b):
    """Vosko, Wilk, Nusair, Can. J. Phys. 58, 1200 (1980), parametrisation 5."""
    n = a + b
    x = (3 / (4 * math.pi * n)) ** (1 / 6)

    def eps(A, B, Cc, x0):
        X, X0, Qq = x * x + B * x + Cc, x0 * x0 + B * x0 + Cc, math.sqrt(4 * Cc - B * B)
        at = torch.atan(Qq / (2 * x + B))
        return A * (torch.log(x * x / X) + 2 * B / Qq * at
                    - B * x0 / X0 * (torch.log((x - x0) ** 2 / X) + 2 * (B + 2 * x0) / Qq * at))

    eP, eF = eps(0.0310907, 3.72744, 12.9352, -0.10498), eps(0.01554535, 7.06042, 18.0578, -0.32500)
    al = eps(-1 / (6 * math.pi ** 2), 1.13107, 13.0045, -0.0047584)
    z, fz = (a - b) / n, _f_zeta(2 * a / n, 2 * b / n)
    return n * (eP + al * fz / (4 / (9 * (2 ** (1 / 3) - 1))) * (1 - z ** 4) + (eF - eP) * fz * z ** 4)


def _pw_eps(a, b, exact_constants):
    """Perdew, Wang, Phys. Rev. B 45, 13244 (1992)."""
    n = a + b
    rs = (3 / (4 * math.pi * n)) ** (1 / 3)

    def g(A, a1, b1, b2, b3, b4):
        return -2 * A * (1 + a1 * rs) * torch.log(1 + 1 / (2 * A * (b1 * rs.sqrt() + b2 * rs + b3 * rs ** 1.5 + b4 * rs * rs)))

    A = (0.0310907, 0.01554535, 0.0168869) if exact_constants else (0.031091, 0.015545, 0.016887)
    fpp = 1.709920934161365617563962776245 if exact_constants else 1.709921
    eP, eF = g(A[0], 0.21370, 7.5957, 3.5876, 1.6382, 0.49294), g(A[1], 0.20548, 14.1189, 6.1977, 3.3662, 0.62517)
    al = -g(A[2], 0.11125, 10.357, 3.6231, 0.88026, 0.49671)
    z, fz = (a - b) / n, _f_zeta(2 * a / n, 2 * b / n)
    return eP + al * fz / fpp * (1 - z ** 4) + (eF - eP) * fz * z ** 4


def _pbe(a, b, saa, sab, sbb):
    """Perdew, Burke, Ernzerhof, Phys. Rev. Lett. 77, 3865 (1996), exchange and correlation."""
    kap, mu, beta, gam = 0.804, 0.2195149727645171, 0.06672455060314922, (1 - math.log(2)) / math.pi ** 2

    def ex(n, s):
        kf = (3 * math.pi ** 2 * n) ** (1 / 3)
        return -0.75 / math.pi * kf * n * (1 + kap - kap / (1 + mu * s / (2 * kf * n) ** 2 / kap))

    n = a + b
    ec = _pw_eps(a, b, True)
    phi = 0.5 * ((2 * a / n) ** (2 / 3) + (2 * b / n) ** (2 / 3))
    kf = (3 * math.pi ** 2 * n) ** (1 / 3)
    t2 = (saa + 2 * sab + sbb) / (2 * phi * (4 * kf / math.pi).sqrt() * n) ** 2
    g3 = gam * phi ** 3
    A = beta / gam / (torch.exp(-ec / g3) - 1)
    H = g3 * torch.log(1 + beta / gam * t2 * (1 + A * t2) / (1 + A * t2 + (A * t2) ** 2))
    return 0.5 * (ex(2 * a, 4 * saa) + ex(2 * b, 4 * sbb)) + n * (ec + H)


def _energy(func, a, b, s):
    if func == PBE:
        return _pbe(a, b, *s)
    return _slater(a, b) + (_vwn(a, b) if func == LDA else (a + b) * _pw_eps(a, b, False))


def _point_terms(func, rho, grad, w):
    """Exc and N sums and the weights of the Fock matrix at every point: w v_rho, and w (2 v_ss g_s + v_ab g_s')."""
    thr = 1e-12
    n = rho[0] + rho[1]
    on = n >= thr
    a, b = (r.clamp(min=thr / 2)[on].requires_grad_() for r in rho)
    s = []
    if func == PBE:
        dot = lambda u, v: sum(p * q for p, q in zip(u, v))[on]  # noqa: E731
        s = [dot(grad[0], grad[0]), dot(grad[0], grad[1]), dot(grad[1], grad[1])]
        s = [x.requires_grad_() for x in s]
    e = _energy(func, a, b, s)
    d = torch.autograd.grad(e.sum(), [a, b] + s)
    full = []
    for v in d:
        t = torch.zeros_like(n)
        t[on] = v
        full.append(t * w)
    E = torch.stack([(w[on] * e.detach()).sum(), (w * n).sum()])
    terms = []
    for k in (0, 1):
        t = [full[k]]
        if func == PBE:
            t += [2 * full[2 + 2 * k] * g + full[3] * go for g, go in zip(grad[k], grad[1 - k])]
        terms.append(t)
    return E, terms


def _chebyshev(n):
    """Modified Gauss-Chebyshev rule of the second kind (Perez-Jorda, Becke, San-Fabian, J. Chem. Phys. 100, 6520)."""
    i = np.arange(1, n + 1)
    a = i * np.pi / (n + 1)
    s, co = np.sin(a), np.cos(a)
    x = 1 - 2.0 * i / (n + 1) + 2 / np.pi * (1 + 2.0 / 3.0 * s * s) * co * s
    wt = 16.0 / 3.0 / (n + 1) * s ** 4
    return torch.as_tensor(x[::-1].copy()).cuda(), torch.as_tensor(wt[::-1].copy()).cuda()


def _dtheta(l, m, x):
    """d theta_l^m / d(angle) at x = cos(angle)."""
    s = ((1 - x) * (1 + x)).sqrt()
    d = m * x / s * _theta(l, m, x)
    return d + math.sqrt((l - m) * (l + m + 1)) * _theta(l, m + 1, x) if m < l else d


def _atom_xc(c, seed):
    lv, mv = _angular(c)
    na, nn = len(lv), c["nnodes"]
    el = _Elements(nn, hg.get_grid(c["rmax"], c["nelem"], 4, c["zexp"]), True)
    P = _spins(c, *_atom_density(c, seed))
    P = (0.5 * P[0], 0.5 * P[0]) if P[1] is None else P
    nr = el.n
    xc, wc = _chebyshev(4 * max(lv) + 12)
    nphi = 4 * max(mv) + 12
    phi = torch.arange(nphi, device="cuda", dtype=F64) * (2 * math.pi / nphi)
    cth, ph = xc.repeat_interleave(nphi), phi.repeat(len(xc))
    wang, sth = wc.repeat_interleave(nphi) * (2 * math.pi / nphi), ((1 - cth) * (1 + cth)).sqrt()
    rot = [torch.exp(1j * m * ph) for m in mv]
    Y = torch.stack([_theta(l, m, cth) * r for l, m, r in zip(lv, mv, rot)])
    Yt = torch.stack([_dtheta(l, m, cth) * r for l, m, r in zip(lv, mv, rot)])
    Yp = torch.stack([1j * m * y for m, y in zip(mv, Y)])
    xq, wq = _chebyshev(5 * nn)
    B, dB = el.B(xq), el.B(xq, 1)
    E = torch.zeros(2, device="cuda", dtype=F64)
    H = [torch.zeros((na, nr, na, nr), device="cuda", dtype=F64) for _ in range(2)]
    for e in range(el.nel):
        r = el.mid[e] + el.h[e] * xq
        R = B / r[:, None] * el.mask[e]
        dR = (dB / el.h[e] - B / r[:, None]) / r[:, None] * el.mask[e]
        f = lambda y, rad: torch.einsum("ka,qi->kiqa", y, rad.to(y.dtype)).reshape(na * nn, -1)  # noqa: E731
        rr, ss = r.repeat_interleave(len(cth)), sth.repeat(len(r))
        b = f(Y, R)
        gb = [f(Y, dR), f(Yt, R) / rr, f(Yp, R) / (rr * ss)]
        w = (wq * el.h[e] * r * r).repeat_interleave(len(cth)) * wang.repeat(len(r))
        g = el.gc[e]
        sel = (torch.arange(na, device="cuda")[:, None] * nr + g[None, :]).reshape(-1)
        msk = el.mask[e].repeat(na)
        rho, grad = [], []
        for p in P:
            pb = (p[sel[:, None], sel[None, :]] * msk[:, None] * msk[None, :]).to(b.dtype) @ b
            rho.append((pb.conj() * b).real.sum(0))
            grad.append([2 * (pb.conj() * d).real.sum(0) for d in gb] if c["func"] == PBE else [])
        Ee, terms = _point_terms(c["func"], rho, grad, w)
        E += Ee
        for s in range(1 if c["restricted"] else 2):
            Z = terms[s][0] * b.conj()
            M = (b @ Z.T).real
            if c["func"] == PBE:
                Xm = ((gb[0] * terms[s][1] + gb[1] * terms[s][2] + gb[2] * terms[s][3]) @ b.conj().T).real
                M = M + Xm + Xm.T
            H[s].reshape(na * nr, na * nr).index_put_((sel[:, None], sel[None, :]), M * msk[:, None] * msk[None, :],
                                                     accumulate=True)
    out = [h.reshape(na * nr, na * nr) for h in H]
    return {"E": E, "Ha": out[0], "Hb": None if c["restricted"] else out[1]}


def _diatomic_xc(c, seed):
    h = _make_diatomic(c)
    P = _spins(c, *_diatomic_density(c, h, seed))
    P = (0.5 * P[0], 0.5 * P[0]) if P[1] is None else P
    lv, mv = [int(l) for l in h.lval], [int(m) for m in h.mval]
    idx, Rh, bval, nbf = torch.as_tensor(h.pure_indices().astype(np.int64)).cuda(), h.Rhalf, np.asarray(h._bval), h.nbf
    h.close()
    el = _Elements(15, bval, False)
    na, nr = len(lv), el.n
    where = torch.full((na * nr,), -1, device="cuda")
    where[idx] = torch.arange(nbf, device="cuda")
    cth, wang = _chebyshev(4 * max(lv) + 12)
    sth2 = (1 - cth) * (1 + cth)
    xq, wq = _chebyshev(75)
    B, dB = el.B(xq), el.B(xq, 1)
    E = torch.zeros(2, device="cuda", dtype=F64)
    H = [torch.zeros((nbf, nbf), device="cuda", dtype=F64) for _ in range(2)]
    for e in range(el.nel):
        mu = el.mid[e] + el.h[e] * xq
        s2 = torch.sinh(mu)[:, None] ** 2 + sth2
        hs = (Rh * s2.sqrt()).reshape(-1)
        w = (2 * math.pi * wang * (wq * el.h[e] * torch.sinh(mu))[:, None] * Rh ** 3 * s2).reshape(-1)
        blocks = []
        rho, grad = [0.0, 0.0], [[0.0, 0.0], [0.0, 0.0]]
        for m in sorted(set(mv)):
            sh = [k for k in range(na) if mv[k] == m]
            Y = torch.stack([_theta(lv[k], m, cth) for k in sh])
            dY = torch.stack([_dtheta(lv[k], m, cth) for k in sh])
            f = lambda y, rad: torch.einsum("ka,qi->kiqa", y, rad).reshape(len(sh) * 15, -1)  # noqa: E731
            pos = where[(torch.as_tensor(sh).cuda()[:, None] * nr + el.gc[e][None, :]).reshape(-1)]
            ok = (el.mask[e].repeat(len(sh)) > 0) & (pos >= 0)
            b = f(Y, B)[ok]
            gb = [f(Y, dB / el.h[e])[ok] / hs, f(dY, B)[ok] / hs]
            pos = pos[ok]
            blocks.append((pos, b, gb))
            for s in (0, 1):
                pb = P[s][pos[:, None], pos[None, :]] @ b
                rho[s] = rho[s] + (pb * b).sum(0)
                for k in (0, 1):
                    grad[s][k] = grad[s][k] + 2 * (pb * gb[k]).sum(0)
        Ee, terms = _point_terms(c["func"], rho, grad if c["func"] == PBE else [[], []], w)
        E += Ee
        for s in range(1 if c["restricted"] else 2):
            for pos, b, gb in blocks:
                M = (b * terms[s][0]) @ b.T
                if c["func"] == PBE:
                    X = (gb[0] * terms[s][1] + gb[1] * terms[s][2]) @ b.T
                    M = M + X + X.T
                H[s].index_put_((pos[:, None], pos[None, :]), M, accumulate=True)
    return {"E": E, "Ha": H[0], "Hb": None if c["restricted"] else H[1]}


def exact(case, seed):
    c = case
    if c["kind"] in ("fock", "fock_host"):
        return _atom_jk(c, seed)
    if c["kind"] == "xc":
        return _atom_xc(c, seed)
    if c["kind"] == "dfock":
        return _diatomic_jk(c, seed)
    if c["kind"] == "dxc":
        return _diatomic_xc(c, seed)
    return None  # a converged solve has no closed form
