"""Performance cases of the H/S setup and its adjoint, through the public entry points.

A case is a plain dict.  `kind` names the call:
  host      Context.setup: host arrays in, HS/HSDIAG back in page-locked host
            memory (the drop-in replacement of calkpt.F:153-185)
  resident  KPoint.run: one k-point's inputs and HS on the device
  batch     Context.setup_batch: a k-list on one crystal, HS on the device
  forces    KPoint.forces: dE/dPOS of the band energy for given eigenvectors
and the other fields name the crystal (`cell`, `natom`, `mult`, `rkmax`,
`lmax`, `lnsmax`, `lo`, `orb`), the arithmetic (`prec`, `s_sph`, `s_hns`), the
k-points (`nk`) and the bands (`nb`).

The crystals are seeded: radial values, potentials and LO coefficients have
the distributions of hack_wein2k_b200.synth, positions are a jittered grid at
the density of its 100-atom cell (about 80 bohr^3 per atom) or its ABO3
supercell, every k-point is a general one.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from hack_wein2k_b200 import lapw1gpu, synth

DEV = "cuda"
LO_CHOICE = {"none": ((), ()), "lapw": ((0, 1, 2), ()), "apw": ((1,), (0, 1, 2))}


def _case(name, kind, **kw):
    c = dict(name=name, kind=kind, cell="grid", natom=1, mult=1, rkmax=7.0, lmax=10, lnsmax=4, lo="lapw", orb=False,
             prec="split", s_sph=5, s_hns=4, nk=1, nb=0)
    c.update(kw)
    return c


def listed():
    return [
        # one-atom metal, host call in the library's default arithmetic: the smallest drop-in call, all latency
        _case("host_1atom_fp64", "host", natom=1, lo="none", prec="fp64"),
        # small unit cell with equivalent atoms and APW+lo (WIEN2k's default basis): the everyday lapw1 call
        _case("host_6atom_apw_fp64", "host", natom=6, mult=3, lo="apw", prec="fp64"),
        # a k-mesh of a small cell: sixteen k-points in one launch
        _case("batch_6atom_16k_fp64", "batch", natom=6, mult=2, lo="apw", prec="fp64", nk=16),
        # LDA+U oxide: orbital potentials on some atoms, local rotations, an odd l cutoff
        _case("resident_18atom_orb_split", "resident", natom=18, mult=2, lo="apw", orb=True, lmax=9, prec="split"),
        # the 40-atom ABO3 supercell (the c1 workload), FP64 and split, inputs resident
        _case("resident_40atom_fp64", "resident", cell="abo3", natom=40, prec="fp64"),
        _case("resident_40atom_split", "resident", cell="abo3", natom=40),
        # the same supercell through the host call, HS copied back: what a Fortran caller sees
        _case("host_40atom_split", "host", cell="abo3", natom=40),
        # k-points of the supercell as one batch (the c2 workload, four of its k-points)
        _case("batch_40atom_4k_split", "batch", cell="abo3", natom=40, nk=4),
        # band-energy gradient of the supercell, in both arithmetics
        _case("forces_40atom_fp64", "forces", cell="abo3", natom=40, prec="fp64", nb=200),
        _case("forces_40atom_split", "forces", cell="abo3", natom=40, nb=200),
        # 100 atoms at RKmax 8 (the size of the c4 workload): the largest setup and the largest gradient
        _case("resident_100atom_split", "resident", natom=100, rkmax=8.0),
        _case("forces_100atom_split", "forces", natom=100, rkmax=8.0, nb=400),
    ]


def draw(rng):
    """One more case: sizes spread over their logarithm between the one-atom
    cell and cells of some sixty atoms, odd counts among them."""
    kind = rng.choice(["host", "resident", "resident", "batch", "forces"])
    prec = rng.choice(["fp64", "split", "split"])
    most = 32 if prec == "fp64" else 64
    natom = max(1, round(math.exp(rng.uniform(math.log(1 if kind != "forces" else 4), math.log(most)))))
    c = _case("", kind, natom=natom, mult=rng.choice([1, 1, 2, 3, 5]), rkmax=round(rng.uniform(5.5, 7.9), 2),
              lmax=rng.choice([8, 9, 10, 10, 10, 11, 12]), lnsmax=rng.choice([2, 3, 4, 4, 4]),
              lo=rng.choice(["none", "lapw", "apw", "apw"]), prec=prec)
    if prec == "split":
        c["s_sph"] = rng.choice([4, 5, 5, 5, 6, 7])
        c["s_hns"] = rng.choice([4, 4, 5, c["s_sph"]])
    if kind == "batch":
        c["nk"] = rng.randint(2, 9)
        c["natom"] = min(natom, 27)
    if kind == "forces":
        c["nb"] = 4 * c["natom"] + rng.randint(1, 16)
    elif rng.random() < 0.2:
        c["orb"] = True
    del c["name"]
    return c


# ---------------------------------------------------------------- inputs
def _grid_cell(rng, natom, mult):
    """natom sites of a 4.3-bohr grid, moved by up to 0.2 bohr per axis, in
    types of `mult` consecutive sites (the last type takes the rest)."""
    g = [1, 1, 1]
    while g[0] * g[1] * g[2] < natom:
        g[g.index(min(g))] += 1
    sites = [(i, j, k) for i in range(g[0]) for j in range(g[1]) for k in range(g[2])]
    pick = sorted(rng.choice(len(sites), size=natom, replace=False))
    a = 4.3
    pos = (np.array([sites[q] for q in pick], dtype=float) + 0.5) * a + rng.uniform(-0.2, 0.2, size=(natom, 3))
    box = [a * n for n in g]
    pos /= np.array(box)
    types = []
    for q in range(0, natom, mult):
        rmt = 1.8 if q == 0 else float(rng.uniform(1.8, 1.9))
        types.append(dict(pos=[list(map(float, x)) for x in pos[q:q + mult]], rmt=rmt))
    return synth.Cell("P", tuple(box), (90.0, 90.0, 90.0), types)


def _problems(case, seed):
    """The case's k-points on its seeded crystal.  The k-points and the cell's
    box belong to the case, so that the basis has one size for all seeds."""
    rng = np.random.default_rng([int(seed), case["natom"], case["nk"]])
    rng_k = np.random.default_rng([case["natom"], case["nk"], int(1000 * case["rkmax"])])
    cell = synth.cell_abo3_222() if case["cell"] == "abo3" else _grid_cell(rng, case["natom"], case["mult"])
    lo_l, apw_l = LO_CHOICE[case["lo"]]
    orb = [(t + 1, (2,)) for t in range(0, len(cell.types), 3)] if case["orb"] else ()
    out, params = [], None
    for _ in range(case["nk"]):
        k = rng_k.uniform(0.05, 0.45, size=3)
        p = synth.synth_problem(cell, case["rkmax"], k, lmax=case["lmax"], lnsmax=case["lnsmax"], lo_l=lo_l,
                                apw_l=apw_l, rotate_local=case["cell"] != "abo3", orb=orb, rng=rng, params=params)
        params = p._params
        out.append(p)
    return out


def _bands(case, p, seed):
    """Eigenvector-like columns (plane-wave weights falling with |k+G|, unit
    length), ascending energies and a smeared occupation, on the host."""
    rng = np.random.default_rng([int(seed), 77])
    nb = case["nb"]
    w = 1.0 / (1.0 + 0.25 * p.rk ** 2)
    w[p.nv:] = 0.05
    c = (rng.standard_normal((nb, p.n)) + 1j * rng.standard_normal((nb, p.n))) * w
    c /= np.linalg.norm(c, axis=1, keepdims=True)
    eps = np.sort(rng.uniform(-1.0, 1.0, size=nb))
    occ = 2.0 / (1.0 + np.exp((eps - 0.6) / 0.05))
    return c, eps, occ


_contexts = {}


def _context(case):
    """The program's library context for the case's arithmetic."""
    key = ("fp64",) if case["prec"] == "fp64" else ("split", case["s_sph"], case["s_hns"])
    if key not in _contexts:
        if key[0] == "fp64":
            _contexts[key] = lapw1gpu.Context(0, prec=lapw1gpu.PREC_FP64)
        else:
            ctx = lapw1gpu.Context(0, prec=lapw1gpu.PREC_SPLIT, slices=key[1])
            ctx.set_slices(key[1], key[2])
            _contexts[key] = ctx
    return _contexts[key]


def prepare(case, seed):
    ctx = _context(case)
    probs = _problems(case, seed)
    s = dict(kind=case["kind"], ctx=ctx, probs=probs)
    if case["kind"] == "host":
        n = probs[0].n
        s["keep"] = torch.empty(2 * n * (n + 1), dtype=torch.float64, pin_memory=True)
        flat = s["keep"].numpy().view(np.complex128)
        s["hs"] = flat[:n * n].reshape((n, n), order="F")
        s["hsdiag"] = flat[n * n:]
        return s
    s["kps"] = [ctx.upload(p) for p in probs]
    if case["kind"] == "forces":
        c, eps, occ = _bands(case, probs[0], seed)
        s["c"], s["eps"], s["occ"] = (torch.from_numpy(x).to(DEV) for x in (c, eps, occ))
        s["grad"] = torch.empty((probs[0].ndf, 3), dtype=torch.float64, device=DEV)
        return s
    s["hs"] = [torch.empty((p.n, p.n), dtype=torch.complex128, device=DEV) for p in probs]
    s["hsdiag"] = [torch.empty(p.n, dtype=torch.complex128, device=DEV) for p in probs]
    return s


def run(state):
    kind, ctx = state["kind"], state["ctx"]
    if kind == "host":
        return ctx.setup(state["probs"][0], hs=state["hs"], hsdiag=state["hsdiag"])
    if kind == "forces":
        p = state["probs"][0]
        state["kps"][0].forces(state["c"].data_ptr(), p.n, state["c"].shape[0], state["occ"].data_ptr(),
                               state["eps"].data_ptr(), state["grad"].data_ptr())
        return state["grad"]
    if kind == "resident":
        state["kps"][0].run(state["hs"][0].data_ptr(), state["probs"][0].n, state["hsdiag"][0].data_ptr())
    else:
        ctx.setup_batch(state["kps"], [h.data_ptr() for h in state["hs"]], [p.n for p in state["probs"]],
                        [d.data_ptr() for d in state["hsdiag"]])
    return state["hs"] + state["hsdiag"]


def _sizes(case):
    """(n, nv, types, atoms) without building the problem: nv from the sphere
    of radius rkmax / min(Rmt) at the cell's volume."""
    if case["cell"] == "abo3":
        nat = ndf = 40
        vol, rmin = 14.8 ** 3, 1.6
    else:
        ndf, nat = case["natom"], -(-case["natom"] // case["mult"])
        g = [1, 1, 1]
        while g[0] * g[1] * g[2] < ndf:
            g[g.index(min(g))] += 1
        vol, rmin = 4.3 ** 3 * g[0] * g[1] * g[2], 1.8
    nv = vol * (case["rkmax"] / rmin) ** 3 / (6.0 * math.pi ** 2)
    lo_l, apw_l = LO_CHOICE[case["lo"]]
    return nv + ndf * sum(2 * l + 1 for l in lo_l + apw_l), nv, nat, ndf


def work(case):
    n, nv, nat, ndf = _sizes(case)
    lt, k = case["lmax"] + 1, 2 * ndf * (case["lnsmax"] + 1) ** 2
    pairs = 0.5 * nv * nv
    inputs = 16.0 * 9 * 625 * nat + 48.0 * n
    if case["kind"] == "forces":
        # density matrices (lower triangles), spherical pairs, projections of the non-spherical part
        flops = 2 * 8.0 * case["nb"] * 0.5 * n * n + 2.0 * (6 * lt * nat + 12 * ndf) * pairs + 8.0 * k * 4 * case["nb"] * n
        return {"bytes": inputs + 16.0 * n * case["nb"] + 24.0 * ndf, "flops": flops}
    flops = 2.0 * (6 * lt * nat + 4 * ndf + 4 * nat) * pairs + 8.0 * k * 0.5 * n * n
    return {"bytes": case["nk"] * (inputs + 16.0 * n * (n + 1)), "flops": case["nk"] * flops}


# ---------------------------------------------------------------- 64-bit values
# H and S of one k-point as sums over l of (2l+1) P_l(k_J.k_I) U_l V_l^H, the
# step-function and potential tables and the non-spherical and orbital terms
# as matrix products, in plain torch FP64 / complex128.
def _bessel(lmax, x):
    """j_0..j_lmax of the 1-d tensor x: power series below 1, else Miller's
    downward recursion normalised by sum (2l+1) j_l^2 = 1."""
    out = torch.zeros(lmax + 1, len(x), dtype=torch.float64, device=x.device)
    xs = torch.where(x < 1.0, x, torch.zeros_like(x))
    pre = torch.ones_like(x)
    for l in range(lmax + 1):
        if l:
            pre = pre * xs / (2 * l + 1)
        term, tot = torch.ones_like(x), torch.ones_like(x)
        for k in range(1, 20):
            term = term * (-0.5 * xs * xs) / (k * (2 * l + 2 * k + 1))
            tot = tot + term
        out[l] = pre * tot
    xb = torch.where(x < 1.0, torch.ones_like(x), x)
    hi, lo = torch.zeros_like(x), torch.full_like(x, 1e-30)
    top = 60
    norm = (2 * top + 1) * lo * lo
    keep = {}
    for l in range(top, 0, -1):
        hi, lo = lo, (2 * l + 1) / xb * lo - hi
        norm = norm + (2 * l - 1) * lo * lo
        if l - 1 <= lmax:
            keep[l - 1] = lo
    for l in range(lmax + 1):
        out[l] = torch.where(x < 1.0, out[l], keep[l] / norm.sqrt())
    return out


def _ylm(v, lmax):
    """Complex Y_lm (Condon-Shortley) of the rows of v, [rows, (lmax+1)^2]."""
    u = v / v.norm(dim=1, keepdim=True)
    z, e = u[:, 2], torch.complex(u[:, 0], u[:, 1])
    out = torch.zeros(len(v), (lmax + 1) ** 2, dtype=torch.complex128, device=v.device)
    for m in range(lmax + 1):
        q = {m: torch.full_like(z, float((-1) ** m * math.prod(range(1, 2 * m, 2))))}
        if m < lmax:
            q[m + 1] = (2 * m + 1) * z * q[m]
        for l in range(m + 2, lmax + 1):
            q[l] = ((2 * l - 1) * z * q[l - 1] - (l + m - 1) * q[l - 2]) / (l - m)
        for l in range(m, lmax + 1):
            nrm = math.sqrt((2 * l + 1) / (4 * math.pi) * math.factorial(l - m) / math.factorial(l + m))
            y = nrm * q[l] * e ** m
            out[:, l * l + l + m] = y
            out[:, l * l + l - m] = (-1) ** m * y.conj()
    return out


class _Exact:
    def __init__(self, p, dev):
        t = lambda a: torch.as_tensor(np.ascontiguousarray(a), device=dev)  # noqa: E731
        self.p, self.dev = p, dev
        self.n, self.nv, self.lt = p.n, p.nv, p.ltop
        self.kz = t(p.kzz.astype(np.int64))
        self.k = torch.stack([t(p.xk), t(p.yk), t(p.zk)], dim=1)
        self.rk = t(p.rk)
        self.pos = t(p.pos.astype(np.float64))
        self.typ = np.repeat(np.arange(p.nat), p.mult)
        kr = self.kz.double() @ self.pos.T
        self.phase = torch.polar(torch.ones_like(kr), 2 * math.pi * (kr - kr.round()))  # [n, ndf]
        # LO rows: (type, l, index) in the order type, l, index, atom, m
        self.lo = [(a, l, j) for a in range(p.nat) for l in range(4) for j in range(int(p.ilo[a, l]))
                   for _ in range((2 * l + 1) * int(p.mult[a]))]
        self.al = torch.zeros(p.nat, self.lt, self.nv, dtype=torch.float64, device=dev)
        self.bl = torch.zeros_like(self.al)
        rk = self.rk[:self.nv]
        for a in range(p.nat):
            r = float(p.rmt[a])
            x = r * rk
            j = _bessel(self.lt, x)
            for l in range(self.lt):
                dj = -j[1] if l == 0 else j[l - 1] - (l + 1) / x * j[l]
                u, ud, du, dud = (float(q[a, l]) for q in (p.p, p.pe, p.dp, p.dpe))
                if p.lapw[a, l]:
                    self.al[a, l] = rk * dj * ud - j[l] * dud
                    self.bl[a, l] = j[l] * du - rk * dj * u
                else:
                    self.al[a, l] = j[l] / u / (r * r)

    def sides(self, l):
        """Row side and the S and H column sides of one l: [n, 4 ndf] complex;
        components (u, udot, lo, kinetic surface term of an LO column)."""
        p, nv = self.p, self.nv
        x = torch.zeros(self.n, p.nat, 4, dtype=torch.float64, device=self.dev)
        s, h = torch.zeros_like(x), torch.zeros_like(x)
        for a in range(p.nat):
            r2 = float(p.rmt[a]) ** 2
            u, ud, du, dud, chn, e = (float(q[a, l]) for q in (p.p, p.pe, p.dp, p.dpe, p.pei, p.e))
            vif = 4 * math.pi * p.vi * r2 * r2
            al, bl = self.al[a, l], self.bl[a, l]
            x[:nv, a, 0], x[:nv, a, 1], x[:nv, a, 3] = al, bl, al * u + bl * ud
            s[:nv, a, 0], s[:nv, a, 1] = vif * al, vif * (chn if p.lapw[a, l] else 0.0) * bl
            h[:nv, a, 0] = vif * ((e + r2 * u * du) * al + r2 * ud * du * bl)
            h[:nv, a, 1] = vif * ((1 + r2 * u * dud) * al + (e * chn + r2 * ud * dud) * bl)
            if l < 4:
                pi12, pe12, dpl = (float(q[a, l]) for q in (p.pi12lo, p.pe12lo, p.dplo))
                for j in range(int(p.ilo[a, l])):
                    rows = [nv + q for q, w in enumerate(self.lo) if w == (a, l, j)]
                    A, B, C, elo = (float(q[a, j, l]) for q in (p.alo, p.blo, p.clo, p.elo))
                    half = 0.5 * (elo + e)
                    vec = lambda *v: torch.tensor(v, dtype=torch.float64, device=self.dev)  # noqa: E731
                    x[rows, a] = vec(A, B, C, 0.0)
                    s[rows, a] = vif * vec(A + pi12 * C, B * chn + pe12 * C, C + pe12 * B + A * pi12, 0.0)
                    h[rows, a] = vif * vec(A * e + 0.5 * B + C * pi12 * half,
                                           B * chn * e + 0.5 * A + 0.5 * C * pi12 + C * pe12 * half,
                                           C * elo + 0.5 * B * pi12 + half * (A * pi12 + pe12 * B),
                                           0.5 * r2 * (A * du + B * dud + C * dpl))
        full = lambda m: (m[:, self.typ] * self.phase[:, :, None]).reshape(self.n, -1)  # noqa: E731
        return full(x), full(s), full(h)

    def legendre(self, c0, c1):
        """(2l+1) P_l of rows 0..n-1 against columns c0..c1-1, l by l; plane-wave
        pairs along one line take x P_(l-1) (hamilt.F:250-281)."""
        x = self.k @ self.k[c0:c1].T
        den = self.rk[:, None] * self.rk[None, c0:c1]
        x = torch.where(den > 1e-8, x / den, x)
        top = x.abs() >= 0.9999999
        top[self.nv:] = False
        if c1 > self.nv:
            top[:, max(0, self.nv - c0):] = False
        p0, p1 = torch.ones_like(x), x
        for l in range(self.lt):
            if l == 0:
                yield l, p0
                continue
            if l > 1:
                q = x * p1
                p0, p1 = p1, torch.where(top, q, q + (l - 1) / l * (q - p0))
            yield l, (2 * l + 1) * p1

    def delta(self, c0, c1):
        """Flat table index of K_J - K_I over the plane-wave rows and columns."""
        kz = self.kz[:self.nv]
        self.half = (kz.max(0).values - kz.min(0).values)
        d = kz[:, None] - kz[None, c0:min(c1, self.nv)] + self.half
        w = 2 * self.half + 1
        return (d[..., 2] * w[1] + d[..., 1]) * w[0] + d[..., 0]

    def box(self):
        h = [int(v) for v in self.half]
        ax = [torch.arange(-q, q + 1, device=self.dev) for q in h]
        z, y, x = torch.meshgrid(ax[2], ax[1], ax[0], indexing="ij")
        return torch.stack([x, y, z], dim=-1).reshape(-1, 3)

    def step(self, d, a):
        """Step-function term of atom a at the integer vectors d (0 at d = 0)."""
        p = self.p
        g = (d.double() @ torch.as_tensor(np.asarray(p.bkzz), device=self.dev).T).norm(dim=1)
        h = g * float(p.rmt[self.typ[a]])
        f = 3 * float(p.v[self.typ[a]]) * (h * h.cos() - h.sin()) / h ** 3
        f = torch.where((d == 0).all(dim=1), torch.zeros_like(f), f)
        q = d.double() @ self.pos[a]
        return torch.polar(torch.ones_like(q), 2 * math.pi * (q - q.round())) * f

    def tables(self):
        p, d = self.p, self.box()
        th = torch.zeros(len(d), dtype=torch.complex128, device=self.dev)
        for a in range(p.ndf):
            th += self.step(d, a)
        th[(d == 0).all(dim=1)] = 1.0 - float(np.sum(p.v * p.mult))
        w1, w2, w3 = p.warp_half
        half = torch.tensor([w1, w2, w3], device=self.dev)
        inside = (d.abs() <= half).all(dim=1)
        c = torch.where(inside[:, None], d + half, torch.zeros_like(d))
        warp = torch.as_tensor(p.warp, device=self.dev)[c[:, 2], c[:, 1], c[:, 0]]
        return th, torch.where(inside, warp, torch.zeros_like(warp))

    def alm(self, a, lmax):
        """(ALM, BLM, CLM) of every row for atom a: [3, n, (lmax+1)^2]."""
        p, t, nv = self.p, int(self.typ[a]), self.nv
        mats = [torch.as_tensor(np.asarray(m, dtype=np.float64), device=self.dev) for m in (p.rotij[a], p.rotloc[t])]
        y = _ylm(self.k @ mats[0] @ mats[1], lmax).conj() * self.phase[:, a:a + 1]
        y = y * (4 * math.pi * math.sqrt(p.vi) * float(p.rmt[t]) ** 2)
        out = torch.zeros(3, self.n, (lmax + 1) ** 2, dtype=torch.complex128, device=self.dev)
        for l in range(lmax + 1):
            sl = slice(l * l, (l + 1) ** 2)
            yl = y[:, sl] * 1j ** l
            out[0, :nv, sl] = yl[:nv] * self.al[t, l][:, None]
            out[1, :nv, sl] = yl[:nv] * self.bl[t, l][:, None]
            for q, (ta, ll, j) in enumerate(self.lo):
                if (ta, ll) == (t, l):
                    for r, arr in enumerate((p.alo, p.blo, p.clo)):
                        out[r, nv + q, sl] = yl[nv + q] * float(arr[t, j, l])
        return out

    def nonspherical(self):
        """Per atom the rows X [n, q] and the q x q matrix M of the update
        HS(i,j) += conj(X(i)) M X(j), i >= j: the HNS and the orbital terms."""
        p, ns = self.p, (self.p.lnsmax + 1) ** 2
        for a in range(p.ndf):
            t = int(self.typ[a])
            x = self.alm(a, p.lnsmax)
            T = torch.as_tensor(p.tns[t].reshape(3, 3, 25, 25)[:, :, :ns, :ns], device=self.dev)
            yield a, x.permute(1, 0, 2).reshape(self.n, -1), T.permute(1, 3, 0, 2).reshape(3 * ns, 3 * ns)
            for i in range(p.natorb):
                if int(p.iatom[i]) - 1 != t:
                    continue
                for q in range(int(p.nlorb[i])):
                    l = int(p.lorb[i, q])
                    xl = self.alm(a, l)[:, :, l * l:(l + 1) ** 2]
                    g = torch.eye(3, dtype=torch.complex128, device=self.dev)
                    g[1, 1] = float(p.pei[t, l])
                    if l < 4:
                        g[0, 2] = g[2, 0] = float(p.pi12lo[t, l])
                        g[1, 2] = g[2, 1] = float(p.pe12lo[t, l])
                    v = torch.as_tensor(p.vorb[i, l, 3 - l:4 + l, 3 - l:4 + l], device=self.dev)
                    yield a, xl.permute(1, 0, 2).reshape(self.n, -1), torch.kron(g, v)

    def setup(self):
        """HS[i, j] and HSDIAG of the packed state."""
        n, nv, dev = self.n, self.nv, self.dev
        S = torch.zeros(n, n, dtype=torch.complex128, device=dev)
        H = torch.zeros_like(S)
        sides = [self.sides(l) for l in range(self.lt)]
        th = wp = None
        for c0 in range(0, n, 1024):
            c1 = min(n, c0 + 1024)
            for l, w in self.legendre(c0, c1):
                u, s, h = sides[l]
                S[:, c0:c1] += w * (u @ s[c0:c1].conj().T)
                H[:, c0:c1] += w * (u @ h[c0:c1].conj().T)
            if c0 < nv:
                ix = self.delta(c0, c1)
                if th is None:
                    th, wp = self.tables()
                e = min(c1, nv)
                S[:nv, c0:e] += th[ix]
                H[:nv, c0:e] += th[ix] * (self.k[:nv] @ self.k[c0:e].T) + wp[ix]
        del sides
        HS = torch.triu(S, 1) + torch.triu(H).T
        hsd = S.diagonal().clone()
        del S, H
        low = torch.zeros_like(HS)
        for _, x, m in self.nonspherical():
            low += x.conj() @ (m @ x.T)
        return HS + torch.tril(low), hsd

    def forces(self, c, eps, occ):
        """dE/dPOS of E = sum_(J<I) 2 Re[conj(H_IJ) rho_JI - conj(S_JI) rhoe_JI]."""
        n, nv, dev = self.n, self.nv, self.dev
        tpk = 2 * math.pi * self.kz.double()
        grad = torch.zeros(self.p.ndf, 3, dtype=torch.float64, device=dev)
        ct = c.T
        rho = 2 * torch.triu((ct * occ) @ c.conj(), 1)
        rhoe = 2 * torch.triu((ct * (occ * eps)) @ c.conj(), 1)
        bins = None
        sides = [self.sides(l) for l in range(self.lt)]
        for c0 in range(0, n, 1024):
            c1 = min(n, c0 + 1024)
            for l, w in self.legendre(c0, c1):
                u, s, h = sides[l]
                qh, qs = w * rho[:, c0:c1], -w * rhoe[:, c0:c1]
                for q, v in ((qh, h[c0:c1]), (qs, s[c0:c1])):
                    f = (u.conj() * (q @ v)).imag.reshape(n, -1, 4).sum(2)
                    grad += f.T @ tpk
                    f = ((q.conj().T @ u).conj() * v).imag.reshape(c1 - c0, -1, 4).sum(2)
                    grad -= f.T @ tpk[c0:c1]
            if c0 < nv:
                ix, e = self.delta(c0, c1), min(c1, nv)
                if bins is None:
                    bins = torch.zeros(int((2 * self.half + 1).prod()), 2, dtype=torch.float64, device=dev)
                b = (self.k[:nv] @ self.k[c0:e].T) * rho[:nv, c0:e] - rhoe[:nv, c0:e]
                bins.index_add_(0, ix.reshape(-1), torch.view_as_real(b).reshape(-1, 2))
        del sides
        d, bc = self.box(), torch.view_as_complex(bins)
        for a in range(self.p.ndf):
            grad[a] += 2 * math.pi * ((self.step(d, a).conj() * bc).imag @ d.double())
        for a, x, m in self.nonspherical():
            z = x @ m.T
            grad[a] += (z.conj() * (rho @ x)).imag.sum(1) @ tpk
            grad[a] -= (x * (rho.T @ z.conj())).imag.sum(1) @ tpk
        return grad


def exact(case, seed):
    probs = _problems(case, seed)
    dev = DEV if torch.cuda.is_available() else "cpu"
    if case["kind"] == "forces":
        c, eps, occ = (torch.from_numpy(q).to(dev) for q in _bands(case, probs[0], seed))
        return _Exact(probs[0], dev).forces(c, eps, occ)
    got = [_Exact(p, dev).setup() for p in probs]
    if case["kind"] == "host":
        return got[0]
    return [h.T.contiguous() for h, _ in got] + [d for _, d in got]
