"""Performance cases: the calls a program makes through the public entry points of ``ipg``.

A case is a dict of plain values; ``prepare`` makes what a program holds before the call (the
system or the device buffers, the potential, the SNAP handle), ``run`` is one pass, ``work`` the
bytes and operations the pass cannot do without and ``exact`` its results in plain 64-bit torch.

Kinds of case
  pair   pair potentials on device buffers (ipg_pair_eval_dev): E, F, W6 of an MD step
  ef     SNAP energy and forces of one system on device buffers (ipg_snap_energy_forces_dev)
  md     SNAP energy and forces of a set of configurations in fixed buffers (DeviceBatch.evaluate)
  train  a force-matching step: E, F, W6, the loss and dL/dbeta (DeviceBatch.train_step)
  desc   compute_all_descriptors of a host system: B, dB, W
  vjp    the pullback of (E, F) to beta and positions for a host system (SNAP.vjp)
  fit    the fitting matrices of many host configurations (SNAP.fitting_matrices)

Crystals are FCC or BCC with jitter; ``n`` below the number of lattice sites leaves vacancies, so
atom counts are odd and neighbor counts uneven.
"""
import ctypes as C
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "interatomicpotentials.jl_b200"))

import ipg  # noqa: E402
from ipg import workloads as W  # noqa: E402
from ipg._lib import PAIR_GRAPH, SNAP_ADJOINT, SNAP_PLAIN, PairTerm, WANT_E, WANT_F, WANT_W, lib  # noqa: E402

BASIS = {"fcc": ((0, 0, 0), (0.5, 0.5, 0), (0.5, 0, 0.5), (0, 0.5, 0.5)), "bcc": ((0, 0, 0), (0.5, 0.5, 0.5))}
# two-species parameters of the workloads, and a third species for the draws
RADII, WEIGHT = (0.5, 0.45, 0.47), (1.0, 0.5, 0.8)


def _snap(name, kind, n, **more):
    return dict({"name": name, "kind": kind, "n": n, "lattice": "bcc", "a": 3.2, "jitter": 0.12, "twojmax": 8,
                 "species": 2, "rcutfac": 5.0, "mode": "adjoint", "chem": False, "quadratic": False, "bzero": False,
                 "open": False}, **more)


def listed():
    return [
        # a small argon box, the smallest MD step: launches and latency count
        dict(name="pair_lj_1000", kind="pair", terms="lj", n=1000, open=False, graph=False),
        # an Ar/Xe mixture with five terms, an ordinary MD step
        dict(name="pair_lc_32000", kind="pair", terms="lc", n=32000, open=False, graph=False),
        # the same mixture at the size of a large run
        dict(name="pair_lc_4m", kind="pair", terms="lc", n=4121204, open=False, graph=False),
        # MD of a small cell with a vacancy, replayed step after step in fixed buffers
        _snap("snap_j8_md_249", "md", 249, nconf=1),
        # a single-species system at the cheaper basis
        _snap("snap_j6_8192", "ef", 8192, a=3.3, jitter=0.1, twojmax=6, species=1, rcutfac=4.7),
        # the two-species system at the largest common basis, the production MD step
        _snap("snap_j8_54000", "ef", 54000),
        # the reference's own force route: every dB/dr formed, then contracted with beta
        _snap("snap_j8_plain_16000", "ef", 16000, mode="plain"),
        # one optimiser step of force matching over a training set of uneven configurations
        _snap("snap_j8_train_512", "train", 0, jitter=0.05, nconf=512, nmin=32, nmax=2000),
        # descriptors of one system for analysis or an external model
        _snap("snap_j8_desc_8192", "desc", 8192),
        # the gradient of a loss on energy and forces with respect to beta and positions
        _snap("snap_j8_vjp_16000", "vjp", 16000),
        # explicit multi-element SNAP
        _snap("snap_j6_chem_1999", "ef", 1999, twojmax=6, chem=True),
        # the least-squares system of a small training set
        _snap("snap_j6_fit_48", "fit", 0, twojmax=6, nconf=48, nmin=32, nmax=250, jitter=0.05),
    ]


def draw(rng):
    log = lambda lo, hi: int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))  # noqa: E731
    kind = rng.choice(["pair", "pair", "ef", "ef", "ef", "md", "train", "desc", "vjp", "fit"])
    if kind == "pair":
        periodic = rng.random() < 0.75
        return dict(kind="pair", terms=rng.choice(["lj", "lc"]), n=log(60, 2000000), open=not periodic,
                    graph=periodic and rng.random() < 0.5)
    c = dict(lattice=rng.choice(["bcc", "fcc"]), jitter=round(rng.uniform(0.03, 0.12), 3),
             a=round(rng.uniform(3.1, 3.4), 3), twojmax=rng.choice([2, 3, 4, 5, 6, 6, 7, 8, 8, 8]),
             species=rng.choice([1, 2, 2, 3]), rcutfac=round(rng.uniform(4.5, 5.2), 3))
    if c["lattice"] == "fcc":  # about the same density as the BCC crystals
        c["a"] = round(c["a"] * 1.26, 3)
    if kind == "ef":
        option = rng.choice(["none", "none", "none", "plain", "chem", "quadratic", "open"])
        hi = {"none": 54000, "plain": 16000, "chem": 2000, "quadratic": 2000, "open": 20000}[option]
        if option in ("chem", "quadratic"):
            c.update(twojmax=rng.choice([2, 4, 5, 6]), species=2)
        c.update(n=log(30, hi), mode="plain" if option == "plain" else "adjoint", chem=option == "chem",
                 quadratic=option == "quadratic", open=option == "open", bzero=rng.random() < 0.25)
    elif kind == "md":
        c.update(n=log(16, 2000), nconf=rng.choice([1, 1, 2, 5]))
    elif kind == "train":
        c.update(n=0, nconf=log(2, 128), nmin=32, nmax=log(100, 2000))
    elif kind == "desc":
        c.update(n=log(30, 8192), bzero=rng.random() < 0.25)
    elif kind == "vjp":
        c.update(n=log(30, 16000))
    else:
        c.update(n=0, nconf=log(2, 48), nmin=32, nmax=log(60, 250), twojmax=rng.choice([2, 4, 5, 6]))
    c = _snap("", kind, c.pop("n"), **c)
    del c["name"]
    return c


# ---- inputs ---------------------------------------------------------------------------------
def _crystal(lattice, a, n, jitter, gen, device="cpu"):
    """(positions [n][3], box [3]): the smallest near-cubic crystal with at least n sites, n of
    them kept in lattice order."""
    per = len(BASIS[lattice])
    c = max(1, math.ceil((n / per) ** (1.0 / 3.0) - 1e-9))
    nc = [c, c, c]
    while nc[0] > 1 and (nc[0] - 1) * nc[1] * nc[2] * per >= n:
        nc[0] -= 1
    ax = [torch.arange(k, dtype=torch.float64, device=device) for k in nc]
    g = torch.stack(torch.meshgrid(*ax, indexing="ij"), -1).reshape(-1, 1, 3)
    pts = (g + torch.tensor(BASIS[lattice], dtype=torch.float64, device=device)).reshape(-1, 3)
    if len(pts) > n:
        pts = pts[torch.randperm(len(pts), generator=gen, device=device)[:n].sort().values]
    pos = pts * a + jitter * torch.randn(pts.shape, generator=gen, dtype=torch.float64, device=device)
    return pos, np.array(nc, dtype=np.float64) * a


def _gen(seed, device="cpu"):
    return torch.Generator(device=device).manual_seed(int(seed))


def _pair_inputs(case, seed):
    """(positions, species ids, L, [(coefficient, potential)], symbols) on the device, atomic units."""
    A = ipg.units.angstrom
    gen = _gen(seed, "cuda")
    if case["terms"] == "lj":
        pos, box = _crystal("fcc", 5.26, case["n"], 0.05, gen, "cuda")
        sp = torch.zeros(case["n"], dtype=torch.int32, device="cuda")
        terms, symbols = [(1.0, ipg.LennardJones(0.0104 * ipg.units.eV, 3.4 * A, 8.5 * A, ["Ar"]))], {"Ar": 0}
    else:
        pos, box = _crystal("fcc", 5.5, case["n"], 0.08, gen, "cuda")
        sp = (torch.rand(case["n"], generator=gen, device="cuda") < 0.5).to(torch.int32)
        terms, symbols = W.lc_potential().flat_terms(), {"Ar": 0, "Xe": 1}
    L = np.full(3, np.inf) if case["open"] else box * A
    return pos * A, sp, L, terms, symbols


def _conf_sizes(case):
    if case["kind"] in ("train", "fit"):  # the set's sizes belong to the case: the same for every seed
        r = np.random.default_rng(case["nconf"] * 10007 + case["nmax"])
        return [int(k) for k in r.integers(case["nmin"], case["nmax"] + 1, case["nconf"])]
    return [case["n"]] * case.get("nconf", 1)


def _snap_inputs(case, seed):
    """[(positions, box lengths, species ids)] per configuration, and beta, on the host."""
    gen = _gen(seed)
    nsp, out = case["species"], []
    p = torch.tensor([1.0, 0.0, 0.0] if nsp == 1 else [0.7, 0.3, 0.0] if nsp == 2 else [0.6, 0.25, 0.15])
    for n in _conf_sizes(case):
        pos, box = _crystal(case["lattice"], case["a"], n, case["jitter"], gen)
        sp = torch.multinomial(p, n, replacement=True, generator=gen)
        out.append((pos.numpy(), np.full(3, np.inf) if case["open"] else box, sp.numpy().astype(np.int32)))
    k = ipg.get_num_snap_coeffs(case["twojmax"], nsp, case["chem"])
    beta = 1e-2 * torch.randn((nsp, k), generator=gen, dtype=torch.float64).numpy()
    if case["quadratic"]:  # small products beside the linear part
        q = 1e-5 * torch.randn((nsp, k * (k + 1) // 2), generator=gen, dtype=torch.float64).numpy()
        beta = np.concatenate([beta, q], axis=1)
    return out, beta, gen


def _system(conf):
    pos, box, sp = conf
    names = np.array(["A", "B", "C"])
    periodic = np.isfinite(box)
    return ipg.System(pos, names[sp].tolist(), np.where(periodic, box, 1.0), tuple(periodic))


def _basis(case):
    nsp = case["species"]
    return ipg.SNAP(case["n"], case["twojmax"], ["A", "B", "C"][:nsp], case["rcutfac"], 0.0, 0.99363, RADII[:nsp],
                    WEIGHT[:nsp], chem_flag=case["chem"], bnorm_flag=case["chem"], bzero_flag=case["bzero"],
                    switch_flag=True, quadratic_flag=case["quadratic"])


def prepare(case, seed):
    s = {"case": case}
    if case["kind"] == "pair":
        s["pos"], s["sp"], s["L"], terms, symbols = _pair_inputs(case, seed)
        s["terms"] = (PairTerm * len(terms))(*[p.term(symbols, c) for c, p in terms])
        s["ctx"] = ipg.default_context()
    else:
        confs, s["beta"], gen = _snap_inputs(case, seed)
        s["snap"] = _basis(case)
        s["ctx"] = s["snap"].ctx
        if case["kind"] == "ef":
            pos, s["L"], sp = confs[0]
            s["pos"], s["sp"] = torch.from_numpy(pos).cuda(), torch.from_numpy(sp).cuda()
        else:
            s["systems"] = [_system(c) for c in confs]
    if case["kind"] in ("pair", "ef"):
        n = case["n"]
        s["E"] = torch.zeros(1, dtype=torch.float64, device="cuda")
        s["F"] = torch.zeros((n, 3), dtype=torch.float64, device="cuda")
        s["W"] = torch.zeros(6, dtype=torch.float64, device="cuda")
    elif case["kind"] in ("md", "train"):
        s["batch"] = ipg.DeviceBatch(s["snap"], s["systems"])
        if case["kind"] == "train":
            s["F_ref"] = (0.1 * torch.randn(s["batch"].F.shape, generator=gen, dtype=torch.float64)).cuda()
    elif case["kind"] == "vjp":
        s["gF"] = torch.randn((case["n"], 3), generator=gen, dtype=torch.float64).numpy()
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    ptr = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
    host = lambda a: a.ctypes.data_as(C.c_void_p)  # noqa: E731
    if kind == "pair":
        flags = WANT_E | WANT_F | WANT_W | (PAIR_GRAPH if case["graph"] else 0)
        s["ctx"].check(lib().ipg_pair_eval_dev(s["ctx"].handle, case["n"], ptr(s["pos"]), ptr(s["sp"]), host(s["L"]),
                                               C.cast(s["terms"], C.c_void_p), len(s["terms"]), ptr(s["E"]),
                                               ptr(s["F"]), ptr(s["W"]), flags))
        return s["E"], s["F"], s["W"]
    if kind == "ef":
        mode = SNAP_PLAIN if case["mode"] == "plain" else SNAP_ADJOINT
        s["ctx"].check(lib().ipg_snap_energy_forces_dev(s["snap"].handle, case["n"], ptr(s["pos"]), ptr(s["sp"]),
                                                        host(s["L"]), host(s["beta"]), 0.0, mode, ptr(s["E"]),
                                                        ptr(s["F"]), ptr(s["W"])))
        return s["E"], s["F"], s["W"]
    if kind == "md":
        return s["batch"].evaluate(s["beta"])
    if kind == "train":
        loss, gbeta = s["batch"].train_step(s["beta"], s["F_ref"])
        return s["batch"].E, s["batch"].F, s["batch"].W, loss, gbeta
    if kind == "desc":
        return ipg.compute_all_descriptors(s["systems"][0], s["snap"])
    if kind == "vjp":
        return s["snap"].vjp(s["systems"][0], s["beta"], 0.7, s["gF"])
    return s["snap"].fitting_matrices(s["systems"])


# ---- work -----------------------------------------------------------------------------------
def _triples(J):
    return [(a, b, j) for a in range(J + 1) for b in range(a + 1) for j in range(a - b, min(J, a + b) + 1, 2)]


def _products(J):
    """(distinct products u1 u2 of the half plane, their uses over every j) of one atom."""
    prod = uses = 0
    for a in range(J + 1):
        for b in range(a + 1):
            js = range(a - b, min(J, a + b) + 1, 2)
            for m1 in range(-a, a + 1, 2):
                for m2 in range(-b, b + 1, 2):
                    if m1 + m2 > 0:
                        continue
                    rows = [j for j in js if abs(m1 + m2) <= j]
                    for k1 in range(-a, a + 1, 2):
                        for k2 in range(-b, b + 1, 2):
                            u = sum(abs(k1 + k2) <= j for j in rows)
                            prod += u > 0
                            uses += u
    return prod, uses


def work(case):
    kind = case["kind"]
    if kind == "pair":
        n, lj = case["n"], case["terms"] == "lj"
        half = 38.9 if lj else 43.1  # half pairs per atom in the bulk crystal
        return {"bytes": 52.0 * n, "flops": n * half * (40.0 if lj else 200.0)}
    sizes = _conf_sizes(case)
    n, J, nsp = sum(sizes), case["twojmax"], case["species"]
    density = len(BASIS[case["lattice"]]) / case["a"] ** 3
    nb = 4.0 / 3.0 * math.pi * (0.97 * case["rcutfac"]) ** 3 * density * n / sum(
        math.ceil((k / 2) ** (1 / 3) - 1e-9) ** 3 * 2 for k in sizes)
    hu = sum((j // 2 + 1) * (j + 1) for j in range(J + 1))
    prod, uses = _products(J)
    elem = nsp ** 2 if case["chem"] else 1
    kn = ipg.get_num_snap_coeffs(J, nsp, case["chem"], case["quadratic"]) * nsp
    u, z, force = 16.0 * hu * nb, (8.0 * prod + 4.0 * uses) * elem, 28.0 * hu * nb
    zt = sum((j // 2 + 1) * (j + 1) for _, _, j in _triples(J))
    db = 3 * 4.0 * zt * nb * elem + u
    io = 28.0 * n + 24.0 * n + 8.0 * kn
    if kind in ("ef", "md"):
        flops = u + z + (db if case["mode"] == "plain" or case["chem"] or case["quadratic"] else force)
        return {"bytes": io, "flops": n * flops}
    if kind == "train":
        return {"bytes": io + 24.0 * n, "flops": n * (u + 2 * z + force + u + 4.0 * zt)}
    if kind == "vjp":
        return {"bytes": io + 24.0 * n, "flops": n * (u + 3 * z + 3 * force + 4.0 * zt)}
    if kind == "desc":
        return {"bytes": 28.0 * n + 8.0 * n * (kn / nsp + 3 * kn), "flops": n * (u + z + db)}
    return {"bytes": 28.0 * n + 8.0 * kn * (3 * n + 7 * len(sizes)), "flops": n * (u + z + db)}


# ---- exact values ---------------------------------------------------------------------------
def _displacement(d, L):
    """Minimum image of d for box lengths L (inf: open axis)."""
    return d - torch.where(torch.isinf(L), torch.zeros_like(d), L * torch.round(d / L))


def _pairs(pos, L, cut, rows=2048):
    """Directed pairs (i, j) within cut[i, j] (a function of index tensors) and x_j - x_i."""
    n, ii, jj, rr = len(pos), [], [], []
    for a in range(0, n, rows):
        d = _displacement(pos[None, :, :] - pos[a:a + rows, None, :], L)
        i = torch.arange(a, min(n, a + rows), device=pos.device)
        ok = (d * d).sum(-1) <= cut(i[:, None], torch.arange(n, device=pos.device)[None, :]) ** 2
        ok[i - a, i] = False
        p, q = ok.nonzero(as_tuple=True)
        ii.append(p + a)
        jj.append(q)
        rr.append(d[p, q])
    return torch.cat(ii), torch.cat(jj), torch.cat(rr)


def _exact_pair(case, seed):
    if case["n"] > 40000:
        return None
    pos, sp, L, terms, symbols = _pair_inputs(case, seed)
    L = torch.from_numpy(np.asarray(L)).cuda()
    rmax = max(p.get_rcutoff() for _, p in terms)
    i, j, d = _pairs(pos, L, lambda a, b: torch.full_like(a * b, rmax, dtype=torch.float64))
    i, j, r = i[i < j], j[i < j], -d[i < j]
    R = r.norm(dim=1)
    V, g = torch.zeros_like(R), torch.zeros_like(R)
    for c, p in terms:
        ids = torch.tensor([symbols[s] for s in p.species], device="cuda")
        on = torch.isin(sp[i], ids) & torch.isin(sp[j], ids) & (R <= p.rcutoff)
        if p.kind == "LJ":
            s6 = (p.sigma / R) ** 6
            v, f = 4 * p.epsilon * (s6 * s6 - s6), 24 * p.epsilon * (2 * s6 * s6 - s6) / R ** 2
        elif p.kind == "BM":
            e = p.A * torch.exp((p.sigma - R) / p.rho)
            v = e + (p.C / R) ** 6 - (p.D / R) ** 8
            f = e / p.rho / R + ((p.C / R) ** 6 - (p.D / R) ** 8) / R ** 2
        else:  # ZBL, the screening function to the base e of the potential
            k = p.Z1 * p.Z2 * p.e ** 2
            x = R / (0.8854 * 0.529 / (p.Z1 ** 0.23 + p.Z2 ** 0.23))
            phi, dphi = torch.zeros_like(R), torch.zeros_like(R)
            for w, b in ((0.18175, 3.19980), (0.50986, 0.94229), (0.28022, 0.40290), (0.02817, 0.20162)):
                phi += w * p.e ** (-b * x)
                dphi -= w * b * p.e ** (-b * x)
            v, f = k * phi / R, k * (phi + x * dphi) / R ** 3
        V += torch.where(on, c * v, 0.0)
        g += torch.where(on, c * f, 0.0)
    f = g[:, None] * r
    F = torch.zeros_like(pos).index_add_(0, i, f).index_add_(0, j, -f)
    w = torch.stack([(r[:, a] * f[:, b]).sum() for a, b in ((0, 0), (1, 1), (2, 2), (2, 1), (2, 0), (1, 0))])
    return V.sum().reshape(1), F, w


def _cg(j1, j2, j):
    """Clebsch-Gordan coefficients [j1+1][j2+1][j+1] of doubled angular momenta (Racah's sum)."""
    f = math.factorial
    out = np.zeros((j1 + 1, j2 + 1, j + 1))
    tri = f((j1 + j2 - j) // 2) * f((j1 - j2 + j) // 2) * f((j2 - j1 + j) // 2) / f((j1 + j2 + j) // 2 + 1)
    for p in range(j1 + 1):
        for q in range(j2 + 1):
            m1, m2 = 2 * p - j1, 2 * q - j2
            m = m1 + m2
            if abs(m) > j:
                continue
            s = 0.0
            for z in range((j1 + j2) + 1):
                a = ((j1 + j2 - j) // 2 - z, (j1 - m1) // 2 - z, (j2 + m2) // 2 - z, (j - j2 + m1) // 2 + z,
                     (j - j1 - m2) // 2 + z)
                if min(a) >= 0:
                    s += (-1) ** z / (f(z) * math.prod(f(k) for k in a))
            out[p, q, (m + j) // 2] = s * math.sqrt((j + 1) * tri * f((j1 + m1) // 2) * f((j1 - m1) // 2) * f(
                (j2 + m2) // 2) * f((j2 - m2) // 2) * f((j + m) // 2) * f((j - m) // 2))
    return out


class _Bispectrum:
    """B of each centre atom from the displacements to its neighbors, by the tensor products of
    the spin representations: U^j is the top component of U^1 x U^(j-1)."""

    def __init__(self, case):
        self.case, self.J, self.nsp = case, case["twojmax"], case["species"]
        J = self.J
        self.idxb = [(a, b, j) for a, b, j in _triples(J) if j >= a]
        c = lambda *t: torch.from_numpy(_cg(*t)).cuda()  # noqa: E731
        self.up = [None, None] + [c(1, j - 1, j) for j in range(2, J + 1)]
        self.mix = {t: c(*t).reshape((t[0] + 1) * (t[1] + 1), -1).to(torch.complex128) for t in self.idxb}
        self.radii = torch.tensor(RADII[:self.nsp], dtype=torch.float64, device="cuda")
        self.weight = torch.tensor(WEIGHT[:self.nsp], dtype=torch.float64, device="cuda")

    def pairs(self, pos, sp, L):
        fac = self.case["rcutfac"]
        return _pairs(pos, L, lambda a, b: (self.radii[sp[a]] + self.radii[sp[b]]) * fac)

    def __call__(self, d, owner, n, si, sj, centre):
        """B [n][K] of the centres; pair p has displacement d[p], centre owner[p], species si, sj."""
        r = d.norm(dim=1)
        rc = (self.radii[si] + self.radii[sj]) * self.case["rcutfac"]
        z0 = r / torch.tan(0.99363 * math.pi * r / rc)
        r0 = torch.sqrt(r * r + z0 * z0)
        a = torch.complex(z0 / r0, -d[:, 2] / r0)
        b = torch.complex(d[:, 1] / r0, -d[:, 0] / r0)
        w = 0.5 * (torch.cos(math.pi * r / rc) + 1.0) * self.weight[sj]
        g = torch.stack([torch.stack([a.conj(), -b.conj()], -1), torch.stack([b, a], -1)], -2)
        chem = self.case["chem"]
        ne = self.nsp if chem else 1
        slot = owner * ne + (sj if chem else 0)
        own = torch.arange(n, device="cuda") * ne + (centre if chem else 0)
        u, tot = torch.ones((len(d), 1, 1), dtype=torch.complex128, device="cuda"), []
        for j in range(self.J + 1):
            if j == 1:
                u = g
            elif j > 1:
                c, v = self.up[j], 0.0
                for s in (0, 1):
                    for t in (0, 1):
                        k = torch.arange(j, device="cuda")
                        x = u * g[:, s, t, None, None] * (c[s, k, k + s][:, None] * c[t, k, k + t][None, :])
                        v = v + torch.nn.functional.pad(x, (t, 1 - t, s, 1 - s))
                u = v
            q = torch.zeros((n * ne, j + 1, j + 1), dtype=torch.complex128, device="cuda")
            q = q.index_add(0, own, torch.eye(j + 1, dtype=torch.complex128, device="cuda").expand(n, -1, -1))
            tot.append(q.index_add(0, slot, u * w[:, None, None]).reshape(n, ne, j + 1, j + 1))
        out = []
        for e1 in range(ne):
            for e2 in range(ne):
                z = []
                for t in self.idxb:
                    x = torch.einsum("nab,ncd->nacbd", tot[t[0]][:, e1], tot[t[1]][:, e2])
                    x = x.reshape(n, *[(t[0] + 1) * (t[1] + 1)] * 2)
                    x = self.mix[t].T @ (x @ self.mix[t])
                    z.append(x / (t[2] + 1) if chem else x)
                for e3 in range(ne):
                    B = torch.stack([(tot[t[2]][:, e3].conj() * x).sum((1, 2)).real for t, x in zip(self.idxb, z)], 1)
                    if self.case["bzero"]:
                        shift = torch.tensor([1.0 if chem else t[2] + 1.0 for t in self.idxb], dtype=torch.float64,
                                             device="cuda")
                        here = (centre == e1) & (centre == e2) & (centre == e3) if chem else centre >= 0
                        B = B - shift * here[:, None]
                    out.append(B)
        B = torch.cat(out, 1)
        if self.case["quadratic"]:
            k, m = torch.triu_indices(B.shape[1], B.shape[1], device="cuda")
            B = torch.cat([B, B[:, k] * B[:, m] * torch.where(k == m, 0.5, 1.0)], 1)
        return B

    def chunks(self, n, i, size):
        """Ranges of centres with their pairs (the pairs are ordered by centre)."""
        for a in range(0, n, size):
            b = min(n, a + size)
            lo, hi = torch.searchsorted(i, torch.tensor([a, b], device="cuda")).tolist()
            yield a, b, slice(lo, hi)


def _exact_snap(case, seed):
    confs, beta, gen = _snap_inputs(case, seed)
    kind, n_all, J = case["kind"], sum(len(c[0]) for c in confs), case["twojmax"]
    # what it would cost, in atoms of a twojmax 8 system, energy and forces
    cost = n_all * {"ef": 1, "md": 1, "train": 2, "desc": 12, "vjp": 4, "fit": 12}[kind] * ((J + 1) / 9.0) ** 4
    cost *= case["species"] ** 3 if case["chem"] else 1
    if cost > 120000:
        return None
    model = _Bispectrum(case)
    bt = torch.from_numpy(beta).cuda()
    K, nsp = bt.shape[1], case["species"]
    gF = torch.randn((n_all, 3), generator=gen, dtype=torch.float64).cuda() if kind in ("vjp", "train") else None
    if kind == "train":
        gF *= 0.1  # the reference forces
    E, F, Wv, at = [], [], [], 0
    gb, gp, Bs, dBs, Ws, As = torch.zeros_like(bt), [], [], [], [], []
    loss = 0.0
    for pos, box, sp in confs:
        n = len(pos)
        x, s, L = torch.from_numpy(pos).cuda(), torch.from_numpy(sp).cuda().long(), torch.from_numpy(box).cuda()
        i, j, d = model.pairs(x, s, L)
        order = torch.argsort(i * n + j)
        i, j, d = i[order], j[order], d[order]
        raw = x[i] - x[j]
        size = max(64, int(1500 * (9.0 / (J + 1)) ** 3 / (nsp ** 2 if case["chem"] else 1)))
        size = max(64, size // 3) if kind in ("vjp", "desc", "fit") else size
        e, f = torch.zeros(1, dtype=torch.float64, device="cuda"), torch.zeros_like(x)
        w = torch.zeros(6, dtype=torch.float64, device="cuda")
        AB = ((0, 0), (1, 1), (2, 2), (1, 2), (0, 2), (0, 1))
        if kind in ("desc", "fit"):
            dB = torch.zeros((n, 3, nsp * K), dtype=torch.float64, device="cuda")
            Wd = torch.zeros((6, nsp * K), dtype=torch.float64, device="cuda")
            B = torch.zeros((n, K), dtype=torch.float64, device="cuda")
            for a, b, p in model.chunks(n, i, size):
                dp = d[p].clone().requires_grad_(True)
                Bc = model(dp, i[p] - a, b - a, s[i[p]], s[j[p]], s[a:b])
                B[a:b] = Bc.detach()
                for k in range(K):
                    (q,) = torch.autograd.grad(Bc[:, k].sum(), dp, retain_graph=True)
                    for t in range(nsp):
                        on = (s[i[p]] == t)[:, None] * q
                        dB[:, :, t * K + k].index_add_(0, i[p], on).index_add_(0, j[p], -on)
                        for v, (m, l) in enumerate(AB):
                            Wd[v, t * K + k] += (on[:, m] * raw[p][:, l]).sum()
            Bs.append(B)
            dBs.append(dB)
            Ws.append(Wd)
            As.append(torch.cat([B[s == t].sum(0) for t in range(nsp)]))
        else:
            for a, b, p in model.chunks(n, i, size):
                dp, bq = d[p].clone().requires_grad_(True), bt.clone().requires_grad_(True)
                Bc = model(dp, i[p] - a, b - a, s[i[p]], s[j[p]], s[a:b])
                ec = (Bc * bq[s[a:b]]).sum()
                (q,) = torch.autograd.grad(ec, dp, create_graph=kind == "vjp")
                e += ec.detach()
                f.index_add_(0, i[p], q.detach()).index_add_(0, j[p], -q.detach())
                w += torch.stack([(q.detach()[:, m] * raw[p][:, l]).sum() for m, l in AB])
                if kind == "vjp":  # d(gE E + gF . F): F = sum over pairs of q on i, -q on j
                    phi = 0.7 * ec + (q * (gF[i[p]] - gF[j[p]])).sum()
                    h, hb = torch.autograd.grad(phi, (dp, bq))
                    gb += hb
                    gp.append((i[p], j[p], h))
            if kind == "train":
                G = 2.0 * (f - gF[at:at + n])
                loss = loss + 0.25 * (G * G).sum()
                for a, b, p in model.chunks(n, i, size):  # dL/dbeta = G . dF/dbeta, a directional derivative of B
                    dp = d[p].clone().requires_grad_(True)
                    Bc = model(dp, i[p] - a, b - a, s[i[p]], s[j[p]], s[a:b])
                    y = torch.ones_like(Bc, requires_grad=True)
                    (q,) = torch.autograd.grad((Bc * y).sum(), dp, create_graph=True)
                    (h,) = torch.autograd.grad((q * (G[i[p]] - G[j[p]])).sum(), y)
                    gb.index_add_(0, s[a:b], h)
        at += n
        E.append(e)
        F.append(f)
        Wv.append(w)
    if kind == "desc":
        return Bs[0].cpu().numpy(), dBs[0].cpu().numpy(), Ws[0].cpu().numpy()
    if kind == "fit":
        return (torch.stack(As).cpu().numpy(), torch.cat([m.reshape(-1, nsp * K) for m in dBs]).cpu().numpy(),
                torch.stack(Ws).cpu().numpy())
    if kind == "vjp":
        g = torch.zeros_like(x)
        for i, j, h in gp:
            g.index_add_(0, j, h).index_add_(0, i, -h)
        return gb.cpu().numpy(), np.float64(0.7), g.cpu().numpy()
    if kind == "ef":
        return E[0], F[0], Wv[0]
    out = (torch.cat(E), torch.cat(F), torch.stack(Wv))
    return out if kind == "md" else out + (loss.reshape(1), gb)


def exact(case, seed):
    if case["kind"] == "pair":
        return _exact_pair(case, seed)
    return _exact_snap(case, seed)
