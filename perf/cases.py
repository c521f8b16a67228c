"""The calls whose speed matters to a user of the library, as cases that can be
timed and checked: H psi sweeps, the band solvers of one SCF iteration, the
subspace eigensolver, the Hartree solve, many small cells at once and the
adjoint forces, on the cells of the benchmark and the tests (Si8, Si64, Si512,
C8 and the set of 32 small cells) and on other sizes of the same ranges.

listed() and draw(rng) give cases, prepare(case, seed) what a program holds
before the call, run(state) one pass, work(case) the bytes and operations the
pass cannot do without, tolerance(case) how far two correct results may be
apart and exact(case, seed) the same pass in 64 bits by plain torch.

Atoms, potentials and bands come from the seed; atom positions are diamond
sites with Gaussian jitter, bands are low-pass filtered noise, S-orthonormal
where the solvers expect that (formed in plain torch, so that two versions of
the library start from the same bits).
"""
from __future__ import annotations

import numpy as np
import torch

from rspacedist_b200 import forces as F
from rspacedist_b200 import kukan as K
from rspacedist_b200 import lib as L
from rspacedist_b200 import system as S

F64, F32 = torch.float64, torch.float32
EDGE = {"si_paw": 10.26, "c_ncps": 6.74}   # lattice constants (bohr)
FD = (-205 / 72, 8 / 5, -1 / 5, 8 / 315, -1 / 560)   # second derivative, +-4 points


# ------------------------------------------------------------------- the cases
def _cell(species, cells, grid, bands, **kw):
    c = {"species": species, "bands": bands, **kw}
    for ax, a, n in zip("xyz", cells, grid):
        c["c" + ax], c["n" + ax] = a, n
    return c


def listed():
    return [
        # one H psi of the smallest cell (Si8, 32^3, 20 bands): latency and launches count
        _cell("si_paw", (1, 1, 1), (32, 32, 32), 20, name="hpsi_f32_si8", kind="hpsi", f64=False),
        # the Si64 supercell at a spacing of 0.33 bohr: rows of 62 points, no multiple of four
        _cell("si_paw", (2, 2, 2), (62, 62, 62), 160, name="hpsi_f32_si64_62", kind="hpsi",
              f64=False),
        # the headline sweep: Si512, 128^3, 1100 bands
        _cell("si_paw", (4, 4, 4), (128, 128, 128), 1100, name="hpsi_f32_si512", kind="hpsi",
              f64=False),
        # 32 independent Si8 and C8 cells of uneven grids in one call
        {"name": "batch_f32_32cells", "kind": "batch", "cells": 32, "bands": 20, "spacing": 0.30},
        # the band update of a large SCF iteration: DIIS sweeps, Cholesky-QR, H psi (Si512)
        _cell("si_paw", (4, 4, 4), (128, 128, 128), 1100, name="diis_f32_si512", kind="diis",
              f64=False),
        # one whole scf_diag of Si64 (Rayleigh-Ritz, DIIS, reorder), mixed and plain FP64
        _cell("si_paw", (2, 2, 2), (64, 64, 64), 160, name="scf_f32_si64", kind="scf", f64=False,
              cg=False),
        _cell("si_paw", (2, 2, 2), (64, 64, 64), 160, name="scf_f64_si64", kind="scf", f64=True,
              cg=False),
        # one scf_diag of Si8 with kukan's default parameters (Rayleigh-Ritz, then CG), FP64
        _cell("si_paw", (1, 1, 1), (32, 32, 32), 20, name="scf_cg_f64_si8", kind="scf", f64=True,
              cg=True),
        # the subspace eigenproblem of Si512
        {"name": "syev_1100", "kind": "syev", "n": 1100},
        # the first Hartree solve (no warm start) on the dense grids of Si64 (mixed) and Si8 (FP64)
        {"name": "hartree_f32_128", "kind": "hartree", "nx": 128, "ny": 128, "nz": 128,
         "h": 20.52 / 128, "atoms": 64, "f64": False},
        {"name": "hartree_f64_64", "kind": "hartree", "nx": 64, "ny": 64, "nz": 64,
         "h": 10.26 / 64, "atoms": 8, "f64": True},
        # the projector part of the atomic forces of Si64: one adjoint pass over the bands
        _cell("si_paw", (2, 2, 2), (64, 64, 64), 160, name="forces_f32_si64", kind="forces",
              f64=False),
    ]


def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["hpsi", "hpsi", "hpsi", "batch", "diis", "scf", "scf", "syev", "hartree",
                       "hartree", "forces"])
    if kind == "batch":
        return {"kind": kind, "cells": _log(rng, 4, 64), "bands": _log(rng, 6, 32),
                "spacing": round(rng.uniform(0.27, 0.36), 3)}
    if kind == "syev":
        return {"kind": kind, "n": _log(rng, 16, 1100)}
    if kind == "hartree":
        n = [2 * _log(rng, 20, 72) for _ in range(3)]
        return {"kind": kind, "nx": n[0], "ny": n[1], "nz": n[2],
                "h": round(rng.uniform(0.14, 0.18), 4), "atoms": _log(rng, 4, 64),
                "f64": rng.random() < 0.4}
    big = {"hpsi": 4, "diis": 3, "scf": 2, "forces": 3}[kind]
    species = rng.choice(["si_paw", "si_paw", "c_ncps"])
    cells = [_log(rng, 1, big) for _ in range(3)]
    h = rng.uniform(0.28, 0.36)
    grid = [max(18, 2 * round(EDGE[species] * c / (2 * h)) + 2 * rng.randrange(-1, 2))
            for c in cells]
    atoms = 8 * cells[0] * cells[1] * cells[2]
    bands = max(4, round(atoms * rng.uniform(1.6, 2.6)))
    cg = kind == "scf" and atoms <= 16 and rng.random() < 0.5
    case = _cell(species, cells, grid, bands, kind=kind, f64=rng.random() < 0.3)
    if kind == "scf":
        case["cg"] = cg
    return case


# ------------------------------------------------------------- inputs of a cell
def _host_cell(case, seed):
    """The cell (atoms, sphere lists, projector tables) of a case."""
    cells = np.array([case["cx"], case["cy"], case["cz"]])
    edge = EDGE[case["species"]] * cells
    ijk = np.stack(np.meshgrid(*[np.arange(c) for c in cells], indexing="ij"), -1).reshape(-1, 1, 3)
    pos = ((S.DIAMOND_BASIS + ijk) * EDGE[case["species"]]).reshape(-1, 3)
    pos = (pos + np.random.default_rng(seed).normal(0.0, 0.05, pos.shape)) % edge - edge / 2
    return S.make_cell(edge, (case["nx"], case["ny"], case["nz"]), pos,
                       S.load_dataset(case["species"]))


def _shape(cell):
    nx, ny, nz = cell.shape
    return nz, ny, nx


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _noise(cell, nb, seed, dtype):
    """Low-pass filtered noise on the grid, of unit norm per band."""
    gen = _gen(seed)
    f = [torch.fft.fftfreq(n, device="cuda", dtype=F64) / h
         for n, h in zip(_shape(cell), cell.h[::-1])]
    k2 = f[0][:, None, None] ** 2 + f[1][:, None] ** 2 + f[2] ** 2
    filt = torch.exp(-k2 / (0.05 / 0.33 ** 2)).to(F32)
    out = torch.empty((nb, cell.N), dtype=dtype, device="cuda")
    step = max(1, (1 << 26) // cell.N)
    for b in range(0, nb, step):
        x = torch.randn((min(step, nb - b), *_shape(cell)), generator=gen, device="cuda")
        x = torch.fft.irfftn(torch.fft.rfftn(x, dim=(1, 2, 3)) * filt[..., :cell.shape[0] // 2 + 1],
                             s=_shape(cell), dim=(1, 2, 3)).reshape(x.shape[0], -1)
        out[b:b + x.shape[0]] = (x / x.norm(dim=1, keepdim=True)) / cell.dvol ** 0.5
    return out


def _veff(cell, seed, dtype):
    return torch.tensor(S.smooth_veff(cell, seed), dtype=dtype, device="cuda")


class _Ham:
    """H, S and the projectors of a cell in 64 bits by plain torch."""

    def __init__(self, cell, veff):
        self.cell, self.veff = cell, None if veff is None else veff.double()
        self.A, self.P, self.N, self.dv = cell.natom, cell.nprjmx, cell.N, cell.dvol
        v = torch.tensor(cell.vnlocp, dtype=F64, device="cuda")      # [A][P][L]
        lst = torch.tensor(cell.lst, device="cuda").long().view(self.A, -1)
        used = (v != 0).any(1) & (torch.arange(lst.shape[1], device="cuda") <
                                  torch.tensor(cell.natinf, device="cuda")[:, None])
        at, pos = used.nonzero(as_tuple=True)
        self.pt, self.v = lst[at, pos], v[at, :, pos]                # [E], [E][P]
        cnt = torch.bincount(at, minlength=self.A)
        self.Lm = int(cnt.max())
        self.slot = at * self.Lm + torch.arange(len(at), device="cuda") - (cnt.cumsum(0) - cnt)[at]
        self.vp = v.new_zeros((self.A * self.Lm, self.P))
        self.vp[self.slot] = self.v
        self.vp = self.vp.view(self.A, self.Lm, self.P)
        self.ptp = lst.new_zeros(self.A * self.Lm)
        self.ptp[self.slot] = self.pt
        # entries of each covered point, padded with a dummy entry
        order = torch.argsort(self.pt, stable=True)
        self.cov, n = torch.unique_consecutive(self.pt[order], return_counts=True)
        self.tab = lst.new_full((len(self.cov), int(n.max())), self.A * self.Lm)
        row = torch.repeat_interleave(torch.arange(len(n), device="cuda"), n)
        col = torch.arange(len(order), device="cuda") - (n.cumsum(0) - n)[row]
        self.tab[row, col] = self.slot[order]
        t = lambda m: None if m is None else torch.tensor(m, dtype=F64, device="cuda")
        self.D, self.S = t(cell.dij), t(cell.sss)

    def dot(self, x):                                                # <p|x>
        g = x[:, self.ptp].double().view(-1, self.A, self.Lm)
        return torch.einsum("bal,alp->bap", g, self.vp)

    def add(self, out, mat, rp):
        """out += sum_a p_a (mat_a rp_a) / dV"""
        t = torch.einsum("bap,aqp->baq", rp, mat) / self.dv
        c = torch.einsum("bap,alp->bal", t, self.vp).reshape(len(rp), -1)
        c = torch.cat([c, c.new_zeros((len(rp), 1))], 1)
        out[:, self.cov] += c[:, self.tab].sum(-1)
        return out

    def lap(self, x):
        x = x.view(-1, *_shape(self.cell))
        out = x * self.veff.view(_shape(self.cell))
        for ax in range(3):
            w = [-0.5 * c / self.cell.h[ax] ** 2 for c in FD]
            out += w[0] * x
            for m in range(1, 5):
                out += w[m] * (x.roll(m, 3 - ax) + x.roll(-m, 3 - ax))
        return out.view(-1, self.N)

    def h(self, x, rp):
        return self.add(self.lap(x), self.D, rp)

    def s(self, x, rp):
        return x.clone() if self.S is None else self.add(x.clone(), self.S, rp)

    def precond(self, x):
        g = x.view(-1, *_shape(self.cell))
        out = 0.5 * g
        for ax in (1, 2, 3):
            out += (g.roll(1, ax) + g.roll(-1, ax)) / 12
        return out.view(-1, self.N)

    def block(self):
        return max(1, (1 << 27) // max(self.N, self.A * self.Lm))

    def apply(self, what, x, *r):
        """what() over blocks of bands"""
        out, n = [], self.block()
        for b in range(0, len(x), n):
            out.append(what(x[b:b + n].double(), *[v[b:b + n] for v in r]))
        return torch.cat(out)


def _upper(m):
    """L^-T of the Cholesky factor of m (64 bits)"""
    return torch.linalg.solve_triangular(torch.linalg.cholesky(m),
                                         torch.eye(len(m), dtype=F64, device="cuda"),
                                         upper=False).T


def _pieces(n):
    return range(0, n, 1 << 17)


def _rotate(x, z):
    """x <- z^T x over pieces of the grid, in place"""
    for p in _pieces(x.shape[1]):
        x[:, p:p + (1 << 17)] = (z.T @ x[:, p:p + (1 << 17)].double()).to(x.dtype)


def _gram(x, y):
    return sum(x[:, p:p + (1 << 17)].double() @ y[:, p:p + (1 << 17)].double().T
               for p in _pieces(x.shape[1]))


def _orthonormal(ham, psi):
    """S-orthonormal psi (in place, by columns of L^-T) and its <p|psi> in 64 bits."""
    rp = ham.apply(ham.dot, psi)
    g = _gram(psi, psi) * ham.dv
    if ham.S is not None:
        g += torch.einsum("bap,apq,caq->bc", rp, ham.S, rp)
    w = _upper(g)
    _rotate(psi, w)
    return torch.einsum("bap,bc->cap", rp, w)


def _bands(cell, case, seed):
    """The library's band state as the solvers meet it, and what it was made of."""
    dtype = F64 if case["f64"] else F32
    ham = _Ham(cell, None)
    psi = _noise(cell, case["bands"], seed, dtype)
    rp = _orthonormal(ham, psi)
    b = K.Bands(K.Geometry(cell), psi, ham.S)
    if ham.S is not None:
        n = ham.block()
        for k in range(0, len(psi), n):
            b.spsi[k:k + n] = ham.s(psi[k:k + n].double(), rp[k:k + n]).to(dtype)
    b.rp.copy_(rp)
    return b


# --------------------------------------------------------------------- a pass
def prepare(case, seed):
    kind = case["kind"]
    st = {"case": case}
    if kind == "syev":
        a = torch.randn((case["n"], case["n"]), generator=_gen(seed), device="cuda", dtype=F64)
        # the subspace Hamiltonian of bands that still move: levels over about 1 Ha
        st["a"] = torch.diag(torch.linspace(-0.3, 0.7, case["n"], dtype=F64, device="cuda")) + \
            (a + a.T) * (0.05 / case["n"] ** 0.5)
        return st
    if kind == "hartree":
        st["shape"] = (case["nx"], case["ny"], case["nz"])
        st["xmax"] = tuple(case["n" + ax] * case["h"] / 2 for ax in "xyz")
        st["rho"] = _gaussians(case, seed)
        st["vh"] = torch.zeros_like(st["rho"])
        return st
    if kind == "batch":
        cells = S.small_cell_set(case["cells"], 2, case["spacing"])
        st["geoms"] = [K.Geometry(c) for c in cells]
        st["psi"] = [_noise(c, case["bands"], seed + k, F32) for k, c in enumerate(cells)]
        st["rp"] = [_Ham(c, None).dot(p).contiguous() for c, p in zip(cells, st["psi"])]
        st["veff"] = [_veff(c, seed + k, F32) for k, c in enumerate(cells)]
        st["dij"] = [torch.tensor(c.dij, dtype=F64, device="cuda") for c in cells]
        st["out"] = [torch.empty_like(p) for p in st["psi"]]
        st["plan"] = K.HpsiBatch(st["geoms"], [case["bands"]] * case["cells"])
        st["plan"].set(st["veff"], st["dij"], st["rp"], st["psi"], st["out"])
        return st
    cell = _host_cell(case, seed)
    dtype = F64 if case["f64"] else F32
    st["dij"] = torch.tensor(cell.dij, dtype=F64, device="cuda")
    if kind == "hpsi":
        st["g"] = K.Geometry(cell)
        st["psi"] = _noise(cell, case["bands"], seed, dtype)
        ham = _Ham(cell, None)
        st["rp"] = ham.apply(ham.dot, st["psi"])
        st["out"] = torch.empty_like(st["psi"])
        st["veff"] = _veff(cell, seed, dtype)
    elif kind == "forces":
        st["cell"] = cell
        st["psi"] = _noise(cell, case["bands"], seed, dtype)
        st["sss"] = None if cell.sss is None else torch.tensor(cell.sss, dtype=F64, device="cuda")
        st["sval"], st["occ"] = _levels(case)
    else:
        st["b"] = _bands(cell, case, seed)
        st["veff"] = _veff(cell, seed, dtype)
        if kind == "scf":
            b = st["b"]
            st["start"] = [(x, x.clone()) for x in {id(t): t for t in (b.psi, b.spsi, b.rp)}.values()]
            st["prm"] = L.solver_prm() if case["cg"] else L.solver_prm(ncgscf=3)
    return st


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "hpsi":
        return K.hpsi(st["g"], st["veff"], st["dij"], st["rp"], st["psi"], out=st["out"])
    if kind == "batch":
        st["plan"].run()
        return st["out"]
    if kind == "syev":
        w, z, _ = K.syev(st["a"])
        return w, z
    if kind == "hartree":
        st["vh"].zero_()
        K.scf_hartree(st["shape"], 4, st["xmax"], st["rho"], st["vh"], mixed=not case["f64"])
        return st["vh"]
    if kind == "forces":
        return F.projector_forces(st["cell"], st["psi"], st["sval"], st["occ"], st["dij"],
                                  st["sss"])
    b = st["b"]
    if kind == "diis":
        # each pass updates the bands further, as one SCF iteration after another does
        K.ksdiis(b, st["veff"], st["dij"])
        return {"psi": b.psi, "spsi": b.spsi, "hpsi": b.hpsi, "rp": b.rp, "sval": b.sval,
                "resid": b.resid}
    for x, x0 in st["start"]:   # the iteration's start bands (a small part of the pass)
        x.copy_(x0)
    b.resid[:] = 0.0
    K.scf_diag(b, st["veff"], st["dij"], 5, st["prm"])
    return {"psi": b.psi, "spsi": b.spsi, "rp": b.rp, "sval": b.sval, "resid": b.resid}


# ------------------------------------------------------------- floors, tolerances
def _entries(case):
    """Nonzero projector list entries of a cell, from the sphere's volume."""
    ds = S.load_dataset(case["species"])
    h3 = 1.0
    for ax in "xyz":
        h3 *= EDGE[case["species"]] * case["c" + ax] / case["n" + ax]
    atoms = 8 * case["cx"] * case["cy"] * case["cz"]
    return atoms * 4.18879 * ds["rcut"] ** 3 / h3, atoms, len(S.projector_layout(ds))


def work(case):
    kind = case["kind"]
    if kind == "syev":
        n = case["n"]
        return {"bytes": 8.0 * (2 * n * n + n), "flops": 9.0 * n ** 3}
    if kind == "hartree":
        # A p, two dot products and three vector updates an iteration; about one
        # iteration per grid point along the longest axis and a tenth of precision
        n = case["nx"] * case["ny"] * case["nz"]
        it = 2.0 * max(case["nx"], case["ny"], case["nz"])
        return {"bytes": 16.0 * n, "flops": it * n * 60.0}
    if kind == "batch":
        n = case["cells"] * 0.5 * ((10.26 / case["spacing"]) ** 3 + (6.74 / case["spacing"]) ** 3)
        return {"bytes": 8.0 * n * case["bands"] + 4.0 * n, "flops": 60.0 * n * case["bands"]}
    n, m = float(case["nx"] * case["ny"] * case["nz"]), case["bands"]
    ent, atoms, P = _entries(case)
    s = 8.0 if case["f64"] else 4.0
    sep = case["species"] == "si_paw"
    h_flops = 50.0 * n * m + 2.0 * ent * P * m
    if kind == "hpsi":
        return {"bytes": 2 * s * n * m + s * n + ent * (P * s + 4) + 8.0 * m * atoms * P,
                "flops": h_flops}
    if kind == "forces":
        return {"bytes": s * n * m, "flops": 8.0 * ent * P * m}
    arrays = 3.0 if sep else 2.0
    if kind == "scf" and case["cg"]:
        # per band at most four iterations: H twice in all, S, three orthogonalisations
        it = 4.0
        return {"bytes": 2 * arrays * s * n * m,
                "flops": 2.0 * n * m * m + 6.0 * n * m * m +
                it * (2.0 * h_flops + 3 * 4.0 * n * m * m / 2 + 40.0 * n * m)}
    gram, rot = float(n * m * m), 2.0 * n * m * m
    diis = 3 * (2.0 * h_flops + 60.0 * n * m) + gram + rot / 2 + h_flops
    if kind == "diis":
        return {"bytes": 2 * arrays * s * n * m, "flops": diis}
    return {"bytes": 2 * arrays * s * n * m, "flops": diis + h_flops + gram + rot + 9.0 * m ** 3}


def tolerance(case):
    kind = case["kind"]
    # eigenvectors carry the rounding of the matrix over the level spacing, so
    # the cases that return them allow a few hundred times the rounding seen
    # (3e-12 and 3e-6 at 160 bands); the others about four times the error seen
    # against 64 bits (4e-7 H psi, 5e-6 H psi of updated bands, 1e-6 potential)
    if kind == "syev":
        return {"rel": 1e-9, "max": 1e-6}
    if kind == "hartree":
        return {"rel": 1e-11} if case["f64"] else {"rel": 4e-6}
    if kind == "scf":
        return {"rel": 1e-9, "max": 1e-6} if case["f64"] else {"rel": 3e-4, "max": 3e-2}
    if kind == "diis":
        return {"rel": 1e-10} if case["f64"] else {"rel": 2e-5, "max": 1e-2}
    if kind == "forces":
        return {"rel": 1e-10} if case["f64"] else {"rel": 1e-9}
    return {"rel": 1e-12} if case.get("f64") else {"rel": 2e-6, "max": 1e-4}


# ------------------------------------------------------------------ in 64 bits
def _gaussians(case, seed):
    """Charge density of normalised Gaussians (sigma 1 bohr, 4 electrons each)."""
    rng = np.random.default_rng(seed)
    d = [torch.arange(case["n" + ax], device="cuda", dtype=F64) * case["h"] for ax in "xyz"]
    edge = [len(x) * case["h"] for x in d]
    rho = torch.zeros((case["nz"], case["ny"], case["nx"]), dtype=F64, device="cuda")
    for c in rng.uniform(0, edge, (case["atoms"], 3)):
        e = [torch.exp(-0.5 * (torch.remainder(x - float(v) + A / 2, A) - A / 2) ** 2)
             for x, v, A in zip(d, c, edge)]
        rho += e[2][:, None, None] * e[1][:, None] * e[0]
    return (rho * (4.0 / (2 * np.pi) ** 1.5)).reshape(-1)


def _levels(case):
    m = case["bands"]
    return np.linspace(-0.2, 0.4, m), np.where(np.arange(m) < 0.8 * m, 2.0, 0.0)


def _positive(z):
    """eigenvectors (columns) with their largest component positive"""
    top = z.gather(-2, z.abs().argmax(-2, keepdim=True))
    return z * torch.where(top < 0, -1.0, 1.0)


def _dots(x, y, dv):
    return (x * y).sum(-1) * dv


def _diis(ham, ps, ss, rp, prm):
    """RMM-DIIS sweeps of a block of bands"""
    dv, c2 = ham.dv, lambda v: v[:, None]
    for _ in range(prm.ndiismax - 1):
        hs = ham.h(ps, rp)
        val = _dots(ps, hs, dv)
        r0 = hs - c2(val) * ss
        rv = ham.precond(r0)
        rq = ham.dot(rv)
        av, asv = ham.h(rv, rq), ham.s(rv, rq)
        a1 = prm.alambda_diis
        p1 = ps + a1 * rv
        slope = 2.0 * (_dots(rv, hs, dv) - val * _dots(rv, ss, dv))
        ray = _dots(p1, hs + a1 * av, dv) / _dots(p1, ss + a1 * asv, dv)
        lam = 0.5 * slope / ((ray - val - slope * a1) / a1 ** 2)
        lam = lam.clamp(max=prm.alambda_max).clamp(min=prm.alambda_min)
        p1, h1, s1 = ps + c2(lam) * rv, hs + c2(lam) * av, ss + c2(lam) * asv
        r1 = h1 - c2(val) * s1
        t = 1.0 / _dots(p1, s1, dv).sqrt()
        one = torch.ones_like(t)
        m = lambda a, b, c: torch.stack([a, b * t, b * t, c * t * t], -1).view(-1, 2, 2)
        rs = m(_dots(ps, ss, dv), _dots(ps, s1, dv), one / (t * t))
        rr = m(_dots(r0, r0, dv), _dots(r0, r1, dv), _dots(r1, r1, dv))
        w, z = torch.linalg.eigh(rs)
        vec = _positive(z).flip(-1) / w.flip(-1).clamp(min=1e-300).sqrt()[:, None, :]
        w2, z2 = torch.linalg.eigh(vec.mT @ rr @ vec)
        c = (vec @ _positive(z2)[..., :1])[..., 0]
        c = c / torch.einsum("bi,bij,bj->b", c, rs, c).sqrt()[:, None]
        a, b = c[:, 0], c[:, 1] * t
        mix = lambda y, y1: c2(a) * y + c2(b) * y1
        ps, ss = mix(ps, p1), mix(ss, s1)
        rp = a[:, None, None] * rp + b[:, None, None] * (rp + lam[:, None, None] * rq)
    return ps, ss, rp, val, w2[:, 0]


def _cg(ham, psi, spsi, rp, prm):
    """band-by-band preconditioned CG; psi, spsi, rp are updated in place"""
    dv, M = ham.dv, len(psi)
    sval, resid = torch.zeros(M, dtype=F64), torch.zeros(M, dtype=F64)
    sep = ham.S is not None
    for l in range(M):
        c = (spsi[:l] @ psi[l]) * dv
        psi[l] -= c @ psi[:l]
        if sep:
            spsi[l] -= c @ spsi[:l]
        rp[l] -= torch.einsum("j,jap->ap", c, rp[:l])
        t = _dots(psi[l], spsi[l], dv).rsqrt()
        for x in ([psi, spsi, rp] if sep else [psi, rp]):
            x[l] *= t
        h = ham.h(psi[l:l + 1], rp[l:l + 1])[0]
        r2, pv, spv, rpp = 1.0, 0.0, 0.0, 0.0
        for _ in range(prm.nsdmax):
            r1, val = r2, _dots(psi[l], h, dv)
            rvec = -(h - val * spsi[l])
            rv = ham.precond(rvec[None])[0]
            rv = rv - ((spsi[:l + 1] @ rv) * dv) @ psi[:l + 1]
            rq = ham.dot(rv[None])
            asv = ham.s(rv[None], rq)[0]
            r2 = _dots(rv, rvec, dv)
            pv, spv, rpp = rv + (r2 / r1) * pv, asv + (r2 / r1) * spv, rq[0] + (r2 / r1) * rpp
            c = (spsi[:l + 1] @ pv) * dv
            p, a = pv - c @ psi[:l + 1], (spv if sep else pv) - c @ spsi[:l + 1]
            q = rpp - torch.einsum("j,jap->ap", c, rp[:l + 1])
            t = _dots(a, p, dv).rsqrt()
            p, a, q = p * t, a * t, q * t
            av = ham.h(p[None], q[None])[0]
            pap, sap = float(_dots(p, av, dv)), float(_dots(psi[l], av, dv))
            v = float(val)
            gamma = (v + pap) / 2 - ((v - pap) ** 2 / 4 + sap ** 2) ** 0.5
            al, be = 1.0, 0.0
            if abs((v - gamma) / gamma) > 1e-14:
                den = (sap ** 2 + (v - gamma) ** 2) ** 0.5
                al, be = sap / den, -(v - gamma) / den
            if al < 1e-14:
                al, be = -al, -be
            psi[l], h = al * psi[l] + be * p, al * h + be * av
            if sep:
                spsi[l] = al * spsi[l] + be * a
            rp[l] = al * rp[l] + be * q
            sval[l], resid[l] = v, float(r2)
            if float(r2) ** 0.5 < prm.epssd:
                break
    return sval, resid


def _exact_bands(case, seed):
    cell = _host_cell(case, seed)
    dtype = F64 if case["f64"] else F32
    ham = _Ham(cell, _veff(cell, seed, dtype))
    psi = _noise(cell, case["bands"], seed, dtype)
    rp = _orthonormal(ham, psi)
    spsi = ham.apply(lambda x, r: ham.s(x, r).to(dtype), psi, rp) if ham.S is not None else None
    prm = L.solver_prm() if case.get("cg") else L.solver_prm(ncgscf=3)
    if case["kind"] == "scf":
        psi = psi.double()
        spsi = psi if spsi is None else spsi.double()
        a = _gram(psi, ham.apply(ham.h, psi, rp)) * ham.dv
        a = a.tril() + a.tril(-1).T
        sval, z = torch.linalg.eigh(a)
        z = _positive(z)
        for x in {id(x): x for x in (psi, spsi)}.values():
            _rotate(x, z)
        rp = torch.einsum("bap,bc->cap", rp, z)
        if case["cg"]:
            sval, resid = _cg(ham, psi, spsi, rp, prm)
            return _sorted(psi, spsi, rp, sval.cuda(), resid.cuda())
    got = {k: [] for k in ("psi", "rp", "sval", "resid")}
    n = max(1, ham.block() // 4)
    for b in range(0, len(psi), n):
        p = psi[b:b + n].double()
        s = p if spsi is None else spsi[b:b + n].double()
        p, s, r, val, res = _diis(ham, p, s, rp[b:b + n], prm)
        for k, x in zip(got, (p, r, val, res)):
            got[k].append(x)
    del psi, spsi
    psi, sval, resid = (torch.cat(got.pop(k)) for k in ("psi", "sval", "resid"))
    rp = _orthonormal(ham, psi)
    spsi = psi if ham.S is None else ham.apply(ham.s, psi, rp)
    if case["kind"] == "scf":
        return _sorted(psi, spsi, rp, sval, resid)
    return {"psi": psi, "spsi": spsi, "hpsi": ham.apply(ham.h, psi, rp), "rp": rp, "sval": sval,
            "resid": resid}


def _sorted(psi, spsi, rp, sval, resid):
    o = torch.argsort(sval, stable=True)
    return {"psi": psi[o], "spsi": spsi[o], "rp": rp[o], "sval": sval[o], "resid": resid[o]}


def _exact_forces(case, seed):
    cell = _host_cell(case, seed)
    psi = _noise(cell, case["bands"], seed, F64 if case["f64"] else F32)
    sval, occ = (torch.tensor(x, device="cuda") for x in _levels(case))
    ds, A = cell.ds, cell.natom
    lay = S.projector_layout(ds)
    t = lambda a: torch.tensor(np.ascontiguousarray(a), device="cuda", dtype=F64)
    D, Sm = t(cell.dij), None if cell.sss is None else t(cell.sss)
    ln = cell.num_list
    force = torch.zeros((A, 3), dtype=F64, device="cuda")
    for a in range(A):
        n = int(cell.natinf[a])
        pt = torch.tensor(cell.lst.reshape(A, ln)[a, :n], device="cuda").long()
        x = [t(cell.lstxyz[k].reshape(A, ln)[a, :n]) * cell.h[k] -
             (cell.atoms[a, k] - (cell.natxyz[k][a] * cell.h[k] - 0.5 * cell.h[k]))
             for k in range(3)]
        r2 = x[0] ** 2 + x[1] ** 2 + x[2] ** 2
        r = r2.sqrt()
        inside = (r < ds["rcut"]).to(F64) * cell.dvol
        rin = torch.where(r > 1e-12, 1.0 / r, torch.zeros_like(r))
        val, grad = [], []
        for ci, l, m in lay:
            tab = t(ds["channels"][ci]["p"])
            j = (r / ds["dr"]).long().clamp(max=len(tab) - 2)
            dp = (tab[j + 1] - tab[j]) / ds["dr"]
            dp = torch.where(r >= (len(tab) - 1) * ds["dr"], 0.0, dp)   # constant past the table
            p = torch.where(dp == 0.0, tab[j + 1], tab[j] + dp * (r - j.to(F64) * ds["dr"]))
            c, poly, d = _harmonic(l, m, x, r2)
            y = c * poly * rin ** l
            val.append(p * y * inside)
            grad.append(torch.stack([(dp * rin * x[k] * y + p * (c * d[k] * rin ** l - l * c * poly *
                                      rin ** (l + 2) * x[k])) * inside for k in range(3)]))
        band = psi[:, pt].double()
        rp = band @ torch.stack(val).T                                  # [b][P]
        g = torch.einsum("bn,pkn->bkp", band, torch.stack(grad))        # [b][3][P]
        M = D[a][None] if Sm is None else D[a][None] - sval[:, None, None] * Sm[a][None]
        force[a] = 2.0 * torch.einsum("b,bi,bij,bkj->k", occ, rp, M.expand(len(occ), -1, -1), g)
    return force


def _harmonic(l, m, x, r2):
    """real harmonics: constant, polynomial and its gradient as the path takes it"""
    X, Y, Z = x
    o, e = torch.zeros_like(X), torch.ones_like(X)
    pi = np.pi
    if l == 0:
        return (1 / 4 / pi) ** 0.5, e, (o, o, o)
    if l == 1:
        return (3 / 4 / pi) ** 0.5, x[m], tuple(e if k == m else o for k in range(3))
    c = (15 / 4 / pi) ** 0.5
    return [((15 / 16 / pi) ** 0.5, X * X - Y * Y, (2 * X, -2 * Y, o)),
            (c, -Z * X, (-Z, o, -X)),
            ((5 / 16 / pi) ** 0.5, 3 * Z * Z - r2, (-2 * X, -2 * Y, 4 * Z)),
            (c, -Y * Z, (o, -Z, -Y)),
            (c, X * Y, (Y, X, o))][m]


def exact(case, seed):
    kind = case["kind"]
    if kind == "syev":
        w, z = torch.linalg.eigh(prepare(case, seed)["a"])
        return w, _positive(z)
    if kind == "hartree":
        rho = _gaussians(case, seed).view(case["nz"], case["ny"], case["nx"])
        k = []
        for n in rho.shape:
            th = 2 * np.pi * torch.arange(n, device="cuda", dtype=F64) / n
            k.append(sum((FD[m] if m == 0 else 2 * FD[m]) * torch.cos(m * th) for m in range(5)) *
                     (-0.5 / case["h"] ** 2))
        lam = k[0][:, None, None] + k[1][:, None] + k[2]
        lam[0, 0, 0] = 1.0
        q = torch.fft.fftn(2 * np.pi * rho) / lam
        q[0, 0, 0] = 0.0
        return torch.fft.ifftn(q).real.reshape(-1)
    if kind == "forces":
        return _exact_forces(case, seed)
    if kind == "batch":
        out = []
        for k, c in enumerate(S.small_cell_set(case["cells"], 2, case["spacing"])):
            ham = _Ham(c, _veff(c, seed + k, F32))
            p = _noise(c, case["bands"], seed + k, F32)
            out.append(ham.h(p.double(), ham.dot(p)))
        return out
    if kind == "hpsi":
        cell = _host_cell(case, seed)
        dtype = F64 if case["f64"] else F32
        ham = _Ham(cell, _veff(cell, seed, dtype))
        psi = _noise(cell, case["bands"], seed, dtype)
        return ham.apply(ham.h, psi, ham.apply(ham.dot, psi))
    return _exact_bands(case, seed)
