"""Timed workloads of the SCFT engine, through its Python entry points.

Five kinds of work cover what a PSCF user has the engine do:

  density   Engine.density + scf_stress + free_energy with host fields: the
            drop-in for the density / scf_stress / free_energy routines that a
            host-side iterator calls once per iteration
  device    Engine.density_device + scf_stress with fields on the GPU
  solve     Engine.iterate_am: a short Anderson solve (the first iterations
            from a starting field), optionally with an imposed space group
            and cell relaxation
  columns   Engine.density_basis: one density per column of a Newton
            Jacobian, fields as star coefficients differing by 1e-8
  gradient  autograd.density: loss of the density and its exact gradient

on lamellar (1-D), hexagonal and rectangular (2-D), cubic and orthorhombic
(3-D) cells, from 64 points to 64 x 128 x 224.  The extents are products of
2, 3, 5 and 7, even and odd, powers of two and others.
"""
import itertools
import math

import numpy as np
import torch

from pscf_b200 import autograd
from pscf_b200.basis import StarBasis
from pscf_b200.engine import FP32, FP64, Engine
from pscf_b200.system import Chain, Solvent, System

LATTICES = {
    "lamellar": (1, "lamellar"), "hexagonal": (2, "hexagonal"), "rectangular": (2, "rectangular"),
    "cubic": (3, "cubic"), "orthorhombic": (3, "orthorhombic"),
}
CHEMISTRIES = ("diblock", "triblock", "blend")


def _case(name, kind, lattice, n, count=1, chem="diblock", f=0.3, ds=0.01, precision="fp64", group="", relax=False,
          iterations=0):
    n = list(n) + [1] * (3 - len(n))
    return {"name": name, "kind": kind, "lattice": lattice, "n1": n[0], "n2": n[1], "n3": n[2], "count": count,
            "chem": chem, "f": f, "ds": ds, "precision": precision, "group": group, "relax": relax,
            "iterations": iterations}


def listed():
    return [
        # one lamella: the smallest call, a host iterator's step on a 1-D profile
        _case("lamellar_64", "density", "lamellar", [64], f=0.5),
        # a chi sweep of lamellae solved together
        _case("solve_lamellar_64_x96", "solve", "lamellar", [64], 96, f=0.4, group="-1", iterations=4),
        # one hexagonal cylinder phase
        _case("hexagonal_64", "density", "hexagonal", [64, 64]),
        # a chi sweep of cylinders solved together
        _case("solve_hexagonal_64_x96", "solve", "hexagonal", [64, 64], 96, group="p 6 m m", iterations=2),
        # triblock on a rectangular cell whose extents are no powers of two
        _case("rectangular_48x40_x6", "density", "rectangular", [48, 40], 6, "triblock"),
        # Newton Jacobian columns of the BCC phase on a 20^3 grid
        _case("columns_bcc_20_x32", "columns", "cubic", [20, 20, 20], 32, group="I m -3 m", ds=0.02),
        # one BCC instance solved with its space group and a relaxing cell
        _case("solve_bcc_32", "solve", "cubic", [32, 32, 32], 1, f=0.25, group="I m -3 m", relax=True, iterations=4),
        # a batch of BCC instances, the throughput workload
        _case("bcc_32_x64", "device", "cubic", [32, 32, 32], 64, f=0.25),
        # polymer and solvent on an orthorhombic grid with odd and ragged extents
        _case("orthorhombic_27x40x50", "density", "orthorhombic", [27, 40, 50], 2, "blend"),
        # gradient of a loss of the gyroid's density
        _case("gradient_gyroid_64", "gradient", "cubic", [64, 64, 64], f=0.4, ds=0.005),
        # the large ABC network phase, propagated in FP32
        _case("network_64x128x224_fp32", "device", "orthorhombic", [64, 128, 224], chem="triblock", ds=0.005,
              precision="fp32"),
        # the large ABC network phase solved with its space group, cell relaxed
        _case("solve_network_64x128x224", "solve", "orthorhombic", [64, 128, 224], chem="triblock", ds=0.005,
              group="F d d d : 2", relax=True, iterations=1),
    ]


EXTENTS = [8, 9, 10, 12, 14, 15, 16, 18, 20, 21, 24, 25, 27, 28, 30, 32, 35, 36, 40, 42, 45, 48, 50, 54, 56, 60, 63, 64]


def draw(rng):
    kind = rng.choice(["density", "density", "device", "solve", "columns", "gradient"])
    dim = rng.choice([1, 2, 3, 3])

    def extent(lo, hi, even=False):
        """The allowed extent nearest (in the logarithm) to a log-uniform one."""
        t = math.log(rng.uniform(lo, hi)) if hi < 10 * lo else rng.uniform(math.log(lo), math.log(hi))
        pool = [e for e in EXTENTS if lo <= e <= hi and not (even and e % 2)]
        return min(pool, key=lambda e: abs(math.log(e) - t))

    f, ds = rng.choice([0.2, 0.25, 0.3, 0.35, 0.4, 0.45, 0.5]), rng.choice([0.005, 0.01, 0.02])
    chem = rng.choice(CHEMISTRIES) if kind in ("density", "device") else "diblock"
    group, relax, iterations, precision = "", False, 0, "fp64"
    if kind == "device" and rng.random() < 0.4:
        precision = "fp32"
    if dim == 1:
        lattice, n = "lamellar", [extent(16, 64)]
        group = "-1"
    elif dim == 2:
        # (odd first extents up to 45: the stress of a larger plane is refused)
        if rng.random() < 0.5:
            m = extent(16, 64)
            m = 60 if m == 63 else m
            lattice, n, group = "hexagonal", [m, m], "p 6 m m"
        else:
            m = extent(16, 64)
            lattice, n = "rectangular", [60 if m == 63 else m, extent(16, 64)]
    elif rng.random() < 0.6:
        m = extent(12, 32 if kind == "columns" else 64, kind in ("columns", "solve"))
        lattice, n, group = "cubic", [m, m, m], "I m -3 m"
    else:
        lattice, n = "orthorhombic", [extent(12, 64), extent(12, 64), extent(12, 64)]
    if kind == "columns" and not group:
        kind = "density"
    if kind in ("solve", "columns"):
        iterations = rng.choice([1, 2, 3]) if kind == "solve" else 0
        relax = kind == "solve" and rng.random() < 0.3
    else:
        group = ""
    points = math.prod(n)
    most = {1: 96, 2: 96, 3: max(1, min(64, (1 << 20) // points))}[dim]
    if kind == "gradient":
        most = min(most, 4)
    if kind == "solve" and dim == 3:
        most = min(most, 8)
    count = int(round(math.exp(rng.uniform(0.0, math.log(most)))))
    c = _case("", kind, lattice, n, count, chem, f, ds, precision, group, relax, iterations)
    del c["name"]
    return c


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
def _grid(case):
    dim = LATTICES[case["lattice"]][0]
    return [case["n1"], case["n2"], case["n3"]][:dim]


def _systems(case):
    """One System per instance: same chain, chi and cell spread over the batch."""
    dim, crystal = LATTICES[case["lattice"]]
    n, f, out = _grid(case), case["f"], []
    for i in range(case["count"]):
        u = i / max(case["count"] - 1, 1)
        x = 14.0 + 6.0 * u                                   # chi N of the A-B pair
        scale = (x / 20.0) ** (1.0 / 6.0)                    # strong-segregation cell scaling
        cell = {"lamellar": [1.7], "hexagonal": [1.9], "rectangular": [1.9, 1.9 * n[-1] / n[0]],
                "cubic": [3.7 if case["kind"] == "gradient" else 1.95],
                "orthorhombic": [4.0, 4.0 * n[min(1, dim - 1)] / n[0], 4.0 * n[-1] / n[0]]}[case["lattice"]]
        cell = [c * scale for c in cell]
        if case["chem"] == "triblock":
            chi = [[0.0, x, 2 * x], [x, 0.0, x], [2 * x, x, 0.0]]
            s = System(dim, n, crystal, cell, [1.0, 1.0, 1.0], chi, [Chain([0, 1, 2], [0.3, 0.4, 0.3])], case["ds"])
        elif case["chem"] == "blend":
            chi = [[0.0, x, 4.0], [x, 0.0, 3.0], [4.0, 3.0, 0.0]]
            s = System(dim, n, crystal, cell, [1.0, 1.1, 1.0], chi,
                       [Chain([0, 1], [f, 1.0 - f], phi=0.7), Chain([0], [0.3], phi=0.2)], case["ds"],
                       solvents=[Solvent(2, 0.1, phi=0.1)])
        else:
            s = System(dim, n, crystal, cell, [1.0, 1.0], [[0.0, x], [x, 0.0]], [Chain([0, 1], [f, 1.0 - f])],
                       case["ds"])
        out.append(s)
    return out


def _profile(case):
    """The phase's first-star function on the grid, scaled to [-1, 1]."""
    n = _grid(case) + [1] * (3 - len(_grid(case)))
    z, y, x = np.meshgrid(*(2 * np.pi * np.arange(m) / m for m in (n[2], n[1], n[0])), indexing="ij")
    if case["lattice"] == "lamellar":
        g = np.cos(x)
    elif case["lattice"] == "hexagonal":
        g = np.cos(x) + np.cos(y) + np.cos(x - y)
    elif case["lattice"] == "rectangular":
        g = np.cos(x) * np.cos(y) + 0.3 * np.cos(2 * y)
    elif case["kind"] == "gradient":                         # gyroid
        g = np.sin(x) * np.cos(y) + np.sin(y) * np.cos(z) + np.sin(z) * np.cos(x)
    elif case["lattice"] == "cubic":                         # spheres at the BCC sites
        g = np.cos(x) * np.cos(y) + np.cos(y) * np.cos(z) + np.cos(z) * np.cos(x)
    else:                                                    # network
        g = np.cos(x) * np.cos(y) * np.cos(z) + 0.5 * np.sin(x) * np.sin(2 * y)
    return (g / np.abs(g).max()).ravel()


def _contour(lengths, ds):
    """First slice of each block and the end, and each block's step: an even
    number of steps nearest to the block's length, at least two."""
    bgn, bds = [0], []
    for L in lengths:
        pairs = max(int(L / ds / 2.0 + 0.5), 1)
        bds.append(L / pairs / 2.0)
        bgn.append(bgn[-1] + 2 * pairs)
    return bgn, bds


def _fields(case, systems, seed):
    """omega [count][n_monomer][nr]: the uniform values, the phase's profile
    with sharpened edges, and N(0, 0.01) noise per instance and monomer."""
    rng = np.random.default_rng(seed)
    g = np.tanh(2.0 * _profile(case))
    g -= g.mean()
    sign = [-1.0, 1.0, -0.5]
    w = rng.standard_normal((case["count"], systems[0].n_monomer, g.size)) * 0.01
    for i, s in enumerate(systems):
        amp = 0.4 * s.chi[0, 1] * (1.0 + 0.05 * rng.standard_normal())
        w0 = s.omega_uniform()
        for a in range(s.n_monomer):
            w[i, a] += w0[a] + sign[a] * amp * g
    return w


def _target(case, systems, seed):
    """Target A density of the gradient's loss: a seeded smooth field around f."""
    rng = np.random.default_rng(seed + 1)
    g = _profile(case)
    t = case["f"] + 0.1 * g[None, :] * (1.0 + 0.2 * rng.standard_normal((case["count"], 1)))
    return torch.from_numpy(t).cuda()


_BASES = {}


def _basis(case):
    key = (case["group"], tuple(_grid(case)))
    if key not in _BASES:
        _BASES[key] = StarBasis(case["group"], _grid(case))
    return _BASES[key]


def _columns(case, systems, seed):
    """Star coefficients [count][n_monomer][n_star]: one state, and one
    coefficient of it raised by 1e-8 per column (column 0 is the state)."""
    one = dict(case, count=1)
    w = _fields(one, systems[:1], seed)[0]
    b = _basis(case)
    base = np.stack([b.to_basis(x) for x in w])
    out = np.repeat(base[None], case["count"], axis=0)
    for j in range(1, case["count"]):
        out[j, (j - 1) % 2, 1 + (j - 1) // 2 % (b.n_star - 1)] += 1e-8
    return out


def prepare(case, seed):
    kind = case["kind"]
    systems = _systems(case)
    if kind == "columns":
        systems = [systems[0]] * case["count"]
    e = Engine(systems, FP32 if case["precision"] == "fp32" else FP64)
    st = {"case": case, "engine": e, "cells": [list(s.cell_param) for s in systems]}
    if kind == "columns":
        for i in range(case["count"]):
            e.set_basis(i, _basis(case))
        st["omega"] = list(_columns(case, systems, seed))
        return st
    w = _fields(case, systems, seed)
    if kind == "solve" and case["group"]:
        for i in range(case["count"]):
            e.set_symmetry(i, case["group"])
    if kind in ("device", "gradient"):
        st["omega"] = torch.from_numpy(w).cuda()
    else:
        st["omega"] = w
    if kind == "device":
        st["rho"] = torch.empty_like(st["omega"])
    if kind == "gradient":
        st["target"] = _target(case, systems, seed)
    return st


def run(st):
    case, e = st["case"], st["engine"]
    kind, nch = case["kind"], len(e.systems[0].chains)
    if kind == "density":
        rho, q = e.density(st["omega"])
        stress = e.scf_stress()
        f, p, mu = e.free_energy()
        out = {"rho": rho, "q": q[:, :nch], "stress": stress, "f": f, "pressure": p, "mu": mu[:, :nch]}
        if e.systems[0].solvents:
            out["q_solvent"] = e.q_solvent[:, :len(e.systems[0].solvents)].copy()
        return out
    if kind == "device":
        q = e.density_device(st["omega"].data_ptr(), st["rho"].data_ptr())
        stress = e.scf_stress()
        if case["precision"] == "fp32":   # kept in the precision of the propagation
            return {"rho": st["rho"].float(), "q": q[:, :nch].astype(np.float32), "stress": stress.astype(np.float32)}
        return {"rho": st["rho"], "q": q[:, :nch], "stress": stress}
    if kind == "columns":
        rho, q = e.density_basis(st["omega"])
        return {"rho": np.stack(rho), "q": q[:, :nch]}
    if kind == "gradient":
        omega = st["omega"].detach().requires_grad_(True)
        rho, lnq = autograd.density(omega, e)
        loss = (rho[:, 0] - st["target"]).square().sum() / rho.shape[2] + 0.1 * lnq.sum()
        loss.backward()
        return {"rho": rho.detach(), "lnq": lnq.detach(), "loss": loss.detach(), "grad": omega.grad}
    if case["relax"]:
        for i, c in enumerate(st["cells"]):
            e.set_cell_param(i, c)
    w, rho, res = e.iterate_am(st["omega"], error_max=1e-10, max_itr=case["iterations"], domain=case["relax"],
                               mix_max=0.3 if case["chem"] == "triblock" else 0.0)
    return {"omega": w, "rho": rho, "f": np.array([r["f_helmholtz"] for r in res]),
            "q": np.array([r["q"] for r in res]), "cell": np.array([r["cell_param"] for r in res])}


def work(case):
    """Contour steps: q read and written, the block's field read (24 bytes a
    point and step in FP64), six real 3-D transforms; and the fields in and
    out.  A stress adds a read of both propagators and their transforms, a
    density its contour sum's read, a gradient twice a density's steps."""
    s = _systems(dict(case, count=1))[0]
    wq = 4 if case["precision"] == "fp32" else 8
    steps = 2 * sum(_contour(c.block_length, s.ds)[0][-1] for c in s.chains)
    nr = s.nr * case["count"]
    fft = 2.5 * nr * math.log2(s.nr)
    densities = case["iterations"] + 2 if case["kind"] == "solve" else 1
    b = densities * nr * (steps * (2 * wq + 8) + steps * wq)
    f = densities * steps * 6 * fft
    if case["kind"] in ("density", "device") or case["relax"]:
        n = case["iterations"] + 1 if case["kind"] == "solve" else 1
        b += n * steps * nr * wq
        f += n * steps * fft
    if case["kind"] == "gradient":
        b, f = 3 * b, 3 * f
    return {"bytes": b + 16 * nr * s.n_monomer, "flops": f}


# ---------------------------------------------------------------------------
# The same results in 64 bits with torch
# ---------------------------------------------------------------------------
def _reciprocal(lattice, cell):
    """b_i . b_j of the reciprocal vectors and its derivatives in the cell parameters."""
    m = np.zeros((3, 3))
    if lattice == "hexagonal":
        m[:2, :2] = (2 * np.pi / cell[0]) ** 2 * 4.0 / 3.0 * np.array([[1.0, 0.5], [0.5, 1.0]])
        return m, [-2.0 / cell[0] * m]
    axes = [cell[0]] * 3 if lattice == "cubic" else list(cell)
    der = []
    for i, a in enumerate(axes):
        m[i, i] = (2 * np.pi / a) ** 2
        d = np.zeros((3, 3))
        d[i, i] = -2.0 / a * m[i, i]
        der.append(d)
    return m, [sum(der)] if lattice == "cubic" else der


class _Ref:
    """density, stress, free energy and Anderson mixing of a batch with one
    chain layout, fields [count][n_monomer][n3][n2][n1]."""

    def __init__(self, case):
        self.case, self.sys = case, _systems(case)
        if case["kind"] == "columns":
            self.sys = [self.sys[0]] * case["count"]
        s = self.s = self.sys[0]
        self.n, self.nr, self.M = s.n, s.nr, s.n_monomer
        self.axes = (-3, -2, -1)
        self.shape = (s.n[2], s.n[1], s.n[0])
        self.chi = self.dev(np.stack([x.chi for x in self.sys]))
        self.half = s.n[0] // 2 + 1
        wx = np.full(self.half, 2.0)
        wx[0] = 1.0
        if s.n[0] % 2 == 0:
            wx[-1] = 1.0
        self.wx = self.dev(wx)
        self.star = None
        self.ops = _group(case["group"], s.n) if case["group"] and case["kind"] == "solve" else None
        if self.ops:
            self.star = self.star_weights()
        self.set_cells([list(x.cell_param) for x in self.sys])

    @staticmethod
    def dev(a):
        return torch.as_tensor(np.asarray(a, dtype=np.float64)).cuda()

    def set_cells(self, cells):
        """k^2 of each wave's shortest image, and its cell derivatives."""
        self.cells, ks, ds, n, dim = cells, [], [], self.n, self.s.dim
        G0 = np.stack(np.meshgrid(np.arange(n[2]), np.arange(n[1]), np.arange(self.half), indexing="ij"))[::-1]
        if len(set(map(tuple, cells))) == 1:
            cells = cells[:1]
        for cell in cells:
            metric, dGG = _reciprocal(self.case["lattice"], cell)
            best, arg = None, None
            for im in itertools.product(*[(1, 0, -1)] * dim):
                g = np.stack([G0[a] + (im[a] * n[a] if a < dim else 0) for a in range(3)]).astype(float)
                k2 = np.einsum("i...,ij,j...->...", g, metric, g)
                if best is None:
                    best, arg = k2, g
                else:
                    less = k2 < best - 1e-8
                    best, arg = np.where(less, k2, best), np.where(less, g, arg)
            ks.append(best)
            ds.append(np.stack([np.einsum("i...,ij,j...->...", arg, d, arg) for d in dGG]))
        self.ksq = self.dev(np.stack(ks))
        self.dksq = self.dev(np.stack(ds))                   # [count or 1][ncp][...]

    def mean(self, x):
        return x.mean(self.axes)

    def propagate(self, w):
        """Slices of every chain in both directions, and Q."""
        qf, qr, Q = [], [], []
        for ch in self.s.chains:
            bgn, bds = _contour(ch.block_length, self.s.ds)
            tabs = []
            for m, d in zip(ch.block_monomer, bds):
                b2 = self.s.kuhn[m] ** 2
                tabs.append((torch.exp(-w[:, m] * d / 2), torch.exp(-w[:, m] * d / 4),
                             torch.exp(-d * b2 / 6 * self.ksq), torch.exp(-d * b2 / 12 * self.ksq)))

            def conv(x, k):
                return torch.fft.irfftn(k * torch.fft.rfftn(x, dim=self.axes), s=self.shape, dim=self.axes)

            def step(q, b):
                e1, e2, k1, k2 = tabs[b]
                q1 = e1 * conv(e1 * q, k1)
                return (4.0 * e2 * conv(e1 * conv(e2 * q, k2), k2) - q1) / 3.0

            one = torch.ones_like(w[:, 0])
            f, r = [one], [one]
            for b in range(len(bds)):
                for _ in range(bgn[b + 1] - bgn[b]):
                    f.append(step(f[-1], b))
            for b in reversed(range(len(bds))):
                for _ in range(bgn[b + 1] - bgn[b]):
                    r.append(step(r[-1], b))
            qf.append(f)
            qr.append(r[::-1])
            Q.append(self.mean(f[-1]))
        return qf, qr, torch.stack(Q, 1)

    def density(self, w):
        self.qf, self.qr, self.Q = self.propagate(w)
        rho = [torch.zeros_like(w[:, 0]) for _ in range(self.M)]
        at = (slice(None), None, None, None)
        qs = []
        for sv in self.s.solvents:
            x = torch.exp(-sv.size * w[:, sv.monomer])
            qs.append(self.mean(x))
            rho[sv.monomer] = rho[sv.monomer] + sv.phi * x / qs[-1][at]
        for c, ch in enumerate(self.s.chains):
            bgn, bds = _contour(ch.block_length, self.s.ds)
            for b, m in enumerate(ch.block_monomer):
                acc = 0.0
                for j in range(bgn[b], bgn[b + 1] + 1):
                    wt = 1.0 if j in (bgn[b], bgn[b + 1]) else (4.0 if (j - bgn[b]) % 2 else 2.0)
                    acc = acc + wt * self.qf[c][j] * self.qr[c][j]
                rho[m] = rho[m] + acc * (bds[b] / 3.0 * ch.phi / sum(ch.block_length)) / self.Q[:, c][at]
        self.Qs = torch.stack(qs, 1) if qs else None
        self.w, self.rho = w, torch.stack(rho, 1)
        return self.rho

    def stress(self):
        weight = self.wx * self.dksq if self.star is None else self.wx * self.star * self.dksq
        out = torch.zeros(len(self.sys), weight.shape[1], dtype=torch.float64, device="cuda")
        for c, ch in enumerate(self.s.chains):
            bgn, bds = _contour(ch.block_length, self.s.ds)
            dot = {}
            for b, m in enumerate(ch.block_monomer):
                for j in range(bgn[b], bgn[b + 1] + 1):
                    if j not in dot:
                        F, R = (torch.fft.rfftn(x[c][j], dim=self.axes) for x in (self.qf, self.qr))
                        pr = F.real * R.real + F.imag * R.imag
                        dot[j] = (weight * pr[:, None]).sum(self.axes)
                    wt = 1.0 if j in (bgn[b], bgn[b + 1]) else (4.0 if (j - bgn[b]) % 2 else 2.0)
                    out += dot[j] * (self.s.kuhn[m] ** 2 * wt * bds[b] / (18.0 * self.nr ** 2) * ch.phi / sum(ch.block_length)) \
                        / self.Q[:, c, None]
        return out

    def free_energy(self):
        w, rho = self.w, self.rho
        W, R = w, rho
        if self.star is not None:
            W, R = (torch.fft.rfftn(x, dim=self.axes) for x in (w, rho))

        def prod(a, b):
            if self.star is None:
                return self.mean(a * b)
            return (self.wx * self.star * (a.real * b.real + a.imag * b.imag)).sum(self.axes) / self.nr ** 2
        phis = self.dev([c.phi for c in self.s.chains])
        lengths = self.dev([sum(c.block_length) for c in self.s.chains])
        mu = torch.log(phis / self.Q)
        f = ((mu - 1.0) * phis / lengths).sum(1)
        g = (mu * phis / lengths).sum(1)
        for k, sv in enumerate(self.s.solvents):
            m = torch.log(sv.phi / self.Qs[:, k])
            f = f + sv.phi * (m - 1.0) / sv.size
            g = g + sv.phi * m / sv.size
        for a in range(self.M):
            f = f - prod(W[:, a], R[:, a])
            for b in range(a + 1, self.M):
                f = f + self.chi[:, a, b] * prod(R[:, a], R[:, b])
        return f, g - f, mu

    def star_weights(self):
        """fl32(sqrt(N))^2 / N of each wave's orbit of N waves under the point group."""
        n = self.n
        g = np.stack(np.meshgrid(np.arange(n[2]), np.arange(n[1]), np.arange(self.half), indexing="ij"))[::-1]
        g = torch.as_tensor(np.ascontiguousarray(g)).cuda()
        keys = []
        for m in {tuple(map(tuple, m)) for m, _ in self.ops}:
            v = [sum(int(m[i][j]) * g[i] for i in range(3)) % n[j] for j in range(3)]
            keys.append((v[0] * n[1] + v[1]) * n[2] + v[2])
        keys = torch.stack(keys).sort(0).values
        cnt = 1 + (keys[1:] != keys[:-1]).sum(0)
        return cnt.float().sqrt().double() ** 2 / cnt.double()

    def symmetrize(self, w):
        if not self.ops:
            return w
        n = self.n
        r = torch.stack(torch.meshgrid(*(torch.arange(m, device="cuda") for m in (n[2], n[1], n[0])), indexing="ij"))
        r, acc = r.flip(0), torch.zeros_like(w)
        for m, t in self.ops:
            i = [(sum(int(m[a][b]) * r[b] for b in range(3)) + int(t[a])) % n[a] for a in range(3)]
            acc += w[:, :, i[2], i[1], i[0]]
        return acc / len(self.ops)

    def solve(self, w):
        """Anderson mixing as iterate_AM: lambda = 1 - 0.9^k, all earlier
        iterates in the history, the cell mixed with the fields."""
        case, at = self.case, (slice(None), None, None, None)
        cap = 0.3 if case["chem"] == "triblock" else 1.0
        w = self.symmetrize(w)
        s = self.s
        phi = np.zeros(self.M)
        for c in s.chains:
            for m, length in zip(c.block_monomer, c.block_length):
                phi[m] += c.phi * length / sum(c.block_length)
        w0 = self.chi @ self.dev(phi)
        w = w + (w0 - self.mean(w))[..., None, None, None]
        ws, ds, cps, dcs = [], [], [], []
        cell = self.dev(self.cells)
        for k in range(1, case["iterations"] + 2):
            rho = self.density(w)
            dev = torch.einsum("iba,ib...->ia...", self.chi, rho)
            sw = w.sum(1)
            if self.M == 3:
                for a, b, c in ((0, 1, 2), (1, 2, 0), (0, 2, 1)):
                    sw = sw + self.chi[:, a, b][at] * rho[:, c]
            dev = dev + (sw / self.M)[:, None] - w
            dev = dev - self.mean(dev)[..., None, None, None]
            dc = -self.stress() if case["relax"] else torch.zeros_like(cell)
            f = self.free_energy()[0]
            if k == case["iterations"] + 1:
                break
            for hist, now in ((ws, w), (ds, dev), (cps, cell), (dcs, dc)):
                hist.append(now)
            lam = min(1.0 - 0.9 ** k, cap)
            h = k - 1
            nw, nd, nc, ndc = w, dev, cell, dc
            if h:
                dd = [dev - ds[h - 1 - m] for m in range(h)]
                cc = [dc - dcs[h - 1 - m] for m in range(h)]

                def ip(x, y, a, b):
                    return (x * y).sum((1, 2, 3, 4)) / self.nr + (a * b).sum(1)
                U = torch.stack([torch.stack([ip(dd[m], dd[n], cc[m], cc[n]) for n in range(h)], 1)
                                 for m in range(h)], 1)
                V = torch.stack([ip(dd[m], dev, cc[m], dc) for m in range(h)], 1)
                C = torch.linalg.solve(U, V)
                for m in range(h):
                    cm = C[:, m][:, None, None, None, None]
                    nw = nw + cm * (ws[h - 1 - m] - w)
                    nd = nd + cm * (ds[h - 1 - m] - dev)
                    nc = nc + C[:, m, None] * (cps[h - 1 - m] - cell)
                    ndc = ndc + C[:, m, None] * (dcs[h - 1 - m] - dc)
            w = self.symmetrize(nw + lam * nd)
            if case["relax"]:
                cell = nc + lam * ndc
                self.set_cells(cell.tolist())
        return w, rho, f, cell


def _group(name, n):
    """(matrix, translation in grid units) of every element on the grid, from generators."""
    eye = np.eye(3, dtype=int)

    def flip(*s):
        return np.diag(s)
    gens = {
        "-1": [(flip(-1, 1, 1), (0, 0, 0))],
        "p 6 m m": [(np.array([[1, -1, 0], [1, 0, 0], [0, 0, 1]]), (0, 0, 0)),
                    (np.array([[0, -1, 0], [-1, 0, 0], [0, 0, 1]]), (0, 0, 0))],
        "I m -3 m": [(flip(-1, 1, 1), (0, 0, 0)), (eye[[1, 0, 2]], (0, 0, 0)), (eye[[1, 2, 0]], (0, 0, 0)),
                     (eye, (.5, .5, .5))],
        "F d d d : 2": [(flip(-1, -1, 1), (.75, .75, 0)), (flip(-1, 1, -1), (.75, 0, .75)), (flip(-1, -1, -1), (0, 0, 0)),
                        (eye, (0, .5, .5)), (eye, (.5, 0, .5)), (eye, (.5, .5, 0))],
    }[name]
    gens = [(m, np.array([round(v * k) for v, k in zip(t, n)])) for m, t in gens]
    found, todo = {}, [(eye, np.zeros(3, dtype=int))]
    while todo:
        m, t = todo.pop()
        key = (tuple(m.ravel().tolist()), tuple((t % n).tolist()))
        if key in found:
            continue
        found[key] = (m, t % n)
        todo += [(gm @ m, gm @ t + gt) for gm, gt in gens]
    return list(found.values())


def exact(case, seed):
    r = _Ref(case)
    kind, count = case["kind"], case["count"]
    shape = (count, r.M) + r.shape
    if kind == "columns":
        # the columns' grid fields, synthesised from the star tables
        k, star, coef = _basis(case).half_grid_tables()
        k, star, coef = torch.as_tensor(k).cuda(), torch.as_tensor(star).cuda(), torch.as_tensor(coef).cuda()
        a = torch.as_tensor(_columns(case, r.sys, seed)).cuda()
        spec = torch.zeros(count, r.M, r.ksq[0].numel(), dtype=torch.complex128, device="cuda")
        spec.index_add_(2, k, a[:, :, star] * coef)
        w = torch.fft.irfftn(spec.reshape(count, r.M, r.n[2], r.n[1], r.half) * r.nr, s=r.shape, dim=r.axes)
        F = torch.fft.rfftn(r.density(w), dim=r.axes).reshape(count, r.M, -1) / r.nr
        wk = r.wx.expand(r.n[2], r.n[1], r.half).reshape(-1)[k]
        out = torch.zeros(a.shape, dtype=torch.float64, device="cuda")
        out.index_add_(2, star, wk * (F[:, :, k] * coef.conj()).real)
        return {"rho": out, "q": r.Q}
    w = r.dev(_fields(case, r.sys, seed)).reshape(shape)

    def flat(x):
        return x.reshape(count, r.M, r.nr)

    def padded(x):
        return torch.nn.functional.pad(x, (0, 6 - x.shape[1]))
    if kind == "solve":
        w, rho, f, cell = r.solve(w)
        return {"omega": flat(w), "rho": flat(rho), "f": f, "q": r.Q, "cell": cell}
    if kind == "gradient":
        w = w.requires_grad_(True)
        rho = r.density(w)
        lnq = torch.log(r.Q)
        t = _target(case, r.sys, seed).reshape((count,) + r.shape)
        loss = (rho[:, 0] - t).square().sum() / r.nr + 0.1 * lnq.sum()
        (grad,) = torch.autograd.grad(loss, w)
        return {"rho": flat(rho.detach()), "lnq": lnq.detach(), "loss": loss.detach(), "grad": flat(grad)}
    rho = flat(r.density(w))
    out = {"rho": rho, "q": r.Q, "stress": padded(r.stress())}
    if kind == "density":
        f, p, mu = r.free_energy()
        out.update({"f": f, "pressure": p, "mu": mu})
        if r.Qs is not None:
            out["q_solvent"] = r.Qs
    return out
