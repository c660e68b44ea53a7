"""Timed cases of the EAM lattice path: what a user of this package has it do.

A case is a dict of plain values; ``kind`` selects the entry points:

  sim      one resident lattice: Sim.run(steps) then Sim.download() (FP64 or mixed)
  ensemble many independent lattices kept resident: Ensemble.run(steps), download of each
  serve    requests that come and go: Ensemble.add, advance to the targets, download, remove
  hooks    the plugin boundary: one Hooks.rho_calc + Hooks.force_calc pair on the host's
           ghost-extended records in page-locked memory
  host     one step through host records in page-locked memory: Sim.step_host

Inputs are thermally disordered BCC lattices (Gaussian displacements and Maxwell-Boltzmann
velocities at the case's temperature) with vacancies and octahedral interstitials, on the
package's tabulated analytic potentials (a0 = 2.855 A, cutoff 5.6 A).  The records of a
mixed-precision run hold single-precision sums widened to the record's doubles and what
follows from them; they are returned in single precision, as its trajectories are kept.

``exact`` integrates the same inputs in 64 bits with plain torch.
"""
from __future__ import annotations

import ctypes as C
import importlib.util
import itertools
import math
import pathlib
import sys
import weakref

import numpy as np
import torch

ROOT = pathlib.Path(__file__).resolve().parents[1]
A0, MASS, RC, DT = 2.855, 55.845, 5.6, 1.0
KB, FTM2V = 8.617333262e-5, 9.64853321233e-3


def _package():
    if "misa_b200" not in sys.modules:
        pkg = ROOT / "misa-md-hip_b200"
        spec = importlib.util.spec_from_file_location("misa_b200", pkg / "__init__.py",
                                                      submodule_search_locations=[str(pkg)])
        mod = importlib.util.module_from_spec(spec)
        sys.modules["misa_b200"] = mod
        spec.loader.exec_module(mod)
    return sys.modules["misa_b200"]


# ------------------------------------------------------------------- cases
def _sim(name, cells, steps, *, prec="fp64", types=1, temp=300.0, vac=0.0, itl=0, skin=0.7, every=0, conv=False):
    return dict(name=name, kind="sim", nx=cells[0], ny=cells[1], nz=cells[2], steps=steps, prec=prec, types=types,
                temp=temp, vac=vac, itl=itl, skin=skin, every=every, conv=conv)


def listed():
    return [
        # the smallest lattice the package takes in earnest (its smoke lattice): launches and latency count
        _sim("fp64_6c", (6, 6, 6), 20, temp=600.0, every=5),
        # the 16,000-atom configuration: 100 steps at 600 K
        _sim("fp64_20c", (20, 20, 20), 100, temp=600.0, every=20),
        # ragged edges, vacancies and interstitials, as a cascade study has them
        _sim("fp64_odd_itl", (37, 52, 45), 60, vac=0.01, itl=24, every=30),
        # the scale configuration: 4.19 M sites, 0.5% vacancies, 200 interstitials, 300 K
        _sim("fp64_128c", (128, 128, 128), 200, vac=0.005, itl=200, every=100),
        # a three-element alloy (the plugin uploads types 0, 1, 2)
        _sim("fp64_alloy", (48, 40, 44), 60, types=3, temp=600.0, vac=0.005, every=30),
        # a ragged lattice in mixed precision with interstitials
        _sim("mixed_odd_itl", (33, 70, 41), 150, prec="mixed", temp=600.0, vac=0.005, itl=16, every=50),
        # the scale lattice in mixed precision
        _sim("mixed_128c", (128, 128, 128), 300, prec="mixed", vac=0.005, itl=200),
        # a hot NVE run: wide skin, lattice <-> interstitial conversion on
        _sim("mixed_nve", (64, 64, 64), 100, prec="mixed", temp=900.0, vac=0.005, itl=25, skin=1.3, every=100, conv=True),
        # a batch of lattices with edges of 8 to 40 cells, kept resident
        dict(name="ensemble_48", kind="ensemble", lats=48, lo=8, hi=40, steps=400, temp=600.0, vac=0.005),
        # short requests of the serving loop, from admission to retirement
        dict(name="serve_8", kind="serve", lats=8, lo=8, hi=30, steps=120, temp=700.0, vac=0.005),
        # the drop-in boundary on a small rank-sized lattice with ragged edges
        dict(name="hooks_30c", kind="hooks", nx=30, ny=27, nz=33, types=1, temp=300.0, vac=0.005),
        # one timestep through host records
        dict(name="host_64c", kind="host", nx=64, ny=64, nz=64, temp=300.0, vac=0.005, itl=25),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["fp64", "fp64", "alloy", "mixed", "mixed", "ensemble", "serve", "hooks", "host"])
    e = [_log(rng, 6, 110) for _ in range(3)]
    sites = 2 * e[0] * e[1] * e[2]
    steps = max(10, min(150, int(1.5e8 / sites)))
    temp = float(rng.choice([150, 300, 300, 600, 900]))
    vac = rng.choice([0.0, 0.002, 0.005, 0.01])
    itl = rng.choice([0, 0, sites // 20000, sites // 8000])
    every = rng.choice([0, 0, 10, max(1, steps // 2)])
    if kind == "fp64":
        c = _sim("", e, steps, temp=temp, vac=vac, itl=itl, every=every)
    elif kind == "alloy":
        e = [min(v, 56) for v in e]
        c = _sim("", e, min(steps, 60), types=rng.choice([2, 3]), temp=temp, vac=vac, every=every)
    elif kind == "mixed":
        c = _sim("", e, steps, prec="mixed", temp=temp, vac=vac, itl=itl, every=every)
    elif kind == "ensemble":
        hi = rng.randint(10, 40)
        c = dict(kind="ensemble", lats=_log(rng, 2, 48), lo=rng.randint(6, hi - 1), hi=hi, steps=rng.randint(50, 400),
                 temp=temp, vac=vac)
    elif kind == "serve":
        hi = rng.randint(9, 32)
        c = dict(kind="serve", lats=rng.randint(1, 10), lo=rng.randint(6, hi - 1), hi=hi, steps=rng.randint(30, 150),
                 temp=temp, vac=vac)
    elif kind == "hooks":
        e = [min(v, 72) for v in e]
        c = dict(kind="hooks", nx=e[0], ny=e[1], nz=e[2], types=rng.choice([1, 1, 2, 3]), temp=temp, vac=vac)
    else:
        e = [min(v, 80) for v in e]
        c = dict(kind="host", nx=e[0], ny=e[1], nz=e[2], temp=temp, vac=vac, itl=rng.choice([0, 4, 16]))
    c.pop("name", None)
    return c


# ------------------------------------------------------------------ inputs
def _cells(case, seed):
    """Edges of every lattice of the case; a batch's edges are part of the case, not of the seed."""
    if "lats" not in case:
        return [(case["nx"], case["ny"], case["nz"])]
    rng = np.random.default_rng(11 + 1000 * case["lats"] + 10 * case["hi"] + case["lo"])
    return [tuple(int(v) for v in rng.integers(case["lo"], case["hi"] + 1, size=3)) for _ in range(case["lats"])]


def _inputs(case, cells, seed, n_itl=0):
    """Displacement u, velocity v, type of every site (box order: x doubled, fastest) and the
    interstitials' positions and velocities."""
    rng = np.random.default_rng([seed, *cells])
    n = 2 * cells[0] * cells[1] * cells[2]
    t = rng.integers(0, case.get("types", 1), size=n).astype(np.int32)
    t[rng.choice(n, size=int(round(case["vac"] * n)), replace=False)] = -1
    live = (t >= 0)[:, None]
    u = rng.standard_normal((n, 3)) * (0.07 * math.sqrt(case["temp"] / 300.0)) * live
    sv = math.sqrt(KB * case["temp"] * FTM2V / MASS)
    v = rng.standard_normal((n, 3)) * sv
    v = (v - v.mean(axis=0)) * live
    pick = rng.choice(cells[0] * cells[1] * cells[2] * 6, size=n_itl, replace=False) if n_itl else np.zeros(0, int)
    octa = np.array([[.5, .5, 0], [.5, 0, .5], [0, .5, .5], [.5, 0, 0], [0, .5, 0], [0, 0, .5]])
    c = pick // 6
    q = (np.stack([c % cells[0], (c // cells[0]) % cells[1], c // (cells[0] * cells[1])], -1) + octa[pick % 6]) * A0
    return u, v, t, q.reshape(-1, 3), rng.standard_normal((n_itl, 3)) * sv


def _ideal(cells):
    nx, ny, nz = cells
    z, y, x = np.ogrid[:nz, :ny, :2 * nx]
    h = 0.5 * (x & 1)
    out = np.empty((nz, ny, 2 * nx, 3))
    out[..., 0] = 0.5 * A0 * x
    out[..., 1] = A0 * (y + h)
    out[..., 2] = A0 * (z + h)
    return out.reshape(-1, 3)


def _records(mb, case, cells, seed, n_itl=0, box=None):
    u, v, t, q, w = _inputs(case, cells, seed, n_itl)
    box = np.zeros(len(t), dtype=mb.ATOM_DTYPE) if box is None else box
    box["id"] = np.arange(1, len(t) + 1)
    box["type"] = t
    box["x"] = _ideal(cells) + u
    box["v"] = v
    itl = np.zeros(n_itl, dtype=mb.ATOM_DTYPE)
    itl["id"] = (1 << 40) + np.arange(n_itl)
    itl["x"], itl["v"] = q, w
    return box, itl


def _tables(mb, types):
    return mb.potential.fe_analytic() if types == 1 else mb.potential.alloy_analytic(types)


def _pinned(mb, n):
    """n zeroed records in page-locked memory of the package's own allocator, released when
    the last view of them is gone."""
    p, got = C.c_void_p(), C.c_int()
    mb.check(mb.lib().mb_create_atoms_mem(C.byref(p), 104, n, 1, 1, C.byref(got)))
    mem = (C.c_uint8 * (104 * n)).from_address(p.value)
    weakref.finalize(mem, mb.lib().mb_release_atoms_mem, p, None).atexit = False
    a = np.frombuffer(mem, dtype=mb.ATOM_DTYPE)
    a[:] = 0
    return a


# ---------------------------------------------------------- prepare and run
def prepare(case, seed):
    mb = _package()
    kind, cells = case["kind"], _cells(case, seed)
    if kind == "sim":
        c, tab, mixed = cells[0], _tables(mb, case["types"]), case["prec"] == "mixed"
        # capacity for the conversions of a hot run: about 0.1% of the sites
        cap = max(case["itl"], 2 * c[0] * c[1] * c[2] // 1000 + 64) if case["conv"] else case["itl"]
        sim = mb.Sim(c, tab, A0, MASS, DT, RC, case["skin"], mb.MB_PREC_MIXED if mixed else mb.MB_PREC_FP64, cap)
        sim.upload(*_records(mb, case, c, seed, case["itl"]))
        if case["conv"]:
            sim.set_conversion(1.0, 0.5)
        return {"case": case, "sim": sim}
    if kind in ("ensemble", "serve"):
        ens = mb.Ensemble(_tables(mb, 1), A0, MASS, DT, RC, 0.7)
        boxes = [_records(mb, case, c, seed + k)[0] for k, c in enumerate(cells)]
        slots = [ens.add(c, b) for c, b in zip(cells, boxes)] if kind == "ensemble" else None
        return {"case": case, "ens": ens, "cells": cells, "boxes": boxes, "slots": slots}
    if kind == "hooks":
        c, tab = cells[0], _tables(mb, case["types"])
        ghost = mb.lattice.ghost_for_reach(A0, RC + 0.7)
        dom = mb.lattice.domain(c, ghost)
        hooks = mb.Hooks(0)
        hooks.domain_init(dom)
        hooks.nei_offset_init(*mb.lattice.stencil_linear(A0, RC + 0.7, dom.ext_size_x, dom.ext_size_y))
        hooks.pot_init(tab)
        mem = _pinned(mb, dom.ext_size_x * dom.ext_size_y * dom.ext_size_z)
        mb.lattice.box_to_ext(_records(mb, case, c, seed)[0], c, ghost, A0, out=mem)
        hooks.rho_calc(mem, RC)  # the host fills the ghosts' df before the force pass
        ext = mem.reshape(dom.ext_size_z, dom.ext_size_y, dom.ext_size_x)
        inner = ext[ghost[2]:-ghost[2], ghost[1]:-ghost[1], ghost[0]:-ghost[0]]["df"]
        ext["df"] = np.pad(inner, [(g, g) for g in reversed(ghost)], mode="wrap")
        box = ext[ghost[2]:-ghost[2], ghost[1]:-ghost[1], ghost[0]:-ghost[0]]
        return {"case": case, "hooks": hooks, "mem": mem, "box": box}
    c = cells[0]
    mem = _pinned(mb, 2 * c[0] * c[1] * c[2])
    _, itl = _records(mb, case, c, seed, case["itl"], box=mem)
    sim = mb.Sim(c, _tables(mb, 1), A0, MASS, DT, RC, 0.7, mb.MB_PREC_FP64, case["itl"])
    return {"case": case, "sim": sim, "mem": mem, "itl": itl}


def _fields(box, single):
    """x, v, f, rho, df of records; single: in single precision (see the top)."""
    if not single:
        return {k: box[k] for k in ("x", "v", "f", "rho", "df")}
    a = torch.from_numpy(box.view(np.float64).reshape(-1, 13))
    return {"x": a[:, 2:5].float(), "v": a[:, 5:8].float(), "f": a[:, 8:11].float(), "rho": a[:, 11].float(),
            "df": a[:, 12].float()}


def _together(boxes):
    parts = [_fields(b, True) for b in boxes]
    return {k: torch.cat([p[k] for p in parts]) for k in parts[0]}


def run(state):
    case, kind = state["case"], state["case"]["kind"]
    if kind == "sim":
        sim, single = state["sim"], case["prec"] == "mixed"
        sim.run(case["steps"], case["every"])
        box, itl = sim.download()
        out = _fields(box, single)
        if case["itl"] and not case["conv"]:
            out["itl"] = _fields(itl, single)
        if case["conv"]:
            out["type"] = box["type"]
        if case["every"]:
            out["energies"] = sim.energies().astype(np.float32 if single else np.float64)
        return out
    if kind == "ensemble":
        state["ens"].run(case["steps"])
        return _together([state["ens"].download(s)[0] for s in state["slots"]])
    if kind == "serve":
        ens = state["ens"]
        slots = [ens.add(c, b, None, case["steps"] - 3 * k) for k, (c, b) in enumerate(zip(state["cells"], state["boxes"]))]
        while ens.advance(50):
            pass
        boxes = [ens.download(s)[0] for s in slots]
        for s in slots:
            ens.remove(s)
        return _together(boxes)
    if kind == "hooks":
        state["hooks"].rho_calc(state["mem"], RC)
        state["hooks"].force_calc(state["mem"], RC)
        return {k: state["box"][k] for k in ("rho", "df", "f")}
    state["sim"].step_host(state["mem"], state["itl"])
    return {**_fields(state["mem"], False), **({"itl": _fields(state["itl"], False)} if case["itl"] else {})}


def work(case):
    """A resident step cannot do without each atom's state once: 192 B per atom-step in FP64
    (rho pass x, type in, df out; force pass x, type, df, v, f in, x, v, f out), 160 B with
    mixed storage; 58 pairs of 20 (rho) + 50 (force) flop and 30 more.  Records that cross
    the boundary are 104 B each."""
    sites = sum(2 * c[0] * c[1] * c[2] for c in _cells(case, 0))
    kind = case["kind"]
    if kind == "hooks":
        g = [(case["nx"] + 4) * 2, case["ny"] + 4, case["nz"] + 4]
        # x, type in and rho, df out; x, type, df in and f out
        return {"bytes": g[0] * g[1] * g[2] * (28 + 36) + sites * (16 + 24), "flops": sites * 4090}
    steps = 1 if kind == "host" else case["steps"]
    if kind == "serve":
        steps = sum(max(1, case["steps"] - 3 * k) for k in range(case["lats"])) / case["lats"]
    per = 160 if kind in ("ensemble", "serve") or case.get("prec") == "mixed" else 192
    records = 104 * sites * (2 if kind in ("serve", "host") else 1)
    return {"bytes": steps * per * sites + records, "flops": steps * 4090 * sites}


# -------------------------------------------------------- the same, in 64 bits
def _pieces(y, dx):
    """Cubic pieces {y, s, c2, c3} of the tabulated-EAM spline (4th-order knot slopes)."""
    s = np.empty_like(y)
    s[0], s[1], s[-2], s[-1] = y[1] - y[0], 0.5 * (y[2] - y[0]), 0.5 * (y[-1] - y[-3]), y[-1] - y[-2]
    s[2:-2] = ((y[:-4] - y[4:]) + 8.0 * (y[3:-1] - y[1:-3])) / 12.0
    dy = np.diff(y)
    c2, c3 = 3 * dy - 2 * s[:-1] - s[1:], s[:-1] + s[1:] - 2 * dy
    return np.stack([y, s, np.append(c2, 0.0), np.append(c3, 0.0)], -1), dx


class _Potential:
    def __init__(self, types, dev):
        self.nt = types
        if types == 1:
            nr = nrho = 5000
            rho_max = 50.0
            sf, sF, amp = [1.0], [1.0], {(0, 0): 0.8}
        else:
            nr = nrho = 2000
            rho_max = 200.0
            sf, sF = [1 + 0.15 * a for a in range(types)], [1 + 0.1 * a for a in range(types)]
            amp = {(a, b): 0.8 + 0.05 * (a + b) for a in range(types) for b in range(a, types)}
        r, rho = np.linspace(0.0, RC, nr), np.linspace(0.0, rho_max, nrho)
        up = lambda rows: (torch.from_numpy(np.stack([p[0] for p in rows])).to(dev), rows[0][1])  # noqa: E731
        self.f = up([_pieces(k * (RC - r) ** 2, RC / (nr - 1)) for k in sf])
        self.F = up([_pieces(-k * np.sqrt(rho), rho_max / (nrho - 1)) for k in sF])
        self.phi = up([_pieces(k * (RC - r) ** 2 * (1.0 - 0.2 * r), RC / (nr - 1)) for k in amp.values()])
        pair = torch.zeros((types, types), dtype=torch.int64)
        for q, (a, b) in enumerate(amp):
            pair[a, b] = pair[b, a] = q
        self.pair, self.rho_max = pair.to(dev), rho_max

    def at(self, table, row, x, want):
        """Values (want 0) or derivatives (1) at x, clamped to the table."""
        tab, dx = table
        n = tab.shape[1]
        t = x / dx
        m = t.to(torch.int64).clamp_(0, n - 2)
        p = (t - m).clamp_(max=1.0)
        c = tab.reshape(-1, 4)[m if self.nt == 1 else row * n + m]
        if want == 0:
            return ((c[..., 3] * p + c[..., 2]) * p + c[..., 1]) * p + c[..., 0]
        return ((3 * c[..., 3] * p + 2 * c[..., 2]) * p + c[..., 1]) / dx

    def embed(self, t, rho):
        d = self.at(self.F, t, rho, 1)
        e = self.at(self.F, t, rho, 0)
        return d, e + d * (rho - self.rho_max).clamp(min=0.0)


class _Plain:
    """Velocity-Verlet of independent periodic lattices (and interstitials of a single one)."""

    def __init__(self, case, lattices, dev):
        self.dev, self.P = dev, _Potential(case.get("types", 1), dev)
        self.reach = RC + case.get("skin", 0.7)
        lim = int(self.reach / (0.5 * A0)) + 1
        hs = [h for h in itertools.product(range(-lim, lim + 1), repeat=3)
              if h > (0, 0, 0) and len({v & 1 for v in h}) == 1 and 0.5 * A0 * math.sqrt(sum(v * v for v in h)) < self.reach]
        idx, at, self.seg = [], 0, []
        for k, (cells, _) in enumerate(lattices):
            nx, ny, nz = cells
            n = 2 * nx * ny * nz
            g = torch.arange(n, device=dev)
            xd, y, z = g % (2 * nx), (g // (2 * nx)) % ny, g // (2 * nx * ny)
            s, cx = xd & 1, xd >> 1
            rows = []
            for h in hs:
                s2 = (s + h[0]) & 1
                d = [torch.div(s + h[a] - s2, 2, rounding_mode="floor") for a in range(3)]
                rows.append((((z + d[2]) % nz) * ny + (y + d[1]) % ny) * (2 * nx) + 2 * ((cx + d[0]) % nx) + s2 + at)
            idx.append(torch.stack(rows))
            at += n
        self.J, self.n = torch.cat(idx, 1) if len(idx) > 1 else idx[0], at
        self.H = torch.tensor(hs, dtype=torch.float64, device=dev).T * (0.5 * A0)
        up = lambda k: torch.from_numpy(np.concatenate([x[k] for _, x in lattices])).to(dev)  # noqa: E731
        self.u, self.v, self.t = up(0).T.contiguous(), up(1).T.contiguous(), up(2).to(torch.int64)
        self.q, self.w = (torch.from_numpy(lattices[0][1][k]).to(dev).T.contiguous() for k in (3, 4))
        self.live, self.ty = self.t >= 0, self.t.clamp(min=0)
        self.cells, self.X = lattices[0][0], None
        self.h = 0.5 * DT * FTM2V / MASS

    def pairs(self):
        """(i, j, d, r): lattice pairs in chunks of stencil vectors, each pair once."""
        step = max(1, (1 << 26) // self.n)
        for a in range(0, self.J.shape[0], step):
            j = self.J[a:a + step]
            d = self.u[:, None, :] - self.u[:, j] - self.H[:, a:a + step, None]
            r2 = (d * d).sum(0)
            on = (r2 < RC * RC) & self.live & self.live[j]
            yield j, d, torch.sqrt(torch.where(on, r2, torch.full_like(r2, 9.0))), on.to(torch.float64)

    def itl_pairs(self):
        """(k, j, d, r) of interstitial k and lattice site j, and (k, l, d, r) among interstitials."""
        nx, ny, nz = self.cells
        o = torch.arange(-5, 6, device=self.dev)
        o = torch.cartesian_prod(o, o, o, torch.arange(2, device=self.dev)).T
        c = [torch.floor(self.q[a] / A0).to(torch.int64)[:, None] + o[a] for a in range(3)]
        rel = torch.stack([A0 * (c[a] + 0.5 * o[3].to(torch.float64)) - self.q[a][:, None] for a in range(3)])
        near = (rel * rel).sum(0) < self.reach ** 2
        k = near.nonzero()[:, 0]
        j = (((c[2] % nz) * ny + c[1] % ny) * (2 * nx) + 2 * (c[0] % nx) + o[3])[near]
        d = -(rel[:, near] + self.u[:, j])
        r = torch.sqrt((d * d).sum(0))
        on = (r < RC) & self.live[j]
        lat = (k[on], j[on], d[:, on], r[on])
        e = self.q[:, :, None] - self.q[:, None, :]
        L = torch.tensor(self.cells, dtype=torch.float64, device=self.dev).reshape(3, 1, 1) * A0
        e = e - L * torch.round(e / L)
        r = torch.sqrt((e * e).sum(0))
        on = (r < RC) & ~torch.eye(len(r), dtype=torch.bool, device=self.dev)
        a, b = on.nonzero().T
        return lat, (a, b, e[:, on], r[on])

    def density(self):
        P, multi = self.P, self.P.nt > 1
        rho = torch.zeros(self.n, dtype=torch.float64, device=self.dev)
        for j, d, r, on in self.pairs():
            a = P.at(P.f, self.ty[j], r, 0) * on
            b = P.at(P.f, self.ty.expand_as(j), r, 0) * on if multi else a
            rho += a.sum(0)
            rho.index_add_(0, j.reshape(-1), b.reshape(-1))
        rho_q = torch.zeros(self.q.shape[1], dtype=torch.float64, device=self.dev)
        if len(rho_q):
            (k, j, _, r), (a, b, _, r2) = self.itl_pairs()
            f = P.at(P.f, torch.zeros_like(k), r, 0)
            rho.index_add_(0, j, f)
            rho_q.index_add_(0, k, f)
            rho_q.index_add_(0, a, P.at(P.f, torch.zeros_like(a), r2, 0))
        self.rho, self.rho_q = rho * self.live, rho_q
        self.df, eF = P.embed(self.ty, self.rho)
        self.df_q, eQ = P.embed(torch.zeros_like(rho_q, dtype=torch.int64), rho_q)
        self.df = self.df * self.live
        return float((eF * self.live).sum() + eQ.sum())

    def forces(self, energy=True):
        P, multi = self.P, self.P.nt > 1
        e = self.density()
        f = torch.zeros_like(self.u)
        for j, d, r, on in self.pairs():
            ti, tj = (self.ty.expand_as(j), self.ty[j]) if multi else (None, None)
            fj = P.at(P.f, tj, r, 1)
            fi = P.at(P.f, ti, r, 1) if multi else fj
            q = P.pair[ti, tj] if multi else None
            s = -(self.df * fj + self.df[j] * fi + P.at(P.phi, q, r, 1)) / r * on
            if energy:
                e += float((P.at(P.phi, q, r, 0) * on).sum())
            d *= s
            f += d.sum(1)
            f.index_add_(1, j.reshape(-1), -d.reshape(3, -1))
        g = torch.zeros_like(self.q)
        if g.shape[1]:
            (k, j, d, r), (a, b, d2, r2) = self.itl_pairs()
            z, z2 = torch.zeros_like(k), torch.zeros_like(a)
            s = -((self.df_q[k] + self.df[j]) * P.at(P.f, z, r, 1) + P.at(P.phi, z, r, 1)) / r * d
            g.index_add_(1, k, s)
            f.index_add_(1, j, -s)
            s2 = -((self.df_q[a] + self.df_q[b]) * P.at(P.f, z2, r2, 1) + P.at(P.phi, z2, r2, 1)) / r2 * d2
            g.index_add_(1, a, s2)
            e += float(P.at(P.phi, z, r, 0).sum() + 0.5 * P.at(P.phi, z2, r2, 0).sum())
        self.f, self.g, self.pe = f * self.live, g, e

    def kinetic(self):
        return float((self.v * self.v).sum() + (self.w * self.w).sum()) * 0.5 * MASS / FTM2V

    def steps(self, n, every, first_forces=True):
        rows = []
        if first_forces:
            self.forces(every > 0)
        else:  # records that come with zero forces
            self.f, self.g = torch.zeros_like(self.u), torch.zeros_like(self.q)
        if every:
            rows.append((0.0, self.pe, self.kinetic()))
        for k in range(1, n + 1):
            self.v += self.h * self.f
            self.w += self.h * self.g
            self.u += DT * self.v
            self.q += DT * self.w
            here = every > 0 and k % every == 0
            self.forces(here)
            self.v += self.h * self.f
            self.w += self.h * self.g
            if here:
                rows.append((float(k), self.pe, self.kinetic()))
        return np.array(rows)


def _out(p, cells_list):
    X = torch.from_numpy(np.concatenate([_ideal(c) for c in cells_list])).to(p.dev)
    x = (X + p.u.T) * p.live[:, None]
    return {"x": x, "v": p.v.T, "f": p.f.T, "rho": p.rho, "df": p.df}


def exact(case, seed):
    if case.get("conv"):
        return None  # which atoms change lists is a decision at each step, not a computed number
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    kind, cells = case["kind"], _cells(case, seed)
    lats = [(c, _inputs(case, c, seed + k, case.get("itl", 0))) for k, c in enumerate(cells)]
    if kind == "serve":  # each lattice has its own number of steps
        outs = []
        for k, lat in enumerate(lats):
            p = _Plain(case, [lat], dev)
            p.steps(max(0, case["steps"] - 3 * k), 0)
            outs.append(_out(p, [lat[0]]))
        return {k: torch.cat([o[k] for o in outs]) for k in outs[0]}
    p = _Plain(case, lats, dev)
    if kind == "hooks":
        p.forces(False)
        n = (cells[0][2], cells[0][1], 2 * cells[0][0])
        # vacant records keep what the host left in them (zeros)
        return {"rho": p.rho.reshape(n), "df": p.df.reshape(n), "f": p.f.T.reshape(*n, 3)}
    rows = p.steps(1 if kind == "host" else case["steps"], case.get("every", 0), kind != "host")
    out = _out(p, cells)
    if case.get("itl"):
        out["itl"] = {"x": p.q.T, "v": p.w.T, "f": p.g.T, "rho": p.rho_q, "df": p.df_q}
    if case.get("every"):
        out["energies"] = rows
    return out
