"""The molecular-dynamics work this framework is measured on: what each case stands for is said in
listed().  Every case goes through the public classes of lpmd2_gb300.gbmd."""
from __future__ import annotations

import math

import numpy as np
import torch

from lpmd2_gb300 import gbmd
from lpmd2_gb300 import inputs as I

SIGMA, EPS = I.LJ_AR["sigma"], I.LJ_AR["epsilon"]
RC_LJ = 2.5 * SIGMA
TAU = I.lj_reduced_units(SIGMA, EPS, I.LJ_AR["mass"])["tau_fs"]

# Material parameters of the repository's tests and benchmark.
SC = dict(e=0.012382, a=3.61, n=9, m=6, c=39.432)
FS = dict(c0=1.2371147, c1=-0.3592185, c2=-0.0385607, A=1.828905, B=1.8, c=3.40, d=3.569745)
FSX = dict(c0=47.1346499, c1=-33.7665655, c2=6.2541999, c3=-0.0122, c4=0.0001, A=1.848, B=0.5, c=3.25, d=4.1)
GUPTA = dict(A=0.2061, r0=2.884, p=10.229, B=1.790, q=4.036)
# plugin, its parameters, cutoff, lattice constant, species, temperature (K), time step (fs)
METALS = {
    "sc": ("suttonchen", SC, 2 * SC["a"], 3.61, "Cu", 300.0, 2.0),
    "fs": ("finnissinclair", FS, FS["d"], 3.6, "Fe", 300.0, 1.0),
    "fsx": ("finnissinclair-ext", FSX, FSX["d"], 3.6, "Mo", 300.0, 1.0),
    "gupta": ("gupta", GUPTA, 6.0, 4.08, "Au", 400.0, 2.0),
}


def _md(name, pot, k, steps, precision, cm, drop=0, integ="velocityverlet", skin=-1.0, nsys=1):
    """One MD case: an FCC start of k^3 cells (4 k^3 atoms, `drop` of them removed) and `steps` steps a
    pass.  skin < 0: the cell manager's default.  nsys > 1: an ensemble of independent systems whose
    sizes are spread log-uniformly from 256 atoms to 4 k^3."""
    c = dict(do="md", pot=pot, k=k, steps=steps, precision=precision, cm=cm, drop=drop, integ=integ, skin=skin, nsys=nsys)
    return dict(c, name=name) if name else c


def listed():
    return [
        # pair forces of one very small system from device buffers: the smallest call there is
        dict(name="static_108", do="static", k=3, drop=0),
        # the tutorial-sized run of the reference: plain minimum image, default (FP64) precision
        _md("lj_864_minimumimage_fp64", "lj", 6, 20, "fp64", "minimumimage"),
        # a small liquid in mixed precision: a study of many such runs is bound by latency
        _md("lj_4k_mixed", "lj", 10, 100, "mixed", "verletlist", skin=0.3 * SIGMA),
        # the benchmark's liquid of 256,000 atoms
        _md("lj_256k_mixed", "lj", 40, 50, "mixed", "verletlist", skin=0.3 * SIGMA),
        # the largest system that the benchmark runs, 2,048,000 atoms
        _md("lj_2m_mixed", "lj", 80, 50, "mixed", "verletlist", skin=0.3 * SIGMA),
        # default precision and the reference's own Verlet list (8 % wider than the cutoff, rebuilt on
        # the `each` clock), on a system with some sites missing
        _md("lj_108k_fp64", "lj", 30, 20, "fp64", "verletlist", drop=37),
        # the benchmark's copper with 1 % vacancies: the two-pass metal force
        _md("cu_495k_mixed", "sc", 50, 50, "mixed", "linkedcell", drop=5000, skin=0.4),
        # copper in default precision on linked cells
        _md("cu_54k_fp64", "sc", 24, 10, "fp64", "linkedcell", drop=553),
        # a metal potential with a short cutoff, mixed precision
        _md("fe_32k_mixed", "fs", 20, 50, "mixed", "linkedcell", drop=13),
        # ensemble of independent systems of uneven sizes
        _md("ensemble_128_mixed", "lj", 20, 100, "mixed", "verletlist", skin=0.3 * SIGMA, nsys=128),
        # a thermodynamic sampling run's integrator other than velocity Verlet
        _md("lj_16k_beeman_mixed", "lj", 16, 50, "mixed", "linkedcell", integ="beeman"),
        # a program that keeps its own positions and asks for energies and forces (UpdateForces
        # behind the reference's plugin interface), default precision
        dict(name="forces_32k_fp64", do="forces", pot="lj", k=20, precision="fp64", cm="linkedcell", drop=101, skin=-1.0),
    ]


def draw(rng):
    def k_between(lo, hi):  # spread over the logarithm of the number of atoms
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def drop_of(k):  # ragged sizes: up to 1 % of the sites missing
        return rng.randrange(0, max(2, 4 * k**3 // 100))

    kind = rng.choice(["static", "small", "lj", "lj", "metal", "metal", "ensemble", "integrator", "forces"])
    if kind == "static":
        k = k_between(3, 8)
        return dict(do="static", k=k, drop=rng.randrange(1, k**3))
    precision = rng.choice(["fp64", "mixed"])
    if kind == "small":
        k = k_between(5, 8)
        return _md("", "lj", k, 20, "fp64", rng.choice(["minimumimage", "linkedcell", "verletlist"]), drop=drop_of(k))
    if kind == "lj":
        k = k_between(5, 60 if precision == "mixed" else 32)
        cm = rng.choice(["linkedcell", "verletlist"])
        skin = rng.choice([-1.0, 0.2 * SIGMA, 0.3 * SIGMA, 0.4 * SIGMA])
        steps = rng.choice([20, 30, 50]) if precision == "mixed" else 20
        return _md("", "lj", k, steps, precision, cm, drop=drop_of(k), skin=skin)
    if kind == "metal":
        pot = rng.choice(["sc", "fs", "fsx", "gupta"])
        k = k_between(6, 40 if precision == "mixed" else 24)
        return _md("", pot, k, 10 if precision == "fp64" else rng.choice([20, 50]), precision,
                   rng.choice(["linkedcell", "verletlist"]), drop=drop_of(k), skin=rng.choice([-1.0, 0.3, 0.5]))
    if kind == "ensemble":
        nsys = rng.choice([16, 33, 64] if precision == "mixed" else [9, 16, 24])
        return _md("", rng.choice(["lj", "sc"]), rng.choice([6, 10, 14]), 50 if precision == "mixed" else 10, precision,
                   "verletlist", skin=0.3 * SIGMA, nsys=nsys)
    if kind == "integrator":
        k = k_between(5, 24)
        return _md("", "lj", k, 20, precision, "linkedcell", drop=drop_of(k), integ="beeman")
    k = k_between(6, 40 if precision == "mixed" else 30)
    return dict(do="forces", pot=rng.choice(["lj", "sc", "gupta"]), k=k, precision=precision, cm="linkedcell",
                drop=drop_of(k), skin=-1.0)


# ----------------------------------------------------------------------------------------------
# Inputs
# ----------------------------------------------------------------------------------------------


def _liquid(k, drop, rho, t_star, seed):
    a = (4.0 / rho) ** (1.0 / 3.0) * SIGMA
    pos, L = I.fcc_fast(k, k, k, a)
    if drop:
        pos = I.remove_sites(pos, drop / len(pos), seed=seed)
    pos = np.mod(I.jitter(pos, 0.05 * SIGMA, seed=seed), L)
    m = np.full(len(pos), I.LJ_AR["mass"])
    return dict(pos=pos, vel=I.maxwell_boltzmann(m, t_star * EPS / I.KBOLTZMANN, seed=seed), mass=m, Z=18, L=L)


def _metal(pot, k, drop, seed):
    _, _, _, a, symbol, T, _ = METALS[pot]
    pos, L = I.fcc_fast(k, k, k, a)
    if drop:
        pos = I.remove_sites(pos, drop / len(pos), seed=seed)
    pos = np.mod(I.jitter(pos, 0.03, seed=seed), L)
    m = np.full(len(pos), I.MASSES[symbol])
    return dict(pos=pos, vel=I.maxwell_boltzmann(m, T, seed=seed), mass=m, Z=I.ATOMIC_NUMBERS[symbol], L=L)


def _systems(case, seed):
    nsys = int(case.get("nsys", 1))
    out = []
    u = I.uniform(seed, 3 * nsys, stream=11).reshape(nsys, 3)
    for s in range(nsys):
        k, rho, t = case["k"], 0.8442, 1.5
        if nsys > 1:
            # the sizes are the case's own (an ensemble's shape does not change with its inputs)
            frac = ((s * 0.6180339887498949) % 1.0)
            k = max(4, int(round(4.0 * (case["k"] / 4.0) ** frac)))
            rho, t = 0.70 + 0.25 * u[s, 1], 0.7 + 1.3 * u[s, 2]
        if case.get("pot", "lj") == "lj":
            out.append(_liquid(k, case.get("drop", 0), rho, t, seed * 100003 + s))
        else:
            out.append(_metal(case["pot"], max(k, 5), case.get("drop", 0), seed * 100003 + s))
    return out


def _constants(case):
    """(plugin, arguments, cutoff, time step)."""
    pot = case.get("pot", "lj")
    if pot == "lj":
        return "lennardjones", f"sigma {SIGMA} epsilon {EPS} cutoff {RC_LJ!r}", RC_LJ, 0.005 * TAU
    plugin, p, rc, _, _, _, dt = METALS[pot]
    args = " ".join(f"{k} {v!r}" for k, v in p.items())
    if pot in ("sc", "gupta"):
        args += f" cutoff {rc!r}"
    return plugin, args, rc, dt


def _wire(sim, case, L):
    plugin, args, rc, dt = _constants(case)
    skin = f" skin {case['skin']!r}" if case["skin"] >= 0 else ""
    if case["cm"] == "minimumimage":
        cm = f"cutoff {rc!r}"
    elif case["cm"] == "linkedcell":
        n = int(float(L[0]) / rc + 1e-9)
        if n > 3 and float(L[0]) / n < rc * (1.0 + 1e-9):  # cells no narrower than the cutoff
            n -= 1
        cm = f"cutoff {rc!r} nx {n} ny {n} nz {n}" + skin
    else:
        # without a skin the reference's own rebuild clock, with one the displacement rule
        cm = f"cutoff {rc!r} maxneighbors 512" + (skin if skin else " each 5")
    sim.set_cell_manager(gbmd.Plugin(case["cm"], cm))
    sim.add_potential(gbmd.Plugin(plugin, args))
    sim.set_integrator(gbmd.Plugin(case.get("integ", "velocityverlet"), f"dt {dt!r}"))
    sim.set_precision(case["precision"])


def prepare(case, seed):
    systems = _systems(case, seed)
    w = systems[0]
    if case["do"] == "static":
        n = len(w["pos"])
        return dict(case=case, n=n, box=w["L"], plugin=gbmd.Plugin("lennardjones", _constants(case)[1]),
                    pos=torch.from_numpy(w["pos"]).cuda(), force=torch.empty((n, 3), dtype=torch.float64, device="cuda"),
                    sums=torch.empty(11, dtype=torch.float64, device="cuda"))
    sizes = [len(x["pos"]) for x in systems]
    # page-locked buffers for the state that is read back
    host = torch.empty((3, sum(sizes), 3), dtype=torch.float64, pin_memory=True)
    state = dict(case=case, systems=systems, sizes=sizes, host=host)
    if case["precision"] == "mixed":
        # frames of a mixed run are kept in single precision, the precision of its pair terms
        state["frame"] = torch.empty((3, sum(sizes), 3), dtype=torch.float32)
    views, at = [], 0
    h = host.numpy()
    for n in sizes:
        views.append(tuple(h[q, at:at + n] for q in range(3)))
        at += n
    state["views"] = views
    if len(systems) > 1:
        sim = gbmd.Batch(sizes, [x["L"] for x in systems])
        for s, x in enumerate(systems):
            sim.set_atoms(s, x["pos"], x["vel"], Z=x["Z"], mass=x["mass"])
    else:
        sim = gbmd.Simulation(sizes[0], w["L"])
        sim.set_atoms(w["pos"], w["vel"], Z=w["Z"], mass=w["mass"])
    _wire(sim, case, w["L"])
    sim.update_forces()
    state["sim"] = sim
    return state


def run(state):
    case = state["case"]
    if case["do"] == "static":
        gbmd.pair_forces_static(state["plugin"], state["pos"].data_ptr(), state["n"], state["box"],
                                state["force"].data_ptr(), state["sums"].data_ptr(),
                                torch.cuda.current_stream().cuda_stream)
        return dict(force=state["force"], sums=state["sums"])
    sim = state["sim"]
    if case["do"] == "forces":
        w = state["systems"][0]
        sim.set_atoms(w["pos"], w["vel"], Z=w["Z"], mass=w["mass"])
        sim.update_forces()
    else:
        sim.do_steps(case["steps"])
    if len(state["sizes"]) > 1:
        thermo = np.stack([sim.thermo(s)["raw"] for s in range(len(state["sizes"]))])
        for s, view in enumerate(state["views"]):
            sim.atoms(s, out=view)
    else:
        thermo = sim.thermo_raw()
        sim.atoms(out=state["views"][0])
    frame = state["host"]
    if "frame" in state:
        frame = state["frame"].copy_(state["host"])
        thermo = thermo.astype(np.float32)
    if case["do"] == "forces":
        return dict(acc=frame[2], thermo=thermo)
    return dict(pos=frame[0], vel=frame[1], acc=frame[2], thermo=thermo)


def work(case):
    """Positions, velocities and accelerations read and written once a step (pair potentials 168 bytes
    an atom, metals 200), and the operations of the pairs inside the cutoff."""
    sizes = []
    for s in range(int(case.get("nsys", 1))):
        k = case["k"]
        if case.get("nsys", 1) > 1:
            k = max(4, int(round(4.0 * (case["k"] / 4.0) ** ((s * 0.6180339887498949) % 1.0))))
            k = k if case["pot"] == "lj" else max(k, 5)
        sizes.append(4 * k**3 - case.get("drop", 0))
    n = sum(sizes)
    pot = case.get("pot", "lj")
    density = 0.8442 / SIGMA**3 if pot == "lj" else 4.0 / METALS[pot][3] ** 3
    rc = RC_LJ if pot == "lj" else METALS[pot][2]
    pairs = 0.5 * 4.18879 * rc**3 * density
    if case["do"] == "static":
        return dict(bytes=n * 48.0 + 88.0, flops=n * pairs * 45.0)
    steps = case.get("steps", 1)
    per_pair = 45.0 if pot == "lj" else 75.0
    return dict(bytes=n * steps * (168.0 if pot == "lj" else 200.0), flops=n * steps * pairs * per_pair)


# ----------------------------------------------------------------------------------------------
# The same, in 64 bits with plain torch
# ----------------------------------------------------------------------------------------------

KIN2EV, KB, PRESS, FORCEFACTOR = 103.64269, 8.6173422e-05, 160217.65, 0.00964853


def _pairs_of(x, L, rl):
    """(i, j) with i < j of one system whose minimum-image distance is below rl."""
    n = x.shape[0]
    nc = [max(1, int(float(q) / rl)) for q in L.tolist()]
    if n <= 3000 or min(nc) < 3:
        got = []
        rows = max(1, int(4e7 // max(n, 1)))
        for a in range(0, n, rows):
            d = x[None, :, :] - x[a:a + rows, None, :]
            d = d - L * torch.round(d / L)
            hit = (d * d).sum(-1) < rl * rl
            i, j = hit.nonzero(as_tuple=True)
            i = i + a
            got.append(torch.stack([i[i < j], j[i < j]]))
        return torch.cat(got, dim=1)
    dev = x.device
    nct = torch.tensor(nc, device=dev)
    c3 = torch.minimum((torch.remainder(x, L) / L * nct).long(), nct - 1)
    cell = (c3[:, 2] * nc[1] + c3[:, 1]) * nc[0] + c3[:, 0]
    order = torch.argsort(cell)
    ncell = nc[0] * nc[1] * nc[2]
    count = torch.bincount(cell, minlength=ncell)
    start = torch.cumsum(count, 0) - count
    most = int(count.max())
    table = torch.full((ncell, most), -1, dtype=torch.long, device=dev)
    sc = cell[order]
    table[sc, torch.arange(n, device=dev) - start[sc]] = order
    got = []
    ids = torch.arange(ncell, device=dev)
    cx, cy, cz = ids % nc[0], (ids // nc[0]) % nc[1], ids // (nc[0] * nc[1])
    chunk = max(1, int(3e7 // (most * most)))
    for dz in (-1, 0, 1):
        for dy in (-1, 0, 1):
            for dx in (-1, 0, 1):
                other = (((cz + dz) % nc[2]) * nc[1] + (cy + dy) % nc[1]) * nc[0] + (cx + dx) % nc[0]
                for a in range(0, ncell, chunk):
                    ti, tj = table[a:a + chunk, :, None], table[other[a:a + chunk]][:, None, :]
                    ok = (ti >= 0) & (tj > ti)
                    b, p, q = ok.nonzero(as_tuple=True)
                    i, j = ti[b, p, 0], tj[b, 0, q]
                    d = x[j] - x[i]
                    d = d - L * torch.round(d / L)
                    hit = (d * d).sum(-1) < rl * rl
                    got.append(torch.stack([i[hit], j[hit]]))
    return torch.cat(got, dim=1)


class _Exact:
    def __init__(self, case, systems, dev):
        self.case, self.dev = case, dev
        t = lambda a: torch.as_tensor(a, dtype=torch.float64, device=dev)
        self.sizes = [len(w["pos"]) for w in systems]
        self.x = t(np.concatenate([w["pos"] for w in systems]))
        self.v = t(np.concatenate([w["vel"] for w in systems]))
        self.m = t(np.concatenate([w["mass"] for w in systems]))[:, None]
        self.L = t(np.concatenate([np.broadcast_to(w["L"], (len(w["pos"]), 3)) for w in systems]))
        self.box = t(np.stack([w["L"] for w in systems]))
        self.sys = torch.repeat_interleave(torch.arange(len(systems), device=dev), torch.tensor(self.sizes, device=dev))
        self.rc = _constants(case)[2]
        if case["do"] == "static" or float(self.box.min()) < 2.2 * self.rc:
            self.skin = 0.0
        else:
            self.skin = min(0.25 * self.rc, 0.49 * float(self.box.min()) - self.rc)
        self.ref = None

    def fit(self, x):
        out = (x < 0) | (x > self.L)
        return torch.where(out, x - self.L * torch.floor(x / self.L), x)

    def neighbours(self, x):
        if self.ref is not None and self.skin > 0:
            d = x - self.ref
            d = d - self.L * torch.round(d / self.L)
            if 2.0 * float(d.square().sum(-1).max()) ** 0.5 < self.skin:
                return
        at, got = 0, []
        for n, box in zip(self.sizes, self.box):
            got.append(_pairs_of(x[at:at + n], box, self.rc + self.skin) + at)
            at += n
        self.ij, self.ref = torch.cat(got, dim=1), x.clone()

    def add(self, i, j, w, sign):
        out = torch.zeros((len(self.x),) + w.shape[1:], dtype=torch.float64, device=self.dev)
        out.index_add_(0, i, w)
        out.index_add_(0, j, w, alpha=sign)
        return out

    def by_system(self, where, w):
        out = torch.zeros((len(self.sizes),) + w.shape[1:], dtype=torch.float64, device=self.dev)
        return out.index_add_(0, self.sys[where], w)

    def evaluate(self, x):
        """Forces (eV/A), and per system potential energy, virial and stress."""
        self.neighbours(x)
        i, j = self.ij
        d = x[j] - x[i]
        d = d - self.L[i] * torch.round(d / self.L[i])
        r2 = d.square().sum(-1)
        near = r2 < self.rc * self.rc
        i, j, d, r2 = i[near], j[near], d[near], r2[near]
        pot = self.case.get("pot", "lj")
        every = torch.arange(len(x), device=self.dev)
        if pot == "lj":
            s6 = (SIGMA * SIGMA / r2) ** 3
            g = -48.0 * EPS / r2 * (s6 * s6 - 0.5 * s6)
            epot = self.by_system(i, 4.0 * EPS * (s6 * s6 - s6))
        else:
            r = r2.sqrt()
            rho_ij, c = self.density(r)
            rho = self.add(i, j, rho_ij, 1.0)
            phi = 1.0 / rho.sqrt()
            e, s = self.metal(r, phi[i] + phi[j])
            g = s / r
            epot = self.by_system(i, e) + self.by_system(every, -c * rho.sqrt())
        f = self.add(i, j, g[:, None] * d, -1.0)
        vir = self.by_system(i, -g * r2)
        stress = self.by_system(i, (-g[:, None, None] * d[:, :, None] * d[:, None, :]).reshape(-1, 9))
        return f, epot, vir, stress

    def density(self, r):
        pot = self.case["pot"]
        p = METALS[pot][1]
        if pot == "sc":
            return (p["a"] / r) ** p["m"], p["c"] * p["e"]
        if pot == "gupta":
            return torch.exp(-2.0 * p["q"] * (r - p["r0"]) / p["r0"]), p["B"]
        rd = r - p["d"]
        w = rd * rd * ((1.0 + p["B"] * rd / p["d"]) if pot == "fs" else (1.0 + p["B"] * p["B"] * rd * rd))
        return torch.where(r <= p["d"], w, torch.zeros_like(r)), p["A"]

    def metal(self, r, phi):
        """Pair energy, and the factor of the unit vector in the force on the first atom."""
        pot = self.case["pot"]
        p = METALS[pot][1]
        if pot == "sc":
            e = p["e"] * (p["a"] / r) ** p["n"]
            return e, -p["n"] * e / r + 0.5 * p["m"] * p["c"] * p["e"] * phi * (p["a"] / r) ** p["m"] / r
        if pot == "gupta":
            u = (r - p["r0"]) / p["r0"]
            ex = torch.exp(-p["p"] * u)
            return p["A"] * ex, -p["A"] * p["p"] / p["r0"] * ex + p["B"] * p["q"] / p["r0"] * phi * torch.exp(-2.0 * p["q"] * u)
        rc, rd = r - p["c"], r - p["d"]
        poly = p["c0"] + p["c1"] * r + p["c2"] * r * r
        dpoly = p["c1"] + 2.0 * p["c2"] * r
        if pot == "fs":
            mb = 2.0 * rd + 3.0 * p["B"] * rd * rd / p["d"]
        else:
            poly = poly + p["c3"] * r**3 + p["c4"] * r**4
            dpoly = dpoly + 3.0 * p["c3"] * r * r + 4.0 * p["c4"] * r**3
            mb = 2.0 * rd + 4.0 * p["B"] ** 2 * rd**3
        inside = r <= p["c"]
        zero = torch.zeros_like(r)
        e = torch.where(inside, rc * rc * poly, zero)
        s = torch.where(inside, 2.0 * rc * poly + rc * rc * dpoly, zero)
        return e, s - torch.where(r <= p["d"], 0.5 * p["A"] * phi * mb, zero)

    def thermo(self, step, v, epot, vir, stress):
        every = torch.arange(len(v), device=self.dev)
        kin = self.by_system(every, (0.5 * self.m * v * v).sum(-1)) * KIN2EV
        n = torch.tensor(self.sizes, dtype=torch.float64, device=self.dev)
        vol = self.box.prod(-1)
        pv = PRESS / vol
        p = self.by_system(every, self.m * v)
        cols = [torch.full_like(kin, float(step)), epot, kin, epot + kin, 2.0 / 3.0 * kin / (KB * n), vir, p[:, 0], p[:, 1],
                p[:, 2], vol, pv / 3.0 * vir, 2.0 / 3.0 * pv * kin, pv * (2.0 / 3.0 * kin + vir / 3.0)]
        out = torch.cat([torch.stack(cols, dim=1), stress], dim=1)
        return out if len(self.sizes) > 1 else out[0]

    def md(self, steps, dt, integ):
        fm = FORCEFACTOR / self.m
        x, v = self.x, self.v
        f, epot, vir, stress = self.evaluate(x)
        a = f * fm
        old = self.evaluate(self.fit(x - v * dt))[0] * fm if integ == "beeman" else None
        for _ in range(steps):
            if integ == "beeman":
                x = self.fit(x + v * dt + (2.0 / 3.0) * a * dt * dt - (1.0 / 6.0) * old * dt * dt)
            else:
                x = self.fit(x + v * dt + 0.5 * a * dt * dt)
            f, epot, vir, stress = self.evaluate(x)
            b = f * fm
            if integ == "beeman":
                v = v + (1.0 / 3.0) * b * dt + (5.0 / 6.0) * a * dt - (1.0 / 6.0) * old * dt
                old = a
            else:
                v = v + 0.5 * dt * (a + b)
            a = b
        return x, v, a, self.thermo(steps, v, epot, vir, stress)


def exact(case, seed):
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    systems = _systems(case, seed)
    E = _Exact(case, systems, dev)
    if case["do"] == "static":
        f, epot, vir, stress = E.evaluate(E.x)
        return dict(force=f, sums=torch.cat([epot, vir, stress[0]]))
    if case["do"] == "forces":
        f, epot, vir, stress = E.evaluate(E.x)
        return dict(acc=f * (FORCEFACTOR / E.m), thermo=E.thermo(0, E.v, epot, vir, stress))
    x, v, a, thermo = E.md(int(case["steps"]), _constants(case)[3], case["integ"])
    return dict(pos=x, vel=v, acc=a, thermo=thermo)
