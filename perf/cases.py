"""Timed cases: what programs have this framework do, at the sizes they do it.

Every case is one pass through the public entry points -- a stretch of
molecular dynamics on a kept ``Engine`` (alone, batched, bonded), a
differentiated trajectory, a descent, a whole ``Simulation.execute()`` -- with
inputs made from a seed by plain torch on the GPU.  ``exact`` restates the
same pass in 64 bits without this package's code.

Outputs.  Positions come back wrapped into the box, so a bead within rounding
of a face may come back on either side of it; passes on many beads therefore
return the velocities (which hold every force of the pass) and the thermo
values, small ones the positions as well.
"""

from __future__ import annotations

import math
import os
import shutil
import tempfile

import numpy as np
import torch

import beads_b200 as beads
from beads_b200.adjoint import trajectory_observables
from beads_b200.engine import Engine, ReplicaSpec

KB_NM_KJMOL = 0.00831446261815324
WCA = 2.0 ** (1.0 / 6.0)
POSITIONS_UP_TO = 8192  # beads: below, passes return positions too
THERMO = ("pair_pe", "bond_pe", "angle_pe", "dihedral_pe", "ke", "virial")

# Force fields: epsilon / sigma tables, cutoff, skin, time step, temperature,
# number density, units, whether the energy is shifted.
_SIG4 = np.array([0.9, 1.0, 1.05, 1.1])
FIELDS = {
    # single-type LJ fluid, reduced units
    "lj": dict(eps=np.array([[1.0]]), sig=np.array([[1.0]]), rc=2.5, skin=0.3, dt=0.005, t=1.0,
               rho=0.8442, units="reduced", shift=False, mass=1.0, share=[1.0]),
    # binary mixture in nm and kJ/mol, 80/20
    "mixture": dict(eps=np.array([[1.0, 0.7], [0.7, 0.5]]),
                    sig=np.array([[0.34, 0.32], [0.32, 0.30]]), rc=0.9, skin=0.1, dt=0.002,
                    t=120.0, rho=20.37, units="nm_kjmol", shift=True, mass=39.95,
                    share=[0.8, 0.2]),
    # the same mixture in reduced units, as it is fitted
    "fit": dict(eps=np.array([[1.0, 0.7], [0.7, 0.5]]),
                sig=np.array([[0.34, 0.32], [0.32, 0.30]]) / 0.34, rc=0.9 / 0.34, skin=0.3,
                dt=0.005, t=1.0, rho=0.8, units="reduced", shift=True, mass=1.0,
                share=[0.8, 0.2]),
    # four types: any table wider than two
    "four": dict(eps=np.sqrt(np.outer([1.0, 0.9, 1.1, 0.8], [1.0, 0.9, 1.1, 0.8])),
                 sig=0.5 * (_SIG4[:, None] + _SIG4[None, :]), rc=2.6, skin=0.3, dt=0.004, t=1.0,
                 rho=0.75, units="reduced", shift=True, mass=1.0, share=[0.4, 0.3, 0.2, 0.1]),
    # bead-spring chains: purely repulsive pairs, harmonic bonds, angles, dihedrals
    "melt": dict(eps=np.array([[1.0]]), sig=np.array([[1.0]]), rc=WCA, skin=0.3, dt=0.005, t=1.0,
                 rho=0.85, units="reduced", shift=True, mass=1.0, share=[1.0]),
}
BONDED = dict(bond_k=500.0, bond_r0=0.97, angle_k=5.0, angle_theta0=150.0, dihedral_k=1.0)


def listed():
    return [
        # a few hundred beads: the shortest calls, where launches are all there is
        {"name": "lj_250", "do": "md", "field": "lj", "n": 250, "steps": 32, "calls": 1,
         "every": 1, "sort": 10, "cap": 512, "thermostat": False},
        # the small benchmark fluid, lists checked every 10 steps
        {"name": "lj_4096", "do": "md", "field": "lj", "n": 4096, "steps": 40, "calls": 1,
         "every": 10, "sort": 10, "cap": 512, "thermostat": False},
        # four particle types, energies written every 10 steps
        {"name": "four_types_20k", "do": "md", "field": "four", "n": 20011, "steps": 10, "calls": 3,
         "every": 1, "sort": 10, "cap": 192, "thermostat": False},
        # a medium binary mixture with a thermostat, odd size
        {"name": "mixture_100k", "do": "md", "field": "mixture", "n": 100003, "steps": 50,
         "calls": 1, "every": 1, "sort": 1, "cap": 128, "thermostat": True},
        # the headline benchmark: the million-bead mixture between two outputs
        {"name": "mixture_1m", "do": "md", "field": "mixture", "n": 1048576, "steps": 40, "calls": 1,
         "every": 1, "sort": 1, "cap": 128, "thermostat": True},
        # many independent boxes of uneven size stepped together
        {"name": "replicas_128", "do": "md", "field": "lj", "n": 0, "replicas": 128, "n_min": 256,
         "n_max": 32768, "steps": 20, "calls": 1, "every": 1, "sort": 10, "cap": 160,
         "thermostat": True},
        # bead-spring melts propagated from given configurations
        {"name": "melt_6k", "do": "melt", "chains": 61, "beads": 100, "steps": 8},
        {"name": "melt_200k", "do": "melt", "chains": 1000, "beads": 200, "steps": 8},
        # differentiated trajectories: forward, replay and reverse sweep
        {"name": "fit_2x600", "do": "fit", "replicas": 2, "n": 600, "steps": 16, "record": 9,
         "checkpoint": 8},
        {"name": "fit_16x4096", "do": "fit", "replicas": 16, "n": 4096, "steps": 40, "record": 33,
         "checkpoint": 20},
        # capped steepest descent of a disordered start, then its energies and forces
        {"name": "relax_30k", "do": "relax", "field": "mixture", "n": 30011, "steps": 60,
         "cap": 256},
        # the drop-in path: spec in, files out, engine set up and torn down
        {"name": "execute_4096", "do": "execute", "field": "lj", "n": 4096, "steps": 60,
         "thermo": 20},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    do = rng.choice(["md", "md", "md", "replicas", "melt", "fit", "relax", "execute"])
    if do == "md":
        field = rng.choice(["lj", "mixture", "four"])
        return {"do": "md", "field": field, "n": _log_int(rng, 200, 600_000),
                "steps": rng.choice([8, 16, 25, 32]), "calls": rng.choice([1, 2]),
                "every": rng.choice([1, 1, 5]), "sort": rng.choice([1, 10]), "cap": 192,
                "thermostat": rng.random() < 0.5}
    if do == "replicas":
        return {"do": "md", "field": rng.choice(["lj", "fit"]), "n": 0,
                "replicas": _log_int(rng, 4, 128), "n_min": 256, "n_max": _log_int(rng, 2000, 32768),
                "steps": rng.choice([8, 16, 20]), "calls": 1, "every": 1, "sort": 10, "cap": 192,
                "thermostat": True}
    if do == "melt":
        return {"do": "melt", "chains": _log_int(rng, 20, 1000), "beads": rng.randrange(20, 201),
                "steps": rng.choice([3, 5, 8])}
    if do == "fit":
        steps = rng.choice([12, 20, 30])
        return {"do": "fit", "replicas": rng.randrange(1, 17), "n": _log_int(rng, 600, 4096),
                "steps": steps, "record": steps - rng.randrange(0, 6),
                "checkpoint": rng.choice([0, 7, 10])}
    if do == "relax":
        return {"do": "relax", "field": rng.choice(["lj", "mixture"]), "n": _log_int(rng, 1000, 60000),
                "steps": rng.choice([20, 40, 60]), "cap": 256}
    return {"do": "execute", "field": rng.choice(["lj", "four"]), "n": _log_int(rng, 500, 20000),
            "steps": rng.choice([30, 60]), "thermo": rng.choice([10, 15])}


# -- plain torch molecular dynamics -------------------------------------------
# Neighbour matrices (row i: its partners, padded with n), LJ and chain forces
# in any precision; used to make inputs and, in 64 bits, as the reference.


def _delta(a, b, box):
    d = a - b
    return d - box * torch.round(d / box)


def _neighbors(x, box, reach, chain=0, apart=0):
    """[n, M] partner indices within `reach`; partners at most `apart` places
    along the same chain of `chain` beads are left out."""
    n, dev = x.shape[0], x.device
    nc = [max(1, int(float(b) // reach)) for b in box]
    ncv = torch.tensor(nc, device=dev)
    k = torch.minimum((torch.remainder(x, box) / box * ncv).long(), ncv - 1)
    cell = k[:, 0] + nc[0] * (k[:, 1] + nc[1] * k[:, 2])
    count = torch.bincount(cell, minlength=nc[0] * nc[1] * nc[2])
    order = torch.argsort(cell, stable=True)
    first = torch.cumsum(count, 0) - count
    table = torch.full((count.numel(), int(count.max())), n, dtype=torch.long, device=dev)
    table[cell[order], torch.arange(n, device=dev) - first[cell[order]]] = order
    steps = [[0] if c == 1 else [0, 1] if c == 2 else [-1, 0, 1] for c in nc]
    xe = torch.cat([x, x.new_zeros(1, 3)])
    rows, at = [], 0
    chunk = max(1, 40_000_000 // (27 * table.shape[1]))
    while at < n:
        i = torch.arange(at, min(n, at + chunk), device=dev)
        cand = []
        for dz in steps[2]:
            for dy in steps[1]:
                for dx in steps[0]:
                    s = torch.remainder(k[i] + torch.tensor([dx, dy, dz], device=dev), ncv)
                    cand.append(table[s[:, 0] + nc[0] * (s[:, 1] + nc[1] * s[:, 2])])
        cand = torch.cat(cand, 1)
        ok = (_delta(x[i][:, None], xe[cand], box).square().sum(-1) < reach * reach)
        ok &= (cand < n) & (cand != i[:, None])
        if apart:
            ok &= ~((cand // chain == i[:, None] // chain) & ((cand - i[:, None]).abs() <= apart))
        place = torch.cumsum(ok, 1) - 1
        out = torch.full((i.numel(), max(1, int(ok.sum(1).max()))), n, dtype=torch.long, device=dev)
        r, c = torch.nonzero(ok, as_tuple=True)
        out[r, place[r, c]] = cand[r, c]
        rows.append(out)
        at += chunk
    wide = max(r.shape[1] for r in rows)
    return torch.cat([torch.nn.functional.pad(r, (0, wide - r.shape[1]), value=n) for r in rows])


def _lj_rows(x, i, nb, types, box, eps, sig, rc, shift, floor):
    n = x.shape[0]
    j = torch.where(nb < n, nb, i[:, None])
    d = _delta(x[i][:, None], x[j], box)
    r2 = d.square().sum(-1)
    inside = (nb < n) & (r2 < rc * rc)
    e, s2 = eps[types[i][:, None], types[j]], sig[types[i][:, None], types[j]].square()
    r2 = torch.where(inside, r2, torch.ones_like(r2))
    if floor:
        r2 = torch.maximum(r2, floor * s2)
    s6 = (s2 / r2) ** 3
    fs = torch.where(inside, 24.0 * e / r2 * (2.0 * s6 * s6 - s6), torch.zeros_like(r2))
    u = 4.0 * e * (s6 * s6 - s6)
    if shift:
        c6 = (s2 / (rc * rc)) ** 3
        u = u - 4.0 * e * (c6 * c6 - c6)
    u = torch.where(inside, u, torch.zeros_like(r2))
    return (fs[..., None] * d).sum(1), 0.5 * u.sum(1), 0.5 * (fs * r2).sum(1)


def _lj(x, nb, types, box, eps, sig, rc, shift, floor=0.0):
    """Forces, energy and virial of each bead; r^2 held to >= floor sigma^2."""
    parts = []
    chunk = x.shape[0] if x.requires_grad or sig.requires_grad else max(1, 12_000_000 // nb.shape[1])
    for at in range(0, x.shape[0], chunk):
        i = torch.arange(at, min(x.shape[0], at + chunk), device=x.device)
        parts.append(_lj_rows(x, i, nb[i], types, box, eps, sig, rc, shift, floor))
    return tuple(torch.cat(p) for p in zip(*parts))


def _chain_energy(x, box, chain, stiff=1.0):
    """(bond, angle, dihedral) energies of chains of `chain` beads."""
    b = _delta(x.view(-1, chain, 3)[:, 1:], x.view(-1, chain, 3)[:, :-1], box)
    length = b.norm(dim=-1)
    eb = 0.5 * BONDED["bond_k"] * (length - BONDED["bond_r0"]).square().sum()
    p, q = -b[:, :-1], b[:, 1:]
    theta = torch.atan2(torch.linalg.cross(p, q).norm(dim=-1), (p * q).sum(-1))
    ea = 0.5 * stiff * BONDED["angle_k"] * (theta - math.radians(BONDED["angle_theta0"])).square().sum()
    m, o = torch.linalg.cross(b[:, :-2], b[:, 1:-1]), torch.linalg.cross(b[:, 1:-1], b[:, 2:])
    cos = (m * o).sum(-1) / (m.norm(dim=-1) * o.norm(dim=-1))
    return eb, ea, BONDED["dihedral_k"] * (1.0 + cos).sum()


def _chain_forces(x, box, chain, stiff=1.0):
    """Forces, the three energies and the virial sum r.F of the bonded terms."""
    y = x.detach().clone().requires_grad_(True)
    scale = torch.ones((), dtype=x.dtype, device=x.device, requires_grad=True)
    # the arms as minimum-image differences of unwrapped chains, so that a
    # common scale of them gives the virial
    b = _delta(y.view(-1, chain, 3)[:, 1:], y.view(-1, chain, 3)[:, :-1], box)
    line = torch.cat([torch.zeros_like(b[:, :1]), torch.cumsum(b, 1)], 1) * scale
    far = torch.full((3,), 1e9, dtype=x.dtype, device=x.device)
    e = _chain_energy(line.reshape(-1, 3), far, chain, stiff)
    gy, gs = torch.autograd.grad(sum(e), [y, scale])
    return -gy, [t.detach() for t in e], -gs


# -- inputs ----------------------------------------------------------------------


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _velocities(n, kt, mass, g):
    v = torch.randn(n, 3, generator=g, device="cuda", dtype=torch.float64) * math.sqrt(kt / mass)
    return v - v.mean(0)


def _wrapped(x, box):
    """float32 coordinates inside [0, box)."""
    top = box.to(torch.float32)
    y = torch.remainder(x, box).to(torch.float32)
    return torch.where(y >= top, torch.nextafter(top, torch.zeros_like(top)), y).clamp_(min=0.0)


def _fluid(n, f, g, quench=30, rho=None):
    """A disordered fluid of n beads: beads scattered off the sites of a
    lattice, then moved apart.  Returns positions, types (0-based) and box."""
    length = max((n / (rho or f["rho"])) ** (1.0 / 3.0), 2.0 * (f["rc"] + f["skin"]) * 1.0001)
    length = float(np.float32(length))
    side = math.ceil(n ** (1.0 / 3.0) - 1e-9)
    a = length / side
    pick = torch.randperm(side ** 3, generator=g, device="cuda")[:n].sort().values
    x = torch.stack([pick // (side * side), pick // side % side, pick % side], 1) + 0.5
    x = (x + 0.13 * torch.randn(n, 3, generator=g, device="cuda", dtype=torch.float64)) * a
    box = torch.full((3,), length, dtype=torch.float64, device="cuda")
    edges = torch.cumsum(torch.tensor(f["share"], dtype=torch.float64), 0) * n
    types = torch.bucketize(torch.randperm(n, generator=g, device="cuda").double() + 0.5,
                            edges[:-1].cuda())
    eps, sig = (torch.tensor(f[k], dtype=torch.float64, device="cuda") for k in ("eps", "sig"))
    s = float(f["sig"].max())
    reach = 1.6 * s
    for it in range(quench):
        if it % 6 == 0:
            nb = _neighbors(x, box, reach)
        force = _lj(x, nb, types, box, eps, sig, 1.4 * s, False, floor=0.49)[0]
        norm = force.norm(dim=1, keepdim=True)
        x = x + 0.02 * s * force / torch.clamp(norm, min=60.0 * float(f["eps"].max()) / s)
    return _wrapped(x, box), types, box


def _chains(chains, beads, f, g):
    """Freely rotating chains with angles about 150 degrees at random places,
    pushed apart; float32 positions and the box."""
    n = chains * beads
    length = float(np.float32((n / f["rho"]) ** (1.0 / 3.0)))
    box = torch.full((3,), length, dtype=torch.float64, device="cuda")

    def randn(*shape):
        return torch.randn(*shape, generator=g, device="cuda", dtype=torch.float64)

    step = torch.nn.functional.normalize(randn(chains, 3), dim=1)
    path = [torch.rand(chains, 3, generator=g, device="cuda", dtype=torch.float64) * length]
    for _ in range(beads - 1):
        path.append(path[-1] + 0.97 * step)
        side = torch.nn.functional.normalize(torch.linalg.cross(step, randn(chains, 3)), dim=1)
        bend = torch.deg2rad(30.0 + 8.0 * randn(chains, 1))
        step = step * torch.cos(bend) + side * torch.sin(bend)
    x = torch.stack(path, 1).reshape(n, 3)
    types = torch.zeros(n, dtype=torch.long, device="cuda")
    eps, sig = (torch.tensor(f[k], dtype=torch.float64, device="cuda") for k in ("eps", "sig"))
    for it in range(320):
        if it % 8 == 0:
            nb = _neighbors(x, box, 1.45, beads, 2)
        # soft pairs that chains can pass through first, then as hard as they are;
        # angles stiffer than the model's, away from the straight ones at which
        # its dihedral forces diverge
        force = _lj(x, nb, types, box, eps, sig, WCA, False, floor=0.75 if it < 160 else 0.6)[0]
        force = min(1.0, 0.01 * 1.035 ** it) * force + _chain_forces(x, box, beads, 20.0)[0]
        x = x + 0.02 * force / torch.clamp(force.norm(dim=1, keepdim=True),
                                           min=60.0 if it < 240 else 200.0)
    return _wrapped(x, box), box


def _field_spec(f, x, v, types, box, case, **more):
    n = x.shape[0]
    return ReplicaSpec(
        positions=x.cpu().numpy(), velocities=v.to(torch.float32).cpu().numpy(),
        types=(types + 1).to(torch.int32).cpu().numpy(),
        box_bound=np.stack([np.zeros(3), box.cpu().numpy()]).astype(np.float32),
        epsilon=f["eps"], sigma=f["sig"], cutoff=f["rc"], dt=f["dt"], units=f["units"],
        masses=np.full(n, f["mass"], np.float32), shift=f["shift"], cutoff_buffer=f["skin"],
        rebuild_check_every=case.get("every", 1), sort_every_rebuild=case.get("sort", 10),
        max_neighbors=case.get("cap", 128),
        thermostat=(f["t"], _tau(f)) if case.get("thermostat") else None, **more)


def _tau(f):
    return 0.1 if f["units"] == "nm_kjmol" else 1.0


def _kt(f):
    return f["t"] * (KB_NM_KJMOL if f["units"] == "nm_kjmol" else 1.0)


def _sizes(case):
    """Beads of every replica of a case: log-uniform, evenly spread, for a batch."""
    if case["do"] == "fit":
        return [case["n"]] * case["replicas"]
    if not case.get("replicas"):
        return [case["n"]]
    lo, hi, m = math.log(case["n_min"]), math.log(case["n_max"]), case["replicas"]
    return [int(math.exp(lo + (hi - lo) * ((k * 61 + 17) % m + 0.37) / m)) for k in range(m)]


def _replicas(case, seed):
    """(positions, velocities, types, box) of every replica."""
    f = FIELDS[case.get("field", "fit")]
    g = _gen(seed)
    out = []
    for k, n in enumerate(_sizes(case)):
        rho = f["rho"] * (0.92 + 0.12 * (k * 29 % 64) / 64) if len(_sizes(case)) > 1 else None
        x, types, box = _fluid(n, f, g, quench=12 if case["do"] == "relax" else 30, rho=rho)
        out.append((x, _velocities(n, _kt(f), f["mass"], g).to(torch.float32), types, box))
    return out


def _pinned(n):
    return torch.zeros(n, 3, dtype=torch.float32).pin_memory()


def _thermo(rows):
    return [[float(row[k]) for k in THERMO] for row in rows]


# -- the cases -------------------------------------------------------------------


def prepare(case, seed):
    return globals()["_prepare_" + case["do"]](case, seed)


def run(state):
    return globals()["_run_" + state["do"]](state)


def exact(case, seed):
    return globals()["_exact_" + case["do"]](case, seed)


def _prepare_md(case, seed):
    f = FIELDS[case["field"]]
    rep = _replicas(case, seed)
    eng = Engine([_field_spec(f, *r, case) for r in rep])
    x0 = torch.cat([r[0] for r in rep]).cpu().numpy()
    v0 = torch.cat([r[1] for r in rep]).cpu().numpy()
    # a program keeps its engine: schedule chosen and steps captured, then the
    # start of this run put in place
    eng.run(case["steps"], case["steps"])
    eng.upload_all(x0, v0)
    n = x0.shape[0]
    return {"do": "md", "eng": eng, "steps": case["steps"], "calls": case["calls"], "n": n,
            "x": _pinned(n), "v": _pinned(n)}


def _run_md(s):
    eng, rows = s["eng"], []
    for _ in range(s["calls"]):
        rows.append(_thermo(eng.run(s["steps"], s["steps"])))
    eng.download_all(s["x"].numpy(), s["v"].numpy())
    out = {"thermo": rows if s["n"] <= POSITIONS_UP_TO else rows[-1][:4], "velocities": s["v"]}
    if s["n"] <= POSITIONS_UP_TO:
        out["positions"] = s["x"]
    return out


class _Exact:
    """One replica's velocity-Verlet dynamics in 64 bits."""

    def __init__(self, f, x, v, types, box, thermostat, chain=0):
        self.f, self.box, self.types, self.chain = f, box.double(), types, chain
        self.x, self.v = x.double(), v.double()
        self.eps, self.sig = (torch.tensor(f[k], dtype=torch.float64, device="cuda")
                              for k in ("eps", "sig"))
        self.thermostat, self.skin, self.origin = thermostat, 0.3 * f["rc"], None
        self.evaluate()

    def neighbours(self):
        x = self.x.detach()
        if self.origin is not None:
            moved = _delta(x, self.origin, self.box).norm(dim=1).max()
            if float(moved) < 0.5 * self.skin:
                return
        self.origin = x.clone()
        self.nb = _neighbors(x, self.box, self.f["rc"] + self.skin, self.chain,
                             2 if self.chain else 0)

    def evaluate(self):
        self.neighbours()
        f = self.f
        self.force, e, w = _lj(self.x, self.nb, self.types, self.box, self.eps, self.sig, f["rc"],
                               f["shift"])
        self.pe, self.virial = [e.sum(), 0.0, 0.0, 0.0], w.sum()
        if self.chain:
            fb, eb, wb = _chain_forces(self.x, self.box, self.chain)
            self.force, self.virial = self.force + fb, self.virial + wb
            self.pe[1:] = eb

    def step(self):
        f = self.f
        h = 0.5 * f["dt"] / f["mass"]
        u = self.v + h * self.force
        self.x = self.x + f["dt"] * u
        self.evaluate()
        self.v = u + h * self.force
        if self.thermostat:
            k = self.kinetic()
            target = 0.5 * (3 * self.x.shape[0] - 3) * _kt(f)
            self.v = self.v * torch.sqrt(1.0 + f["dt"] / _tau(f) * (target / k - 1.0))

    def kinetic(self):
        return 0.5 * self.f["mass"] * self.v.square().sum()

    def row(self):
        return [float(p) for p in self.pe] + [float(self.kinetic()), float(self.virial)]


def _exact_md(case, seed):
    f = FIELDS[case["field"]]
    sims = [_Exact(f, x, v, types, box, case["thermostat"])
            for x, v, types, box in _replicas(case, seed)]
    rows = []
    for _ in range(case["calls"]):
        for s in sims:
            for _ in range(case["steps"]):
                s.step()
        rows.append([s.row() for s in sims])
    n = sum(s.x.shape[0] for s in sims)
    out = {"thermo": rows if n <= POSITIONS_UP_TO else rows[-1][:4],
           "velocities": torch.cat([s.v for s in sims])}
    if n <= POSITIONS_UP_TO:
        out["positions"] = torch.cat([torch.remainder(s.x, s.box) for s in sims])
    return out


def _melt_terms(chains, beads):
    first = (np.arange(chains) * beads + 1)[:, None]

    def terms(width):
        at = first + np.arange(beads - width + 1)[None, :]
        cols = [(at + k).ravel() for k in range(width)]
        return np.stack(cols + [np.ones(at.size, np.int64)], 1).astype(np.uint32)

    return terms(2), terms(3), terms(4)


def _melt_start(case, seed):
    f, g = FIELDS["melt"], _gen(seed)
    x, box = _chains(case["chains"], case["beads"], f, g)
    v = _velocities(x.shape[0], _kt(f), f["mass"], g).to(torch.float32)
    return x, v, torch.zeros(x.shape[0], dtype=torch.long, device="cuda"), box


def _prepare_melt(case, seed):
    x, v, types, box = _melt_start(case, seed)
    bonds, angles, dihedrals = _melt_terms(case["chains"], case["beads"])
    spec = _field_spec(
        FIELDS["melt"], x, v, types, box, {"thermostat": True}, bonds=bonds, angles=angles,
        dihedrals=dihedrals, exclusion_distance=2, dihedral_d=[1], dihedral_n=[1],
        molecule_ids=np.repeat(np.arange(1, case["chains"] + 1, dtype=np.uint32), case["beads"]),
        **{k: [b] for k, b in BONDED.items()})
    eng = Engine(spec)
    eng.run(case["steps"], case["steps"])
    n = x.shape[0]
    hx, hv = _pinned(n), _pinned(n)
    hx.copy_(x)
    hv.copy_(v)
    return {"do": "melt", "eng": eng, "steps": case["steps"], "n": n, "x0": hx, "v0": hv,
            "x": _pinned(n), "v": _pinned(n)}


def _run_melt(s):
    eng = s["eng"]
    eng.upload_all(s["x0"].numpy(), s["v0"].numpy())
    row = _thermo(eng.run(s["steps"], s["steps"]))
    eng.download_all(s["x"].numpy(), s["v"].numpy())
    out = {"thermo": row, "velocities": s["v"]}
    if s["n"] <= POSITIONS_UP_TO:
        out["positions"] = s["x"]
    return out


def _exact_melt(case, seed):
    s = _Exact(FIELDS["melt"], *_melt_start(case, seed), True, chain=case["beads"])
    for _ in range(case["steps"]):
        s.step()
    out = {"thermo": [s.row()], "velocities": s.v}
    if s.x.shape[0] <= POSITIONS_UP_TO:
        out["positions"] = torch.remainder(s.x, s.box)
    return out


def _prepare_fit(case, seed):
    f = FIELDS["fit"]
    rep = _replicas(case, seed)
    eng = Engine([_field_spec(f, *r, {"thermostat": True, "cap": 192}) for r in rep])
    eng.run(8)
    g = _gen(seed + 1)
    eps, sig = (torch.tensor(f[k], dtype=torch.float32).requires_grad_(True) for k in ("eps", "sig"))
    s = {"do": "fit", "eng": eng, "case": case, "eps": eps, "sig": sig,
         "x": torch.cat([r[0] for r in rep]).cpu().requires_grad_(True),
         "v": torch.cat([r[1] for r in rep]).cpu().requires_grad_(True),
         "volume": torch.tensor([float(r[3].prod()) for r in rep]),
         "target": (torch.rand(2, case["replicas"], generator=g, device="cuda")).cpu()}
    _run_fit(s)  # schedule chosen, segments captured
    return s


def _fit_loss(obs, n, volume, target):
    """Energy per bead and pressure of the recorded window against targets."""
    pe = obs[:, :, 0].mean(0) / n
    press = ((2.0 * obs[:, :, 2] + obs[:, :, 1]) / (3.0 * volume)).mean(0)
    return ((pe + 5.0 + target[0]) ** 2 + (press - target[1]) ** 2).sum()


def _run_fit(s):
    c = s["case"]
    leaves = [s["eps"], s["sig"], s["x"], s["v"]]
    obs = trajectory_observables(s["eng"], *leaves, steps=c["steps"], record_from=c["record"],
                                 checkpoint_every=c["checkpoint"]).to(torch.float32)
    grads = torch.autograd.grad(_fit_loss(obs, c["n"], s["volume"], s["target"]), leaves)
    return {"observables": obs.detach(), "grads": list(grads)}


def _exact_fit(case, seed):
    beads_total = case["replicas"] * case["n"]
    if beads_total * case["steps"] > 100_000:
        return None  # the 64-bit graph of every step would not fit
    f = FIELDS["fit"]
    eps, sig = (torch.tensor(f[k], dtype=torch.float32, device="cuda").double().requires_grad_(True)
                for k in ("eps", "sig"))
    rep = _replicas(case, seed)
    target = torch.rand(2, case["replicas"], generator=_gen(seed + 1), device="cuda")
    rows, xs, vs = [], [], []
    for x, v, types, box in rep:
        xs.append(x.double().requires_grad_(True))
        vs.append(v.double().requires_grad_(True))
        s = _Exact(f, x, v, types, box, True)
        s.x, s.v, s.eps, s.sig = xs[-1], vs[-1], eps, sig
        s.evaluate()
        obs = []
        for m in range(case["steps"] + 1):
            if m:
                s.step()
            if m >= case["record"]:
                obs.append(torch.stack([s.pe[0], s.virial, s.kinetic()]))
        rows.append(torch.stack(obs))
    obs = torch.stack(rows, 1)
    volume = torch.stack([r[3].prod() for r in rep])
    leaves = [eps, sig, *xs, *vs]
    g = torch.autograd.grad(_fit_loss(obs, case["n"], volume, target.double()), leaves)
    m = case["replicas"]
    # one entry of the tables per ordered pair, as the dynamics reads them
    return {"observables": obs.detach().cpu(),
            "grads": [g[0].cpu(), g[1].cpu(), torch.cat(g[2:2 + m]).cpu(),
                      torch.cat(g[2 + m:]).cpu()]}


def _descent(f):
    """dmax and fref of the capped descent."""
    s, e = float(f["sig"].max()), float(f["eps"].max())
    return 0.01 * s, 70.0 * e / s


def _prepare_relax(case, seed):
    f = FIELDS[case["field"]]
    (x, v, types, box), = _replicas(case, seed)
    eng = Engine(_field_spec(f, x, v, types, box, {"cap": case["cap"]}))
    hx = _pinned(x.shape[0])
    hx.copy_(x)
    return {"do": "relax", "eng": eng, "x0": hx, "steps": case["steps"], "move": _descent(f)}


def _run_relax(s):
    eng = s["eng"]
    eng.upload_all(s["x0"].numpy())
    eng.minimize(s["steps"], *s["move"])
    row = _thermo(eng.eval())
    return {"energies": [row[0][0], row[0][5]], "forces": eng.state()["forces"]}


def _exact_relax(case, seed):
    f = FIELDS[case["field"]]
    (x, v, types, box), = _replicas(case, seed)
    s = _Exact(f, x, v, types, box, False)
    dmax, fref = _descent(f)
    for _ in range(case["steps"]):
        s.neighbours()
        force = _lj(s.x, s.nb, types, s.box, s.eps, s.sig, f["rc"], f["shift"], floor=0.49)[0]
        s.x = s.x + dmax * force / torch.clamp(force.norm(dim=1, keepdim=True), min=fref)
    s.evaluate()
    return {"energies": [float(s.pe[0]), float(s.virial)], "forces": s.force}


def _prepare_execute(case, seed):
    f = FIELDS[case["field"]]
    (x, v, types, box), = _replicas(case, seed)
    return {"do": "execute", "case": case, "x": x.cpu().numpy(), "v": v.cpu().numpy(),
            "types": (types + 1).to(torch.int32).cpu().numpy(), "box": box.cpu().numpy()}


def _run_execute(s):
    c = s["case"]
    f = FIELDS[c["field"]]
    n, length = c["n"], s["box"]
    system = beads.System(units=f["units"], box_bound=np.stack([np.zeros(3), length]),
                          positions=s["x"], velocities=s["v"], types=s["types"],
                          masses=np.full(n, f["mass"]))
    ff = beads.ForceField()
    ff.pair_style("lj", cutoff=f["rc"], shift=f["shift"])
    for i in range(len(f["share"])):
        for j in range(i, len(f["share"])):
            ff.pair_coeff("lj", type_i=i + 1, type_j=j + 1, epsilon=float(f["eps"][i, j]),
                          sigma=float(f["sig"][i, j]))
    sim = beads.Simulation(system=system, forcefield=ff,
                           dynamics=beads.Dynamics("velocity_verlet", dt=f["dt"]))
    folder = tempfile.mkdtemp(prefix="beads_")
    try:
        at = os.path.join(folder, "run")
        sim.set_runsteps(c["steps"]).set_neighbor(cutoff_buffer=f["skin"], max_neighbors=256)
        sim.set_thermo(every=c["thermo"], prefix=at).save_final_state(prefix=at)
        sim.set_logging(echo="none")
        sim.execute()
        files = {os.path.splitext(p)[1]: os.path.join(folder, p) for p in os.listdir(folder)}
        with open(files[".csv"]) as h:
            head = h.readline().strip().split(",")
            rows = np.loadtxt(h, delimiter=",", ndmin=2)
        rest = next(p for e, p in files.items() if e != ".csv")
        state = beads.io.read_state(rest)
        order = np.argsort(state["tags"])
    finally:
        shutil.rmtree(folder)
    return {"thermo": [[float(r[head.index(k)]) for k in ("pe", "ke")] for r in rows],
            "velocities": np.asarray(state["velocities"], np.float32)[order],
            "unwrapped": (np.asarray(state["positions"], np.float64)
                          + np.asarray(state["images"]) * length).astype(np.float32)[order]}


def _exact_execute(case, seed):
    f = FIELDS[case["field"]]
    (x, v, types, box), = _replicas(case, seed)
    s = _Exact(f, x, v, types, box, False)
    rows = [[float(s.pe[0]), float(s.kinetic())]]
    for m in range(1, case["steps"] + 1):
        s.step()
        if m % case["thermo"] == 0:
            rows.append([float(s.pe[0]), float(s.kinetic())])
    return {"thermo": rows, "velocities": s.v, "unwrapped": s.x}


# -- work ------------------------------------------------------------------------


def work(case):
    """Bytes: a step reads and writes every bead's position and velocity (48 B;
    twice for a differentiated step).  Flops: a step evaluates every pair
    inside the cutoff once (35 with both beads' forces), 30 per bead for the
    integration, 150 per bonded term; a reverse step 80 more a pair."""
    f = FIELDS[case.get("field", "fit" if case["do"] == "fit" else "melt")]
    n = case["chains"] * case["beads"] if case["do"] == "melt" else sum(_sizes(case))
    steps = case["steps"] * case.get("calls", 1)
    per_bead = 0.5 * f["rho"] * 4.0 / 3.0 * math.pi * f["rc"] ** 3
    flops = steps * n * (35.0 * per_bead + 30.0)
    if case["do"] == "melt":
        flops += steps * n * 3 * 150.0
    if case["do"] == "fit":
        flops += steps * n * 80.0 * per_bead
    return {"bytes": 48.0 * n * (steps if case["do"] != "fit" else 2 * steps), "flops": flops}
