"""The calls this framework's speed is followed on, each through its public entry points.

Four kinds, by what a user's program does with the step engine:

  md      one engine of one system: a stride of MD steps, then the state read
          back (a trajectory frame, a checkpoint)
  batch   one engine of many systems of uneven sizes: a stride of steps of all
          of them, then every system's state
  forces  energies by group, virial and forces at given positions: the call a
          minimiser's line search and a report make
  mesh    reciprocal-space PME on the caller's own device buffers

`listed` holds the cases by name, `draw` gives more of the same ranges:
2,000-30,000 atoms (the sizes of the ensemble workload; NPT boxes up to
100,000), cubes, rhombic dodecahedra and truncated octahedra of TIP3P, with or
without an ff14SB helix, meshes by the library's rule (odd and ragged sizes).

`exact` restates each call in 64-bit torch, from the definitions: smooth PME
with order-5 splines, Lennard-Jones with the Lorentz-Berthelot rules, the
bonded terms, LFMiddle and Verlet with constraints, and the counter-based
thermostat noise.
"""

from __future__ import annotations

import ctypes
import functools
import math
import sys
from pathlib import Path

import numpy as np
import torch

sys.path.insert(0, str(Path(__file__).resolve().parent.parent / "making-it-rain-webgpu_b200"))

from mdb200 import abi, peptide, steploop, synth  # noqa: E402

CUTOFF, EWALD_TOLERANCE = 1.0, 5e-4
TIME_STEP, TEMPERATURE, FRICTION = 0.002, 300.0, 1.0
ATOMS_PER_NM3 = 3 * synth.WATER_DENSITY_PER_NM3
CELL_VOLUME = {"cube": 1.0, "dodecahedron": math.sqrt(0.5), "octahedron": 4 * math.sqrt(3) / 9}
# List settings (skin, sort cell, tile atoms, prune at rebuild, inner skin) as the
# library's autotuner returns them: for one system alone, and in a batch by size bucket.
TUNED_ALONE = (0.5, 0.25, 8, 2, 0.1)
TUNED_BATCH = {10: (0.25, 0.2, 8, 2, -1.0), 11: (0.5, 0.2, 8, 2, 0.1), 12: (0.15, 0.25, 8, 2, -1.0),
               13: (0.25, 0.2, 8, 2, 0.06), 14: (0.4, 0.25, 8, 2, 0.1)}


def listed():
    return [
        # a 2,652-atom TIP3P box, mesh 30^3: the smallest system anybody runs; launches and latency count
        dict(name="md water 2652", kind="md", shape="cube", solute="none", residues=0, width=3.0, mesh=30, steps=30,
             tuned=False, integrator="lfmiddle", friction=FRICTION, frequency=0),
        # the same box size without a thermostat: the energy-conservation runs
        dict(name="md water verlet", kind="md", shape="dodecahedron", solute="none", residues=0, width=3.7, mesh=0,
             steps=30, tuned=False, integrator="verlet", friction=0.0, frequency=0),
        # a solvated, salted Ala20 helix as a new user runs it, at the library's default list settings
        dict(name="md peptide 12k", kind="md", shape="cube", solute="helix", residues=20, width=5.0, mesh=50, steps=30,
             tuned=False, integrator="lfmiddle", friction=FRICTION, frequency=0),
        # a 60-residue chain in a truncated octahedron, about 27,000 atoms, list settings tuned: production of one system
        dict(name="md octahedron 27k", kind="md", shape="octahedron", solute="coil", residues=60, width=0.0, mesh=0,
             steps=30, tuned=True, integrator="lfmiddle", friction=FRICTION, frequency=0),
        # 100,000 atoms at constant pressure, a volume move every 25 steps
        dict(name="md npt 100k", kind="md", shape="cube", solute="none", residues=0, width=10.0, mesh=0, steps=25,
             tuned=True, integrator="lfmiddle", friction=FRICTION, frequency=25),
        # eight small systems in one engine, defaults: a handful of replicas
        dict(name="batch small 8", kind="batch", systems=8, low=2000, high=5000, steps=30, tuned=False, frequency=0),
        # 64 systems of 2,000-30,000 atoms in one engine, tuned: the ensemble workload
        dict(name="batch ensemble 64", kind="batch", systems=64, low=2000, high=30000, steps=20, tuned=True, frequency=0),
        # sixteen of them at constant pressure: every system's volume moves in rounds
        dict(name="batch npt 16", kind="batch", systems=16, low=2000, high=30000, steps=25, tuned=True, frequency=25),
        # one evaluation of a small box: a step of a minimiser's line search
        dict(name="forces water 2652", kind="forces", shape="cube", solute="none", residues=0, width=3.0, mesh=30,
             tuned=False),
        # one evaluation of the 27,000-atom system: a report
        dict(name="forces octahedron 27k", kind="forces", shape="octahedron", solute="coil", residues=60, width=0.0,
             mesh=0, tuned=True),
        # the mesh part alone at the 12,000-atom size, on the caller's stream
        dict(name="mesh 50", kind="mesh", shape="cube", atoms=12276, width=5.0, mesh_x=50, mesh_y=50, mesh_z=50),
        # and at the largest mesh it takes, not a cube
        dict(name="mesh 64 ragged", kind="mesh", shape="octahedron", atoms=26211, width=7.0, mesh_x=64, mesh_y=63,
             mesh_z=60),
    ]


def draw(rng):
    kind = rng.choice(["md", "md", "md", "batch", "batch", "forces", "mesh"])
    if kind == "batch":
        count = round(math.exp(rng.uniform(math.log(2), math.log(32))))
        low = round(math.exp(rng.uniform(math.log(2000), math.log(8000))))
        high = round(low * math.exp(rng.uniform(0.1, math.log(30000 / low))))
        return dict(kind=kind, systems=count, low=low, high=high, steps=rng.randint(10, 25),
                    tuned=rng.random() < 0.7, frequency=rng.choice([0, 0, 25]))
    shape = rng.choice(sorted(CELL_VOLUME))
    atoms = math.exp(rng.uniform(math.log(2300), math.log(30000)))
    width = round((atoms / (ATOMS_PER_NM3 * CELL_VOLUME[shape])) ** (1 / 3), 2)
    if kind == "mesh":
        smooth = [n for n in range(20, 65) if _smooth(n)]
        mesh = [rng.choice(smooth) for _ in range(3)]
        return dict(kind=kind, shape=shape, atoms=round(atoms), width=width, mesh_x=mesh[0], mesh_y=mesh[1],
                    mesh_z=mesh[2])
    residues = rng.choice([0, 0, 10, 20, 30])
    box = synth.box_vectors(shape, width)
    while residues and 2 * peptide.bounding_radius(_helix(residues)[1]) + 1.0 > _narrowest(box):
        residues -= 10
    case = dict(kind=kind, shape=shape, solute="helix" if residues else "none", residues=residues, width=width, mesh=0,
                tuned=rng.random() < 0.5)
    if kind == "md":
        verlet = rng.random() < 0.2
        case.update(steps=rng.randint(12, 30), integrator="verlet" if verlet else "lfmiddle",
                    friction=0.0 if verlet else rng.choice([FRICTION, FRICTION, 5.0]),
                    frequency=0 if verlet else rng.choice([0, 0, 25]))
    return case


# ------------------------------------------------------------------ systems --
def _smooth(n: int) -> bool:
    for p in (2, 3, 5, 7):
        while n % p == 0:
            n //= p
    return n == 1


def _narrowest(box) -> float:
    a, b, c = box
    v = abs(np.linalg.det(box))
    return float(min(v / np.linalg.norm(np.cross(p, q)) for p, q in ((b, c), (c, a), (a, b))))


@functools.lru_cache(maxsize=None)
def _helix(residues: int):
    return peptide.helix(["ALA"] * residues)


@functools.lru_cache(maxsize=None)
def _coil():
    return peptide.coil()


def _one_system(case, seed: int):
    """The case's system and its start: molecules laid out and turned, and velocities drawn, by the seed."""
    barostat = (1.0, TEMPERATURE, case["frequency"]) if case.get("frequency") else None
    grid = (case["mesh"],) * 3
    if case["solute"] == "none":
        return synth.water_box(width=case["width"], shape=case["shape"], seed=seed, grid=grid, barostat=barostat)
    solute, xyz = _coil() if case["solute"] == "coil" else _helix(case["residues"])
    width = case["width"] or 2.0 * peptide.bounding_radius(xyz) + 1.0
    return synth.solvated(solute, xyz, width=width, shape=case["shape"], seed=seed, grid=grid, barostat=barostat)


def _batch_plan(case):
    """Sizes of a batch: log-uniform steps from low to high, cubes and dodecahedra in turn, every other one with a
    helix where one fits at 1.0 nm padding."""
    plan = []
    for k in range(case["systems"]):
        atoms = case["low"] * (case["high"] / case["low"]) ** ((k + 0.5) / case["systems"])
        shape = ("cube", "dodecahedron")[k % 2]
        width = (atoms / (ATOMS_PER_NM3 * CELL_VOLUME[shape])) ** (1 / 3)
        width = max(width, 2.02 * CUTOFF / _narrowest(synth.box_vectors(shape, 1.0)))
        residues = (0, 0, 10, 20, 0, 0, 30, 40)[k % 8]
        while residues and 2 * peptide.bounding_radius(_helix(residues)[1]) + 1.0 > _narrowest(
                synth.box_vectors(shape, width)):
            residues -= 10
        plan.append(dict(shape=shape, solute="helix" if residues else "none", residues=residues, width=width, mesh=0,
                         frequency=case["frequency"]))
    return plan


def _members(case, seed: int):
    if case["kind"] == "batch":
        return [_one_system(m, seed * 1000 + k) for k, m in enumerate(_batch_plan(case))]
    return [_one_system(case, seed)]


def _options(case, systems, seed: int):
    tuning = None
    if case["tuned"]:
        if case["kind"] == "batch":
            last = max(TUNED_BATCH)
            tuning = [TUNED_BATCH[min(last, steploop.size_bucket(s.particle_count))] for s in systems]
        else:
            tuning = [TUNED_ALONE]
    return steploop.RunOptions(time_step=TIME_STEP, temperature=TEMPERATURE, friction=case.get("friction", FRICTION),
                               seed=seed, integrator=case.get("integrator", "lfmiddle"), tuning=tuning)


def _charges(case, seed: int):
    """Positions (n, 3) and charges of a mesh case: points uniform in the cell, alternating charges, neutral."""
    rng = np.random.default_rng(seed)
    n, box = case["atoms"], synth.box_vectors(case["shape"], case["width"])
    positions = rng.uniform(size=(n, 3)) @ box
    charges = np.where(np.arange(n) % 3 == 0, -0.8, 0.4) * rng.uniform(0.9, 1.1, size=n)
    return positions, charges - charges.mean(), box


# ----------------------------------------------------------- prepare and run --
def prepare(case, seed):
    if case["kind"] == "mesh":
        positions, charges, box = _charges(case, seed)
        n = case["atoms"]
        state = dict(kind="mesh", n=n, positions=torch.from_numpy(positions).cuda(), charges=torch.from_numpy(charges).cuda(),
                     forces=torch.empty((n, 3), dtype=torch.float64, device="cuda"),
                     energy=torch.empty(1, dtype=torch.float64, device="cuda"),
                     box=(ctypes.c_double * 9)(*box.reshape(-1)),
                     mesh=(ctypes.c_int32 * 3)(case["mesh_x"], case["mesh_y"], case["mesh_z"]), library=abi.load())
        return state
    members = _members(case, seed)
    systems, states = [m[0] for m in members], [m[1] for m in members]
    loop = steploop.StepLoop.batch(systems, states, _options(case, systems, seed))
    state = dict(kind=case["kind"], loop=loop, steps=case.get("steps", 0))
    if case["kind"] == "forces":
        # the trial configurations of a search, near the state's
        rng = np.random.default_rng(seed)
        state["positions"] = states[0].positions + rng.normal(scale=1e-3, size=states[0].positions.shape)
    return state


def run(state):
    if state["kind"] == "mesh":
        status = state["library"].mdb_reciprocal_noalloc(
            state["n"], state["positions"].data_ptr(), state["charges"].data_ptr(), state["box"], _ewald_alpha(),
            state["mesh"], state["forces"].data_ptr(), state["energy"].data_ptr(),
            torch.cuda.current_stream().cuda_stream)
        assert status == abi.OK
        return {"forces": state["forces"], "energy": state["energy"]}
    loop = state["loop"]
    if state["kind"] == "forces":
        loop.set_positions(state["positions"])
        energies, forces = loop.evaluate()
        return {"energies": np.array([energies[k] for k in ENERGIES]), "virial": np.array(energies["virial"]),
                "forces": forces}
    loop.run(state["steps"])
    return {"positions": np.concatenate([loop.positions(k) for k in range(loop.system_count)]),
           "velocities": np.concatenate([loop.velocities(k) for k in range(loop.system_count)])}


ENERGIES = ("bond", "angle", "torsion", "direct_coulomb", "direct_lj", "exclusion_correction", "exceptions",
            "dispersion", "reciprocal_mesh", "self_energy", "net_charge", "direct_group", "reciprocal_group",
            "potential")


# --------------------------------------------------------------------- work --
def work(case):
    """Per step: every atom's state (position, velocity, residual: 48 bytes) read and written, its parameters (20
    bytes) read; 74 flop per unique pair inside the cutoff, 1,000 per atom for the splines (125 points, charge and
    three force components), 2.5 K log2 K per real transform each way, 200 per atom for the integrator.  A forces
    pass reads positions and parameters and writes forces."""
    def flops(atoms, mesh_points):
        pairs = 0.5 * atoms * ATOMS_PER_NM3 * 4.18879 * CUTOFF**3
        return 74 * pairs + 1000 * atoms + 5 * mesh_points * math.log2(mesh_points)

    if case["kind"] == "mesh":
        k = case["mesh_x"] * case["mesh_y"] * case["mesh_z"]
        return {"bytes": 56 * case["atoms"], "flops": 1000 * case["atoms"] + 5 * k * math.log2(k)}
    plan = _batch_plan(case) if case["kind"] == "batch" else [case]
    atoms = ops = 0.0
    for m in plan:
        width = m["width"] or 7.1
        n = ATOMS_PER_NM3 * CELL_VOLUME[m["shape"]] * width**3
        k = n / ATOMS_PER_NM3 / CELL_VOLUME[m["shape"]] * 1000  # mesh spacing of 0.1 nm over the diagonal
        atoms += n
        ops += flops(n, k)
    if case["kind"] == "forces":
        return {"bytes": 68 * atoms, "flops": ops}
    return {"bytes": case["steps"] * (2 * 48 + 20) * atoms, "flops": case["steps"] * (ops + 200 * atoms)}


def tolerance(case):
    """About four times what the same pass shows with its pair forces summed in another order (32-atom instead of 8-atom
    tiles), in relative 2-norm: forces 2e-7, virial 1e-7; mesh forces 8e-7 (the f32 transforms; against `exact`).  A
    trajectory multiplies such a difference by e in about every 10.5 steps of the first hundred from these starts:
    velocities were apart by 2.5e-5 at step 40, 6e-5 at 50, 1e-4 at 60, 5e-4 at 80 and 2e-3 at 100, single atoms by up
    to a hundred times that, and two passes in a row on one state go through twice the steps."""
    if case["kind"] == "forces":
        return {"rel": 1e-6}
    if case["kind"] == "mesh":
        return {"rel": 3e-6}
    rel = 1e-4 * math.exp(max(0.0, 2 * case["steps"] - 40) / 10.5)
    return {"rel": rel, "max": min(0.9, 200 * rel)}


# ------------------------------------------------------- the same in 64 bits --
KE = 138.93545764498457  # kJ/mol nm / e^2
KB = 0.008314462618153242


def _ewald_alpha() -> float:
    return math.sqrt(-math.log(2 * EWALD_TOLERANCE)) / CUTOFF


def _mesh_for(system, box):
    grid = [int(g) for g in system.nonbonded.grid]
    for k in range(3):
        if grid[k] <= 0:
            grid[k] = max(6, math.ceil(2 * _ewald_alpha() * box[k][k] / (3 * EWALD_TOLERANCE**0.2)))
            while not _smooth(grid[k]):
                grid[k] += 1
    return grid


def _image(d, box):
    """Nearest image by reduction against c, then b, then a."""
    for k in (2, 1, 0):
        d = d - torch.round(d[..., k:k + 1] / box[k, k]) * box[k]
    return d


def _splines(x, box, grid):
    """Mesh indices (n, 3, 5), weights and derivatives of the order-5 cardinal B-spline."""
    u = torch.linalg.solve(box.T, x.T).T * torch.tensor(grid, dtype=x.dtype, device=x.device)
    cell = torch.floor(u)
    w = u - cell
    m = [w, 1 - w]  # M_2 at w, w + 1
    for order in (3, 4, 5):
        previous, low = m, m
        zero = torch.zeros_like(w)
        at = lambda v, j: v[j] if 0 <= j < len(v) else zero  # noqa: E731
        m = [((w + j) * at(low, j) + (order - w - j) * at(low, j - 1)) / (order - 1) for j in range(order)]
    derivative = [at(previous, j) - at(previous, j - 1) for j in range(5)]
    index = torch.stack([cell.long() - j for j in range(5)], -1) % torch.tensor(grid, device=x.device)[:, None]
    return index, torch.stack(m, -1), torch.stack(derivative, -1)


def _mesh_sum(x, q, box, grid, alpha):
    """Energy, forces and virial of the smooth PME mesh sum."""
    device, f8 = x.device, torch.float64
    index, w, dw = _splines(x, box, grid)
    K = torch.tensor(grid, dtype=f8, device=device)
    flat = ((index[:, 0, :, None, None] * grid[1] + index[:, 1, None, :, None]) * grid[2] + index[:, 2, None, None, :])
    weight = w[:, 0, :, None, None] * w[:, 1, None, :, None] * w[:, 2, None, None, :]
    mesh = torch.zeros(grid[0] * grid[1] * grid[2], dtype=f8, device=device)
    mesh.index_add_(0, flat.reshape(-1), (q[:, None, None, None] * weight).reshape(-1))
    Q = torch.fft.fftn(mesh.view(*grid))
    signed = [torch.fft.fftfreq(g, 1.0 / g, dtype=f8, device=device) for g in grid]
    m = torch.stack(torch.meshgrid(*signed, indexing="ij"), -1)
    k = 2 * math.pi * m @ torch.linalg.inv(box).T  # rows of inv(box).T: the reciprocal vectors
    k2 = (k * k).sum(-1)
    k2[0, 0, 0] = 1.0
    moduli = []
    for axis in range(3):
        n = grid[axis]
        j = torch.arange(n, dtype=f8, device=device)
        phase = [2 * math.pi * j * t / n for t in range(4)]
        knots = (1 / 24, 11 / 24, 11 / 24, 1 / 24)
        re = sum(c * torch.cos(p) for c, p in zip(knots, phase))
        im = sum(c * torch.sin(p) for c, p in zip(knots, phase))
        b = re * re + im * im
        b = torch.where(b < 1e-7, 0.5 * (torch.roll(b, 1) + torch.roll(b, -1)), b)
        moduli.append(b)
    volume = torch.linalg.det(box).abs()
    factor = KE * 2 * math.pi / volume * torch.exp(-k2 / (4 * alpha * alpha)) / (
        k2 * moduli[0][:, None, None] * moduli[1][None, :, None] * moduli[2][None, None, :])
    factor[0, 0, 0] = 0.0
    ek = factor * (Q.real**2 + Q.imag**2)
    energy = ek.sum()
    c = 2 * (1 / k2 + 1 / (4 * alpha * alpha))
    virial = torch.eye(3, dtype=f8, device=device) * energy - torch.einsum("xyz,xyza,xyzb->ab", ek * c, k, k)
    phi = torch.fft.ifftn(2 * factor * Q).real.reshape(-1) * mesh.numel()
    local = phi[flat]
    du = torch.stack([(local * dw[:, 0, :, None, None] * w[:, 1, None, :, None] * w[:, 2, None, None, :]).sum((1, 2, 3)),
                      (local * w[:, 0, :, None, None] * dw[:, 1, None, :, None] * w[:, 2, None, None, :]).sum((1, 2, 3)),
                      (local * w[:, 0, :, None, None] * w[:, 1, None, :, None] * dw[:, 2, None, None, :]).sum((1, 2, 3))],
                     -1)
    forces = -q[:, None] * ((du * K) @ torch.linalg.inv(box).T)
    return energy, forces, virial


class _Reference:
    """Forces and energies of one system in 64-bit torch."""

    SKIN = 0.2

    def __init__(self, system, box, device):
        f8 = lambda a: torch.as_tensor(np.asarray(a, dtype=np.float64), device=device)  # noqa: E731
        i8 = lambda a: torch.as_tensor(np.asarray(a, dtype=np.int64), device=device)  # noqa: E731
        nb = system.nonbonded
        self.device, self.box, self.alpha = device, f8(box), _ewald_alpha()
        self.grid = _mesh_for(system, box)
        self.q, self.sigma, self.epsilon = f8(nb.charge), f8(nb.sigma), f8(nb.epsilon)
        self.n = len(nb.charge)
        p, s = i8(nb.exception_p1), i8(nb.exception_p2)
        self.except_i, self.except_j = p, s
        self.excluded = torch.sort(torch.minimum(p, s) * self.n + torch.maximum(p, s)).values
        self.except_qq, self.except_sigma, self.except_eps = (f8(nb.exception_charge_prod), f8(nb.exception_sigma),
                                                              f8(nb.exception_epsilon))
        self.bonds = self.angles = self.torsions = None
        if system.bonds is not None:
            a, b, r0, k = system.bonds
            self.bonds = i8(a), i8(b), f8(r0), f8(k)
        if system.angles is not None:
            a, b, c, t0, k = system.angles
            self.angles = i8(a), i8(b), i8(c), f8(t0), f8(k)
        if system.torsions is not None:
            a, b, c, d, n, phase, k = system.torsions
            self.torsions = i8(a), i8(b), i8(c), i8(d), f8(n), f8(phase), f8(k)
        self.pairs_at = None
        volume = float(torch.linalg.det(self.box).abs())
        classes = {}
        for sg, ep in zip(np.asarray(nb.sigma).tolist(), np.asarray(nb.epsilon).tolist()):
            classes[sg, ep] = classes.get((sg, ep), 0) + 1
        items, s6, s12 = list(classes.items()), 0.0, 0.0
        for x, ((s1, e1), c1) in enumerate(items):
            for y, ((s2, e2), c2) in enumerate(items[x:]):
                many = c1 * (c1 + 1) / 2 if y == 0 else c1 * c2
                sg6 = (0.5 * (s1 + s2)) ** 6
                s6 += many * math.sqrt(e1 * e2) * sg6
                s12 += many * math.sqrt(e1 * e2) * sg6 * sg6
        count = self.n * (self.n + 1) / 2
        self.dispersion = 8 * math.pi * self.n**2 / volume * (s12 / count / (9 * CUTOFF**9) - s6 / count / (3 * CUTOFF**3))
        self.self_energy = -KE * self.alpha * float((self.q**2).sum()) / math.sqrt(math.pi)
        self.net_charge = -math.pi * float(self.q.sum()) ** 2 * KE / (2 * self.alpha**2 * volume)

    def _pair_list(self, x):
        if self.pairs_at is not None and (x - self.pairs_at).norm(dim=1).max() < 0.5 * self.SKIN:
            return
        step = max(1, 30_000_000 // self.n)
        found = []
        for lo in range(0, self.n, step):
            d = _image(x[None, lo:] - x[lo:lo + step, None], self.box)
            i, j = torch.nonzero((d * d).sum(-1) < (CUTOFF + self.SKIN) ** 2, as_tuple=True)
            keep = j > i
            found.append(torch.stack([i[keep] + lo, j[keep] + lo]))
        i, j = torch.cat(found, 1)
        if len(self.excluded):
            key = i * self.n + j
            at = torch.searchsorted(self.excluded, key).clamp(max=len(self.excluded) - 1)
            keep = self.excluded[at] != key
            i, j = i[keep], j[keep]
        self.i, self.j, self.pairs_at = i, j, x.clone()

    def _pairwise(self, f, virial, i, j, d, slope):
        """Adds slope(r) = (dE/dr)/r along d = x_j - x_i of each pair to the forces and the virial."""
        g = slope[:, None] * d
        f.index_add_(0, i, g)
        f.index_add_(0, j, -g)
        virial -= d.T @ g

    def evaluate(self, x):
        f, virial, e, alpha = torch.zeros_like(x), torch.zeros_like(self.box), {}, self.alpha
        two = 2 * alpha / math.sqrt(math.pi)
        self._pair_list(x)
        d = _image(x[self.j] - x[self.i], self.box)
        near = (d * d).sum(-1) < CUTOFF**2
        i, j, d = self.i[near], self.j[near], d[near]
        r = d.norm(dim=1)
        qq = KE * self.q[i] * self.q[j]
        eps4 = 4 * torch.sqrt(self.epsilon[i] * self.epsilon[j])
        s6 = (0.5 * (self.sigma[i] + self.sigma[j]) / r) ** 6
        screened = torch.erfc(alpha * r)
        e["direct_coulomb"] = (qq * screened / r).sum()
        e["direct_lj"] = (eps4 * (s6 * s6 - s6)).sum()
        slope = -qq * (screened / r + two * torch.exp(-((alpha * r) ** 2))) / r**2 + eps4 * (6 * s6 - 12 * s6 * s6) / r**2
        self._pairwise(f, virial, i, j, d, slope)
        i, j = self.except_i, self.except_j
        d = _image(x[j] - x[i], self.box)
        r = d.norm(dim=1)
        qq, own = KE * self.q[i] * self.q[j], KE * self.except_qq
        s6 = (self.except_sigma / r) ** 6
        inside = torch.erf(alpha * r)
        e["exclusion_correction"] = -(qq * inside / r).sum()
        e["exceptions"] = (own / r + 4 * self.except_eps * (s6 * s6 - s6)).sum()
        slope = (qq * (inside / r - two * torch.exp(-((alpha * r) ** 2))) - own / r
                 + 4 * self.except_eps * (6 * s6 - 12 * s6 * s6)) / r**2
        self._pairwise(f, virial, i, j, d, slope)
        e.update(self._bonded(x, f, virial))
        mesh, force, w = _mesh_sum(x, self.q, self.box, self.grid, alpha)
        f += force
        virial += w + (self.dispersion + self.net_charge) * torch.eye(3, dtype=x.dtype, device=x.device)
        e["reciprocal_mesh"], e["dispersion"] = mesh, self.dispersion
        e["self_energy"], e["net_charge"] = self.self_energy, self.net_charge
        e = {k: float(v) for k, v in e.items()}
        e["direct_group"] = (e["direct_coulomb"] + e["direct_lj"] + e["exclusion_correction"] + e["exceptions"]
                             + e["dispersion"])
        e["reciprocal_group"] = e["reciprocal_mesh"] + e["self_energy"] + e["net_charge"]
        e["potential"] = e["bond"] + e["angle"] + e["torsion"] + e["direct_group"] + e["reciprocal_group"]
        return e, f, virial

    def _bonded(self, x, f, virial):
        e = dict(bond=0.0, angle=0.0, torsion=0.0)
        if self.bonds is None and self.angles is None and self.torsions is None:
            return e
        with torch.enable_grad():
            x = x.detach().clone().requires_grad_(True)
            if self.bonds is not None:
                a, b, r0, k = self.bonds
                e["bond"] = (0.5 * k * ((x[b] - x[a]).norm(dim=1) - r0) ** 2).sum()
            if self.angles is not None:
                a, b, c, t0, k = self.angles
                u, v = x[a] - x[b], x[c] - x[b]
                theta = torch.atan2(torch.linalg.cross(u, v).norm(dim=1), (u * v).sum(1))
                e["angle"] = (0.5 * k * (theta - t0) ** 2).sum()
            if self.torsions is not None:
                a, b, c, d, n, phase, k = self.torsions
                b1, b2, b3 = x[b] - x[a], x[c] - x[b], x[d] - x[c]
                n1, n2 = torch.linalg.cross(b1, b2), torch.linalg.cross(b2, b3)
                phi = torch.atan2(b2.norm(dim=1) * (b1 * n2).sum(1), (n1 * n2).sum(1))
                e["torsion"] = (k * (1 + torch.cos(n * phi - phase))).sum()
            g, = torch.autograd.grad(sum(v for v in e.values()), x)
        f -= g
        virial -= x.detach().T @ g
        return {k: float(v.detach()) if torch.is_tensor(v) else v for k, v in e.items()}


def _noise(n: int, step: int, seed: int):
    """Standard normals (n, 3) of the thermostat: Threefry-2x32-20 (Salmon et al. 2011) of the particle and the step,
    then Box-Muller."""
    def threefry(c0, c1, k0, k1):
        ks = [np.uint32(k0), np.uint32(k1), np.uint32(0x1BD11BDA ^ k0 ^ k1)]
        x0, x1 = c0 + ks[0], c1 + ks[1]
        for r in range(20):
            turn = (13, 15, 26, 6, 17, 29, 16, 24)[r % 8]
            x0 = x0 + x1
            x1 = ((x1 << np.uint32(turn)) | (x1 >> np.uint32(32 - turn))) ^ x0
            if r % 4 == 3:
                x0 = x0 + ks[(r // 4 + 1) % 3]
                x1 = x1 + ks[(r // 4 + 2) % 3] + np.uint32(r // 4 + 1)
        return x0, x1

    with np.errstate(over="ignore"):
        b0, b1 = threefry(np.arange(2 * n, dtype=np.uint32), np.full(2 * n, step, dtype=np.uint32), seed, 0x9E3779B9)
    u0, u1 = (((b >> np.uint32(9)).astype(np.float64) + 0.5) * 2.0**-23 for b in (b0, b1))
    radius, angle = np.sqrt(-2 * np.log(u0)), 2 * math.pi * u1
    pair = np.stack([radius * np.cos(angle), radius * np.sin(angle)], -1).reshape(n, 4)
    return pair[:, :3]


def _trajectory(system, state, case, seed: int, device):
    """Positions and velocities after the case's steps from the start state."""
    ref = _Reference(system, state.box, device)
    f8 = lambda a: torch.as_tensor(np.asarray(a, dtype=np.float64), device=device)  # noqa: E731
    x, v, mass = f8(state.positions), f8(state.velocities), f8(system.masses)[:, None]
    ci, cj = (torch.as_tensor(np.asarray(c, dtype=np.int64), device=device)
              for c in (system.constraint_p1, system.constraint_p2))
    d2 = f8(system.constraint_distance) ** 2
    reduced = 0.5 / (1 / mass[ci, 0] + 1 / mass[cj, 0])
    dt, verlet = TIME_STEP, case.get("integrator") == "verlet"
    friction = case.get("friction", FRICTION)
    keep, kick = math.exp(-dt * friction), math.sqrt(1 - math.exp(-2 * dt * friction))

    def spread(target, bond, amount):
        g = bond * amount[:, None]
        target.index_add_(0, ci, g / mass[ci])
        target.index_add_(0, cj, -g / mass[cj])

    for step in range(case["steps"]):
        v = v - (mass * v).sum(0) / mass.sum()
        v = v + dt * ref.evaluate(x)[1] / mass
        bond = x[ci] - x[cj]
        length2 = (bond * bond).sum(1)
        if verlet:
            trial = x + dt * v
        else:
            for _ in range(120):  # mass-weighted sweeps over all constraints at once, a factor of about 0.8 each
                spread(v, bond, -2 * reduced * ((v[ci] - v[cj]) * bond).sum(1) / length2)
            trial = x + 0.5 * dt * v
            v = keep * v + kick * torch.sqrt(KB * TEMPERATURE / mass) * f8(_noise(len(x), step, seed))
            trial = trial + 0.5 * dt * v
        end = trial.clone()
        for _ in range(120):
            now = end[ci] - end[cj]
            spread(end, bond, reduced * (d2 - (now * now).sum(1)) / (now * bond).sum(1))
        v = (end - x) / dt if verlet else v + (end - trial) / dt
        x = end
    return x, v


def exact(case, seed):
    device = "cuda" if torch.cuda.is_available() else "cpu"
    if case["kind"] == "mesh":
        positions, charges, box = _charges(case, seed)
        energy, forces, _ = _mesh_sum(torch.as_tensor(positions, device=device), torch.as_tensor(charges, device=device),
                                      torch.as_tensor(box, device=device), [case["mesh_x"], case["mesh_y"], case["mesh_z"]],
                                      _ewald_alpha())
        return {"forces": forces, "energy": energy.reshape(1)}
    if case["kind"] == "forces":
        (system, state), = _members(case, seed)
        rng = np.random.default_rng(seed)
        x = state.positions + rng.normal(scale=1e-3, size=state.positions.shape)
        e, f, virial = _Reference(system, state.box, device).evaluate(torch.as_tensor(x, device=device))
        return {"energies": np.array([e[k] for k in ENERGIES]), "virial": virial.reshape(-1).cpu().numpy(),
                "forces": f.cpu().numpy()}
    # a volume move hangs on an accept or reject that is not a computed number; the large ensembles take minutes
    if case["frequency"] or case.get("systems", 1) * case["steps"] > 400:
        return None
    ends = [_trajectory(*member, case, seed, device) for member in _members(case, seed)]
    # velocities after tens of steps carry the trajectory's own growth of rounding; positions barely do
    return {"positions": torch.cat([x for x, _ in ends]).cpu().numpy(), "velocities": None}
