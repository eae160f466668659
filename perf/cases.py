"""The measured cases of the MD engine: what a user's program asks of it, over the sizes, boxes and
options the package's configurations cover.

A case is one of four calls:

  run       advance a system some steps and read the state back, with an energy report where a
            program logs one (the production loop: a block of steps, a log line, a frame)
  evaluate  forces and energies of given coordinates (re-scoring a frame, checking a structure)
  minimise  steepest descent from a raw structure, as before every simulation
  batch     many uneven systems advanced together

Inputs are synthetic TIP3P water boxes and solvated chains (`rainmd_b200.synthetic`): the topology,
the lattice sites and the solute belong to the case; the seed sets the waters' orientations and
displacements, relaxed here by rigid-body descent (without the engine, so that every version of
the engine starts from the same numbers), the velocities and the thermostat's seed.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from rainmd_b200 import synthetic
from rainmd_b200.simulation import BatchSimulation, GpuSimulation
from rainmd_b200.topology import build_system

KE = 138.935456          # kJ/mol nm / e^2
KB = 0.008314462618      # kJ/mol/K
TEMPERATURE = 300.0
TIMESTEP = 0.002
DEVICE = "cuda" if torch.cuda.is_available() else "cpu"
WATER_VOLUME = 18.0154 * 1.66053906660e-3 / 0.997  # nm^3 a molecule


def _run(atoms, steps, block, *, chain=0, box="cubic", pressure=None, order=4, solver=1, cutoff=0.9, skin=0.25,
         grid="1A", energy=True):
    return {"kind": "run", "atoms": atoms, "chain": chain, "box": box, "pressure": pressure, "steps": steps,
            "block": block, "order": order, "solver": solver, "cutoff": cutoff, "skin": skin, "grid": grid,
            "energy": energy}


def _evaluate(atoms, *, chain=0, box="cubic", order=4, cutoff=0.9, skin=0.25, grid="1A"):
    return {"kind": "evaluate", "atoms": atoms, "chain": chain, "box": box, "order": order, "solver": 1,
            "cutoff": cutoff, "skin": skin, "grid": grid}


def listed():
    return [
        # one frame of the reference's published 1,190-atom system scored: the smallest call
        {"name": "evaluate-1190", **_evaluate(1190, chain=22, skin=0.15)},
        # a viewer stepping a small box a few steps a frame
        {"name": "stepping-2854", **_run(2854, 5, 5, skin=0.15, energy=False)},
        # the reference's published configuration: 1,190 atoms, NPT, a volume move every 25 steps
        {"name": "npt-1190", **_run(1190, 50, 25, chain=22, pressure=1.0, skin=0.15)},
        # a small water box in NVT
        {"name": "nvt-2854", **_run(2854, 50, 50)},
        # a truncated octahedron, spline order 5
        {"name": "octahedron-5001", **_run(5001, 50, 50, box="octahedron", order=5, skin=0.15)},
        # the engine's defaults: SHAKE, order 5, 1 nm cutoff, derived skin and grid
        {"name": "defaults-9002", **_run(9002, 50, 0, chain=200, order=5, solver=0, cutoff=1.0, skin=0.0, grid="derived")},
        # the benchmark's box in NPT
        {"name": "npt-23558", **_run(23558, 50, 25, pressure=1.0)},
        # a frame of that size scored
        {"name": "evaluate-23558", **_evaluate(23558)},
        # a raw structure of that size relaxed
        {"name": "minimise-23558", "kind": "minimise", "atoms": 23558, "chain": 300, "box": "cubic", "order": 4,
         "solver": 1, "cutoff": 0.9, "skin": 0.25, "grid": "1A", "iterations": 10},
        # a large box in NVT
        {"name": "nvt-99999", **_run(99999, 50, 50)},
        # the largest configured size, a chain in water in NPT
        {"name": "npt-250000", **_run(250000, 25, 25, chain=300, pressure=1.0)},
        # uneven solvated chains in one handle
        {"name": "batch-24", "kind": "batch", "count": 24, "low": 1000, "high": 12000, "pressure": None, "steps": 50,
         "block": 50, "order": 4, "solver": 1, "cutoff": 0.9, "skin": 0.15, "grid": "1A"},
    ]


def draw(rng):
    kind = rng.choices(["run", "evaluate", "minimise", "batch"], [6, 2, 1, 1])[0]
    order, grid = rng.choice([4, 4, 5]), rng.choice(["1A", "1A", "derived"])
    if kind == "batch":
        low = rng.randint(1000, 2500)
        return {"kind": "batch", "count": rng.randint(2, 24), "low": low, "high": rng.randint(2 * low, 12000),
                "pressure": rng.choice([None, 1.0]), "steps": rng.randint(20, 50), "block": 25, "order": order,
                "solver": rng.choice([1, 1, 0]), "cutoff": 0.9, "skin": 0.15, "grid": "1A"}
    largest = {"run": 250000, "evaluate": 100000, "minimise": 30000}[kind]
    atoms = int(round(math.exp(rng.uniform(math.log(1190), math.log(largest)))))
    box = rng.choice(["cubic", "cubic", "octahedron"]) if atoms >= 2000 else "cubic"
    if box == "octahedron":
        atoms -= atoms % 3  # waters alone
    chain = rng.randint(20, min(300, atoms // 20)) if box == "cubic" and rng.random() < 0.5 else 0
    cutoff = rng.choice([0.8, 0.9, 1.0]) if atoms >= 4000 else rng.choice([0.8, 0.9])
    skin = round(rng.uniform(0.1, 0.3), 2) if atoms >= 4000 else 0.12
    if kind == "evaluate":
        return _evaluate(atoms, chain=chain, box=box, order=order, cutoff=cutoff, skin=skin, grid=grid)
    if kind == "minimise":
        return {"kind": "minimise", "atoms": atoms, "chain": chain, "box": box, "order": order, "solver": 1,
                "cutoff": cutoff, "skin": skin, "grid": grid, "iterations": rng.randint(5, 12)}
    steps = max(10, min(rng.randint(20, 50), 6000000 // atoms))
    return _run(atoms, steps, rng.choice([0, 25, steps]), chain=chain, box=box, pressure=rng.choice([None, 1.0]),
                order=order, solver=rng.choice([1, 1, 0]), cutoff=cutoff, skin=skin, grid=grid,
                energy=rng.random() < 0.8)


# ------------------------------------------------------------------------------- inputs
def _transformable(n):
    while True:
        r = n
        for p in (2, 3, 5):
            while r % p == 0:
                r //= p
        if r == 1:
            return n
        n += 1


def _octahedron(n_water):
    """Box vectors of a truncated octahedron holding n_water at liquid density, and the sites: the
    cell cut n x n x n is a body-centred cubic lattice."""
    length = (n_water * WATER_VOLUME / (4.0 * math.sqrt(3.0) / 9.0)) ** (1.0 / 3.0)
    box = length * np.array([[1.0, 0.0, 0.0], [1 / 3, 2 * math.sqrt(2) / 3, 0.0], [-1 / 3, math.sqrt(2) / 3,
                                                                                    math.sqrt(6) / 3]])
    n = int(math.ceil(n_water ** (1.0 / 3.0) - 1e-9))
    g = (np.arange(n) + 0.5) / n
    sites = np.array(np.meshgrid(g, g, g, indexing="ij")).reshape(3, -1).T @ box
    return box.reshape(-1), sites


@functools.lru_cache(maxsize=40)
def _structure(atoms, chain, box, cutoff, structure_seed):
    """(system, positions [N, 3], index of each water's oxygen, its neighbouring waters)."""
    vectors = None
    if chain:
        topology, flat = synthetic.solvated_chain(atoms, chain, seed=structure_seed,
                                                  box_length=2.265 if atoms == 1190 else None)
    else:
        topology, flat = synthetic.water_box(atoms, seed=structure_seed)
    positions = np.asarray(flat, dtype=np.float64).reshape(-1, 3)
    oxygen = np.nonzero(np.asarray(topology["atomTypes"]) == synthetic.TYPE_ORDER.index("OW"))[0]
    if box == "octahedron":
        vectors, sites = _octahedron(len(oxygen))
        rng = np.random.default_rng(structure_seed)
        sites = sites[np.sort(rng.permutation(len(sites))[:len(oxygen)])] + rng.uniform(-0.01, 0.01, (len(oxygen), 3))
        for k in range(3):
            positions[oxygen + k] += sites - positions[oxygen]
    system = build_system(topology, cutoff=cutoff, box_vectors=vectors)
    matrix = np.asarray(system["boxVectors"], dtype=np.float64).reshape(3, 3)
    return system, positions, oxygen, _nearest(positions[oxygen], matrix, min(24, len(oxygen) - 1))


def _nearest(points, matrix, k):
    """The k nearest points of each by minimum image."""
    x = torch.tensor(points, dtype=torch.float32, device=DEVICE)
    m = torch.tensor(matrix, dtype=torch.float32, device=DEVICE)
    frac = x @ torch.linalg.inv(m)
    rows = max(1, 40_000_000 // len(points))
    out = []
    for a in range(0, len(points), rows):
        d = frac[a:a + rows, None, :] - frac[None, :, :]
        r2 = ((d - torch.round(d)) @ m).square().sum(-1)
        out.append(torch.topk(r2, k + 1, largest=False).indices)
    near = torch.cat(out)
    self_at = near == torch.arange(len(points), device=near.device)[:, None]
    # the point itself goes to the end and is dropped
    order = torch.argsort(self_at.to(torch.int8), dim=1, stable=True)
    return torch.gather(near, 1, order)[:, :k].cpu().numpy()


def _relaxed(structure, seed, iterations=80):
    """Positions with the waters' orientations drawn from the seed and relaxed together with small
    displacements: rigid-body descent on the TIP3P energy of neighbouring waters, steps capped."""
    system, base, oxygen, near = structure
    f64 = dict(dtype=torch.float64, device=DEVICE)
    m = torch.tensor(np.asarray(system["boxVectors"]).reshape(3, 3), **f64)
    inv = torch.linalg.inv(m)
    rng = np.random.default_rng([seed, 7])
    positions = base.copy()
    sites = base[oxygen] + rng.uniform(-0.005, 0.005, (len(oxygen), 3))
    q = rng.normal(size=(len(oxygen), 4))
    q /= np.linalg.norm(q, axis=1, keepdims=True)
    w, a, b, c = q.T
    rot = np.stack([np.stack([1 - 2 * (b * b + c * c), 2 * (a * b - c * w), 2 * (a * c + b * w)], -1),
                    np.stack([2 * (a * b + c * w), 1 - 2 * (a * a + c * c), 2 * (b * c - a * w)], -1),
                    np.stack([2 * (a * c - b * w), 2 * (b * c + a * w), 1 - 2 * (a * a + b * b)], -1)], 1)
    half = math.radians(104.52) / 2
    arms = np.array([[0.09572 * math.sin(half), 0.09572 * math.cos(half), 0.0],
                     [-0.09572 * math.sin(half), 0.09572 * math.cos(half), 0.0]])
    x = torch.tensor(sites, **f64)
    h = torch.tensor(np.einsum("wij,kj->wki", rot, arms), **f64)  # the hydrogens about the oxygen
    nb = torch.tensor(near, device=DEVICE)
    charge = torch.tensor([-0.834, 0.417, 0.417], **f64)
    sigma6, epsilon = 0.315061 ** 6, 0.1521 * 4.184
    origin = x.clone()
    for it in range(iterations):
        body = torch.cat([torch.zeros_like(x)[:, None], h], 1)  # [M, 3, 3], about the oxygen
        d = (x[:, None] - x[nb]) @ inv
        d = (d - torch.round(d)) @ m  # [M, K, 3]
        r2 = d.square().sum(-1)
        s6 = sigma6 / r2 ** 3
        force = ((24 * epsilon * (2 * s6 * s6 - s6) / r2)[..., None] * d).sum(1)
        arm = body[:, None, :, None] - body[nb][:, :, None] + d[:, :, None, None]  # [M, K, site, site, 3]
        r = arm.square().sum(-1).clamp_min(0.0064).rsqrt()
        per_site = ((KE * charge[:, None] * charge * r ** 3)[..., None] * arm).sum((1, 3))
        force = force + per_site.sum(1)
        torque = torch.linalg.cross(body, per_site, dim=-1).sum(1)
        fade = 1.0 - 0.9 * it / iterations
        size = torque.norm(dim=-1, keepdim=True).clamp_min(1e-9)
        axis, angle = torque / size, (size * 1.5e-3).clamp_max(0.2 * fade)
        cos, sin = torch.cos(angle)[:, None], torch.sin(angle)[:, None]
        u = axis[:, None].expand_as(h)
        h = h * cos + torch.linalg.cross(u, h, dim=-1) * sin + u * ((u * h).sum(-1, keepdim=True) * (1 - cos))
        size = force.norm(dim=-1, keepdim=True).clamp_min(1e-9)
        move = x + force / size * (size * 1e-6).clamp_max(0.002 * fade) - origin
        far = move.norm(dim=-1, keepdim=True).clamp_min(1e-9)
        x = origin + move * (0.03 / far).clamp_max(1.0)
    x, h = x.cpu().numpy(), h.cpu().numpy()
    positions[oxygen] = x
    positions[oxygen + 1], positions[oxygen + 2] = x + h[:, 0], x + h[:, 1]
    # seven decimals, then the 32-bit value the device holds: the same on every machine
    return np.round(positions, 7).astype(np.float32).astype(np.float64).reshape(-1)


def _velocities(system, seed):
    masses = np.asarray(system["topology"]["masses"])
    rng = np.random.default_rng([seed, 11])
    v = rng.normal(size=(len(masses), 3)) * np.sqrt(KB * TEMPERATURE / masses)[:, None]
    return np.round(v, 6).astype(np.float32).astype(np.float64).reshape(-1)


def _grid(case, system):
    box = np.asarray(system["boxVectors"], dtype=np.float64).reshape(3, 3)
    if case["grid"] == "derived":
        return None
    return [_transformable(int(math.ceil(np.linalg.norm(box[d]) / 0.1))) for d in range(3)]


def _options(case, system, seed):
    o = {"timestep": TIMESTEP, "temperature": TEMPERATURE, "friction": 1.0, "seed": seed & 0xffff,
         "pmeOrder": case["order"], "waterSolver": case["solver"], "grid": _grid(case, system),
         # rows with room for the densest surroundings of these raw structures: a row that
         # overflows drops pairs until the block's end, and no two runs then agree
         "neighbourSlack": 3.0}
    if case["skin"]:
        o["skin"] = case["skin"]
    if case.get("pressure") is not None:
        o.update({"pressure": case["pressure"], "barostatInterval": 25})
    return o


def _single(case):
    return _structure(case["atoms"], case["chain"], case["box"], case["cutoff"], case["atoms"])


@functools.lru_cache(maxsize=8)
def _batch_sizes(count, low, high):
    rng = np.random.default_rng(count * 100003 + low)
    sizes = np.exp(rng.uniform(math.log(low), math.log(high), size=count)).astype(int)
    return [(int(n), int(rng.integers(20, max(21, min(300, n // 10))))) for n in sizes]


def prepare(case, seed):
    if case["kind"] == "batch":
        made = [_structure(n, c, "cubic", case["cutoff"], k + 1)
                for k, (n, c) in enumerate(_batch_sizes(case["count"], case["low"], case["high"]))]
        sim = BatchSimulation([s[0] for s in made], [_options(case, s[0], seed + k) for k, s in enumerate(made)])
        for k, s in enumerate(made):
            sim.setState(k, _relaxed(s, seed + 1000 * k), _velocities(s[0], seed + 1000 * k))
        sim.initialise()
        return {"case": case, "sim": sim}
    structure = _single(case)
    sim = GpuSimulation(structure[0], _options(case, structure[0], seed))
    positions = _relaxed(structure, seed, 80 if case["kind"] != "minimise" else 20)
    state = {"case": case, "sim": sim, "positions": positions}
    if case["kind"] == "run":
        sim.setState(positions, _velocities(structure[0], seed))
        sim.initialise()
    return state


TERMS = ("potential", "kinetic", "harmonicBond", "harmonicAngle", "periodicTorsion", "lennardJones", "dispersion",
         "coulombDirect", "coulombReciprocal", "coulombSelf")


def _report(e):
    return np.array([e[k] for k in TERMS])


def run(state):
    case, sim = state["case"], state["sim"]
    if case["kind"] == "batch":
        sim.run(case["steps"], blockSize=case["block"])
        read = [sim.readState(k) for k in range(sim.count)]
        return {k: np.concatenate([np.atleast_1d(r[k]) for r in read])
                for k in ("positions", "velocities", "forces", "boxVectors")}
    if case["kind"] == "run":
        sim.run(case["steps"], blockSize=case["block"] or None)
        out = {"energies": _report(sim.energy())} if case["energy"] else {}
        read = sim.readState()
        return {**out, **{k: read[k] for k in ("positions", "velocities", "forces", "boxVectors")}}
    sim.setState(state["positions"])
    sim.initialise()
    if case["kind"] == "evaluate":
        e = sim.energy()
        return {"energies": _report(e), "volumeDerivative": e["volumeDerivative"], "forces": sim.readState()["forces"]}
    m = sim.minimise(maxIterations=case["iterations"], forceTolerance=10.0)
    read = sim.readState()
    return {"positions": read["positions"], "forces": read["forces"],
            "result": np.array([m["potential"], m["max_force"], m["max_step"]]),
            "counts": np.array([m["iterations"], m["rejected"], m["stalled"], m["converged"]], dtype=np.int64)}


# ------------------------------------------------------------------------------- what a pass needs
def _evaluation_work(system, grid, order, cutoff):
    n = system["topology"]["atomCount"]
    box = np.asarray(system["boxVectors"], dtype=np.float64)
    pairs = 0.5 * n * n / abs(box[0] * box[4] * box[8]) * 4.0 / 3.0 * math.pi * cutoff ** 3
    points = float(np.prod(grid))
    # a pair: distance, Lennard-Jones, screened Coulomb, force on both atoms; the grid: charges
    # spread and forces gathered over order^3 points an atom, two transforms, the convolution
    flops = 50.0 * pairs + n * order ** 3 * 10.0 + 5.0 * points * math.log2(points) + 8.0 * points
    return {"bytes": 16.0 * n + 12.0 * n, "flops": flops}  # positions and charges in, forces out


def work(case):
    if case["kind"] == "batch":
        systems = [_structure(n, c, "cubic", case["cutoff"], k + 1)[0]
                   for k, (n, c) in enumerate(_batch_sizes(case["count"], case["low"], case["high"]))]
    else:
        systems = [_single(case)[0]]
    total = {"bytes": 0.0, "flops": 0.0}
    for system in systems:
        n = system["topology"]["atomCount"]
        one = _evaluation_work(system, _grid(case, system) or _derived_grid(case, system), case["order"], case["cutoff"])
        if case["kind"] == "evaluate":
            evaluations, bytes_each, flops_each = 2, 0.0, 0.0  # initialise() and energy()
        elif case["kind"] == "minimise":
            evaluations, bytes_each, flops_each = case["iterations"] + 2, 24.0 * n, 12.0 * n
        else:
            evaluations, bytes_each, flops_each = case["steps"], 64.0 * n, 300.0 * n  # positions and velocities
            if case.get("energy"):
                evaluations += 1
            if case.get("pressure") is not None:
                evaluations += case["steps"] // 25
        total["bytes"] += evaluations * (one["bytes"] + bytes_each) + 36.0 * n
        total["flops"] += evaluations * (one["flops"] + flops_each)
    return total


def _derived_grid(case, system):
    box = np.asarray(system["boxVectors"], dtype=np.float64).reshape(3, 3)
    alpha = math.sqrt(-math.log(2 * 5e-4)) / case["cutoff"]
    return [_transformable(max(2, int(math.ceil(2.0 * alpha * np.linalg.norm(box[d]) / (3.0 * 5e-4 ** 0.2)))))
            for d in range(3)]


def tolerance(case):
    """About four times what the default path differs by from the same path with every pair's force
    summed in another order and in 32 bits (per-atom rows, forceAccumulation 1), over two passes."""
    if case["kind"] == "evaluate":
        return {"rel": 5e-6, "max": 1e-4}
    if case["kind"] == "minimise":
        return {"rel": 5e-4, "max": 5e-2}
    if case["kind"] == "run" and case["steps"] <= 10:
        return {"rel": 5e-5, "max": 2e-3}
    # 32-bit rounding grows along a trajectory, tenfold in about 25 steps of these boxes
    return {"rel": 5e-3, "max": 0.5}


# ------------------------------------------------------------------------------- 64 bits
def _min_image(d, box):
    k = torch.round(d[..., 2] / box[2, 2])
    d = d - k[..., None] * box[2]
    k = torch.round(d[..., 1] / box[1, 1])
    d = d - k[..., None] * box[1]
    k = torch.round(d[..., 0] / box[0, 0])
    return d - k[..., None] * box[0]


def _spline(u, order):
    """Cardinal B-spline weights and derivatives of the `order` points ending at floor(u)."""
    x = u[:, None] + torch.arange(order - 1, -1, -1, dtype=u.dtype, device=u.device)

    def value(x, p):
        if p == 2:
            return (1 - (x - 1).abs()).clamp_min(0)
        return (x * value(x, p - 1) + (p - x) * value(x - 1, p - 1)) / (p - 1)

    return value(x, order), value(x, order - 1) - value(x - 1, order - 1)


def _modulus(n, order):
    w, _ = _spline(torch.zeros(1, dtype=torch.float64), order)
    k = torch.arange(order, dtype=torch.float64)
    m = torch.arange(n, dtype=torch.float64)
    phase = 2 * math.pi * m[:, None] * k[None] / n
    raw = (w * torch.cos(phase)).sum(1) ** 2 + (w * torch.sin(phase)).sum(1) ** 2
    return torch.where(raw < 1e-7, 0.5 * (raw.roll(1) + raw.roll(-1)), raw).to(DEVICE)


def _bonded(system, x, box):
    """Harmonic bonds, angles and torsions: energies and forces (by differentiation)."""
    t = system["topology"]
    hb, an, di = system["harmonicBonds"], t["angles"], t["dihedrals"]
    dev = dict(device=DEVICE)
    x = x.detach().clone().requires_grad_(True)
    zero = torch.zeros((), dtype=torch.float64, **dev)
    energies = [zero, zero, zero]

    def at(k):
        return torch.as_tensor(np.asarray(k, dtype=np.int64), **dev)

    def val(k):
        return torch.as_tensor(np.asarray(k, dtype=np.float64), **dev)

    if hb["count"]:
        r = (x[at(hb["atomA"])] - x[at(hb["atomB"])]).norm(dim=-1)
        energies[0] = (0.5 * val(hb["k"]) * (r - val(hb["r0"])) ** 2).sum()
    if an["count"]:
        u = x[at(an["atomA"])] - x[at(an["atomB"])]
        v = x[at(an["atomC"])] - x[at(an["atomB"])]
        theta = torch.atan2(torch.linalg.cross(u, v, dim=-1).norm(dim=-1), (u * v).sum(-1))
        energies[1] = (0.5 * val(an["k"]) * (theta - val(an["theta0"])) ** 2).sum()
    if di["count"]:
        a, b, c, d = (x[at(di[k])] for k in ("atomA", "atomB", "atomC", "atomD"))
        b1, b2, b3 = b - a, c - b, d - c
        n1, n2 = torch.linalg.cross(b1, b2, dim=-1), torch.linalg.cross(b2, b3, dim=-1)
        phi = torch.atan2((torch.linalg.cross(n1, n2, dim=-1) * b2).sum(-1) / b2.norm(dim=-1), (n1 * n2).sum(-1))
        energies[2] = (val(di["k"]) * (1 + torch.cos(val(di["periodicity"]) * phi - val(di["phase"])))).sum()
    total = energies[0] + energies[1] + energies[2]
    force = -torch.autograd.grad(total, x)[0] if total.requires_grad else torch.zeros_like(x)
    return [float(e.detach()) for e in energies], force


def _potential(case, system, positions):
    """(energy terms as _report lists them, kinetic left at 0; forces [N, 3]) in 64 bits: all pairs by
    minimum image, smooth particle-mesh Ewald on the case's grid, bonded terms."""
    f64 = dict(dtype=torch.float64, device=DEVICE)
    t = system["topology"]
    n = t["atomCount"]
    box = torch.tensor(np.asarray(system["boxVectors"]).reshape(3, 3), **f64)
    x = torch.tensor(positions.reshape(-1, 3), **f64)
    q = torch.tensor(np.asarray(t["charges"]), **f64)
    types = torch.tensor(np.asarray(t["atomTypes"]).astype(np.int64), device=DEVICE)
    tc = t["typeCount"]
    lj_a, lj_b = (torch.tensor(np.asarray(t[k]), **f64).reshape(tc, tc) for k in ("ljA", "ljB"))
    cutoff = case["cutoff"]
    alpha = math.sqrt(-math.log(2 * 5e-4)) / cutoff
    gauss = 2 * alpha / math.sqrt(math.pi)
    volume = float(torch.linalg.det(box).abs())
    force = torch.zeros(n, 3, **f64)
    e_lj = e_dir = 0.0

    start, partners = np.asarray(t["exclusions"]["start"]), np.asarray(t["exclusions"]["partners"]).astype(np.int64)
    owner = np.repeat(np.arange(n), np.diff(start))
    ea = torch.tensor(np.concatenate([owner, partners]), device=DEVICE)
    eb = torch.tensor(np.concatenate([partners, owner]), device=DEVICE)
    rows = max(1, 20_000_000 // n)
    for a in range(0, n, rows):
        stop = min(n, a + rows)
        d = _min_image(x[a:stop, None] - x[None], box)
        r2 = d.square().sum(-1)
        mine = (ea >= a) & (ea < stop)
        r2[ea[mine] - a, eb[mine]] = 1e9
        r2[torch.arange(stop - a, device=DEVICE), torch.arange(a, stop, device=DEVICE)] = 1e9
        i, j = torch.nonzero(r2 <= cutoff * cutoff, as_tuple=True)
        r2, d = r2[i, j], d[i, j]
        i = i + a
        inv2 = 1 / r2
        r = r2.sqrt()
        a12, b6 = lj_a[types[i], types[j]] * inv2 ** 6, lj_b[types[i], types[j]] * inv2 ** 3
        qq = KE * q[i] * q[j]
        screened = torch.special.erfc(alpha * r)
        scalar = (12 * a12 - 6 * b6) * inv2 + qq * (screened / r + gauss * torch.exp(-(alpha * r) ** 2)) * inv2
        force.index_add_(0, i, scalar[:, None] * d)
        e_lj += 0.5 * float((a12 - b6).sum())
        e_dir += 0.5 * float((qq * screened / r).sum())
    ex = system["exceptions"]
    if ex["count"]:
        i, j = (torch.tensor(np.asarray(ex[k]).astype(np.int64), device=DEVICE) for k in ("atomA", "atomB"))
        cp, la, lb = (torch.tensor(np.asarray(ex[k], dtype=np.float64), device=DEVICE)
                      for k in ("chargeProduct", "ljA", "ljB"))
        d = _min_image(x[i] - x[j], box)
        r2 = d.square().sum(-1)
        inv2, r = 1 / r2, r2.sqrt()
        a12, b6 = la * inv2 ** 6, lb * inv2 ** 3
        full = KE * q[i] * q[j]
        erf = torch.special.erf(alpha * r)
        scalar = (12 * a12 - 6 * b6) * inv2 + KE * cp / r * inv2
        scalar = scalar - full * (erf / r - gauss * torch.exp(-(alpha * r) ** 2)) * inv2
        force.index_add_(0, i, scalar[:, None] * d)
        force.index_add_(0, j, -scalar[:, None] * d)
        e_lj += float((a12 - b6).sum())
        e_dir += float((KE * cp / r - full * erf / r).sum())

    # reciprocal space
    grid = _grid(case, system) or _derived_grid(case, system)
    order = case["order"]
    inv = torch.linalg.inv(box)
    scaled = x @ inv
    scaled = (scaled - torch.floor(scaled)) * torch.tensor([float(g) for g in grid], **f64)
    cell = torch.floor(scaled)
    w, dw, at = [], [], []
    for k in range(3):
        a, b = _spline(scaled[:, k] - cell[:, k], order)
        w.append(a)
        dw.append(b)
        at.append((cell[:, k, None].long() + torch.arange(order, device=DEVICE) - order + 1) % grid[k])
    flat = ((at[0][:, :, None, None] * grid[1] + at[1][:, None, :, None]) * grid[2] + at[2][:, None, None, :]).reshape(n, -1)
    weight = (w[0][:, :, None, None] * w[1][:, None, :, None] * w[2][:, None, None, :]).reshape(n, -1)
    charge = torch.zeros(grid[0] * grid[1] * grid[2], **f64)
    charge.index_add_(0, flat.reshape(-1), (weight * q[:, None]).reshape(-1))
    spectrum = torch.fft.fftn(charge.reshape(*grid))
    k = [torch.fft.fftfreq(g, 1.0 / g, **f64) for g in grid]
    m = (k[0][:, None, None, None] * inv[:, 0] + k[1][None, :, None, None] * inv[:, 1] + k[2][None, None, :, None] * inv[:, 2])
    m2 = m.square().sum(-1)
    m2[0, 0, 0] = 1.0
    mod = [_modulus(g, order) for g in grid]
    kernel = torch.exp(-math.pi ** 2 * m2 / alpha ** 2) / (m2 * mod[0][:, None, None] * mod[1][None, :, None] * mod[2])
    kernel[0, 0, 0] = 0.0
    e_rec = float((kernel * spectrum.abs() ** 2).sum()) * KE / (2 * math.pi * volume)
    phi = (torch.fft.ifftn(kernel * spectrum).real * charge.numel() * KE / (math.pi * volume)).reshape(-1)[flat]
    gradient = []
    for axis in range(3):
        s = [dw[d] if d == axis else w[d] for d in range(3)]
        full = (s[0][:, :, None, None] * s[1][:, None, :, None] * s[2][:, None, None, :]).reshape(n, -1)
        gradient.append((full * phi).sum(1) * grid[axis])
    force -= q[:, None] * (torch.stack(gradient, 1) @ inv.T)
    bonded, extra = _bonded(system, x, box)
    force += extra

    self_term = -KE * alpha * float((q * q).sum()) / math.sqrt(math.pi)
    self_term += -KE * math.pi * float(q.sum()) ** 2 / (2 * alpha ** 2 * volume)
    counts = torch.bincount(types, minlength=tc).double()
    share = n / (n + 1.0)
    da = float((counts[:, None] * counts[None] * lj_a).sum() + (counts * lj_a.diagonal()).sum()) * share
    db = float((counts[:, None] * counts[None] * lj_b).sum() + (counts * lj_b.diagonal()).sum()) * share
    dispersion = 2 * math.pi / volume * (da / (9 * cutoff ** 9) - db / (3 * cutoff ** 3))
    total = sum(bonded) + e_lj + dispersion + e_dir + e_rec + self_term
    return np.array([total, 0.0, *bonded, e_lj, dispersion, e_dir, e_rec, self_term]), force


def _normals(seed, atoms, step):
    """The counter-based normal triple of each atom at a step."""
    def mix(s):
        s = s ^ (s >> np.uint32(16))
        s = s * np.uint32(0x7feb352d)
        s = s ^ (s >> np.uint32(15))
        s = s * np.uint32(0x846ca68b)
        return s ^ (s >> np.uint32(16))

    def uniform(c):
        s = mix(np.uint32(seed) ^ (np.arange(atoms, dtype=np.uint32) * np.uint32(0x9e3779b1)))
        s = mix(s ^ np.uint32((step * 0x85ebca6b) & 0xffffffff))
        s = mix(s ^ np.uint32((c * 0xc2b2ae35) & 0xffffffff))
        return ((s >> np.uint32(9)).astype(np.float64) + 0.5) / 8388608.0

    u = [uniform(c) for c in range(4)]
    r1, r2 = np.sqrt(-2 * np.log(u[0])), np.sqrt(-2 * np.log(u[2]))
    return np.stack([r1 * np.cos(2 * math.pi * u[1]), r1 * np.sin(2 * math.pi * u[1]), r2 * np.cos(2 * math.pi * u[3])], 1)


def _dynamics(case, system, positions, velocities, seed):
    """BAOAB steps with every constraint solved to 64-bit accuracy."""
    f64 = dict(dtype=torch.float64, device=DEVICE)
    x = torch.tensor(positions.reshape(-1, 3), **f64)
    v = torch.tensor(velocities.reshape(-1, 3), **f64)
    n = len(x)
    im = 1.0 / torch.tensor(np.asarray(system["topology"]["masses"]), **f64)[:, None]
    con = system["constraints"]
    # three constraints a water, listed water by water
    ca, cb = (torch.tensor(np.asarray(con[k]).astype(np.int64), device=DEVICE).reshape(-1, 3) for k in ("atomA", "atomB"))
    length2 = torch.tensor(np.asarray(con["distance"]), **f64).reshape(-1, 3) ** 2
    h = 0.5 * TIMESTEP

    def project_v(v):
        for _ in range(100):
            for k in range(3):
                a, b = ca[:, k], cb[:, k]
                d = x[a] - x[b]
                lam = ((v[a] - v[b]) * d).sum(-1, keepdim=True) / ((im[a] + im[b]) * d.square().sum(-1, keepdim=True))
                v[a] -= lam * im[a] * d
                v[b] += lam * im[b] * d
        return v

    def drift(x, v):
        old, new = x, x + h * v
        free = new.clone()
        for _ in range(100):
            for k in range(3):
                a, b = ca[:, k], cb[:, k]
                d, ref = new[a] - new[b], old[a] - old[b]
                lam = (d.square().sum(-1) - length2[:, k])[:, None] / (2 * (im[a] + im[b]) * (d * ref).sum(-1, keepdim=True))
                new[a] -= lam * im[a] * ref
                new[b] += lam * im[b] * ref
        return new, v + (new - free) / h

    decay = math.exp(-TIMESTEP)
    kick = torch.sqrt((1 - decay ** 2) * KB * TEMPERATURE * im)
    _, f = _potential(case, system, x.cpu().numpy())
    for step in range(case["steps"]):
        v = project_v(v + h * im * f)
        x, v = drift(x, v)
        noise = torch.tensor(_normals(seed & 0xffff, n, step), **f64)
        v = project_v(decay * v + kick * noise)
        x, v = drift(x, v)
        _, f = _potential(case, system, x.cpu().numpy())
        v = project_v(v + h * im * f)
    return x, v, f


def exact(case, seed):
    """Evaluations, and runs of a few steps of a box in NVT. Longer runs (and minimisations) have no
    such value: 32-bit rounding grows along a trajectory, and volume moves and line searches decide."""
    if case["kind"] == "evaluate" and case["atoms"] <= 100000:
        structure = _single(case)
        terms, force = _potential(case, structure[0], _relaxed(structure, seed))
        return {"energies": terms, "volumeDerivative": None, "forces": force.reshape(-1)}
    if case["kind"] == "run" and case["steps"] <= 10 and case["pressure"] is None and case["atoms"] <= 30000 \
            and not case["energy"]:
        structure = _single(case)
        system = structure[0]
        x, v, f = _dynamics(case, system, _relaxed(structure, seed), _velocities(system, seed), seed)
        return {"positions": x.reshape(-1), "velocities": v.reshape(-1), "forces": f.reshape(-1),
                "boxVectors": np.asarray(system["boxVectors"], dtype=np.float64)}
    return None
