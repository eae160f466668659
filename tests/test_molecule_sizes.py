"""Molecules of every size in the kernels that walk them (the molecular virial, the scaling of centroids): those of
up to 8 atoms are a thread's, the larger ones a warp's. Waters of one box are joined into uneven molecules, so that
positions and forces are the same whatever the partition, and both kernels are compared with 64-bit sums.
"""
import time

import numpy as np
import pytest

from rainmd_b200 import synthetic
from rainmd_b200.simulation import GpuSimulation
from rainmd_b200.topology import build_system

pytestmark = pytest.mark.gpu


def box(atoms, waters):
    """A water box whose molecules join `waters[0]`, `waters[1]`, ... waters in turn."""
    topology, pos = synthetic.water_box(atoms, seed=6)
    system = build_system(topology, cutoff=0.9)
    count = topology["atomCount"] // 3
    molecule = np.repeat(np.arange(count), np.resize(waters, count))[:count]
    joined = np.repeat(molecule, 3)[:topology["atomCount"]].astype(np.int32)
    system["topology"] = {**topology, "moleculeOfAtom": joined}
    system["molecules"] = {**system["molecules"], "count": int(joined.max()) + 1}
    return system, joined, pos


def engine(system, pos):
    sim = GpuSimulation(system, {"pmeOrder": 4, "skin": 0.1, "waterSolver": 1, "neighbourSlack": 3.0})
    sim.setState(pos)
    sim.initialise()
    return sim


def centres(x, molecule, masses):
    total = np.bincount(molecule, masses)
    return np.stack([np.bincount(molecule, masses * x[:, c]) / total for c in range(3)], 1)[molecule]


@pytest.mark.parametrize("waters", [[1], [2], [3], [1, 3, 2, 7], [1, 1, 40, 2, 11], [33], [2000]])
def test_virial_and_scaling(waters):
    water, _, pos = box(3000, [1])
    system, molecule, _ = box(3000, waters)
    masses = np.asarray(system["topology"]["masses"], dtype=np.float64)
    one, other = engine(water, pos), engine(system, pos)
    a, b = one.energy(), other.energy()
    state = other.readState()
    assert np.array_equal(state["forces"], one.readState()["forces"])
    x = state["positions"].reshape(-1, 3).astype(np.float64)
    f = state["forces"].reshape(-1, 3).astype(np.float64)

    def virial(m):
        return np.sum(f * (x - centres(x, m, masses)))

    # forces read back in 32 bits
    arm = x - centres(x, molecule, masses)
    bar = 2.0 ** -23 * np.sum(np.abs(f) * (np.abs(arm) + 0.1))
    expect = (virial(molecule) - virial(np.arange(len(x)) // 3)) / 3.0
    assert abs((b["volumeDerivative"] - a["volumeDerivative"]) - expect) < bar
    other.scaleVolume(1.01)
    got = other.readState()["positions"].reshape(-1, 3)
    assert np.max(np.abs(got - (x + 0.01 * centres(x, molecule, masses)))) <= 2.0 ** -23 * np.max(np.abs(x)) * 1.01


def test_large_molecules_are_not_walked_in_turn():
    """An energy report of a box whose molecules hold 1,200 atoms takes at most 2.5 times that of its waters: with a
    warp a molecule it is about 1.3 times, with a warp that walks 32 of them 4.4 times."""
    times = []
    for waters in ([1], [400]):
        system, _, pos = box(24000, waters)
        sim = engine(system, pos)
        for _ in range(5):
            sim.energy()
        runs = []
        for _ in range(31):
            begin = time.perf_counter()
            sim.energy()
            runs.append(time.perf_counter() - begin)
        times.append(sorted(runs)[8])
        sim.release()
    assert times[1] < 2.5 * times[0], times
