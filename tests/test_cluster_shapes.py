"""Constraint clusters of a fixed shape (a rigid 3-site triangle; a heavy atom with one, two or
three hydrogens) take the register form of SHAKE and RATTLE, the others the general one. Writing a
constraint's two atoms the other way round leaves the constraint what it is and sends its cluster to
the general form, so the two forms are compared on the same system.
"""
import copy

import numpy as np
import pytest

from goldens import system_for
from rainmd_b200 import synthetic
from rainmd_b200.simulation import GpuSimulation
from rainmd_b200.topology import build_system

pytestmark = pytest.mark.gpu


def hydrogens(count):
    """A water box in which every molecule's constraints are those of a heavy atom with `count`
    hydrogens (1: O-H1; 2: O-H1 and O-H2) or the triangle (0)."""
    topology, pos = synthetic.water_box(2001, seed=4)
    system = build_system(topology, cutoff=0.9)
    if count:
        c = system["constraints"]
        keep = np.arange(c["count"]) % 3 < count
        for k in ("atomA", "atomB", "distance"):
            c[k] = c[k][keep]
        c["count"] = int(keep.sum())
        system["degreesOfFreedom"] = 3 * topology["atomCount"] - c["count"] - 3
    return system, pos


def turned(system):
    out = copy.copy(system)
    c = system["constraints"]
    out["constraints"] = {**c, "atomA": c["atomB"], "atomB": c["atomA"]}
    return out


@pytest.mark.parametrize("case", ["triangle", "one", "two", "solute"])
def test_fixed_shapes_match_the_general_form(case):
    if case == "solute":  # CH3, NH and CH groups and waters
        system, pos, _ = system_for("ala-wat")
    else:
        system, pos = hydrogens({"triangle": 0, "one": 1, "two": 2}[case])
    runs = []
    for s in (system, turned(system)):
        sim = GpuSimulation(s, {"pmeOrder": 4, "grid": [30, 30, 30], "skin": 0.1, "temperature": 300.0, "seed": 5,
                                "neighbourSlack": 3.0, "timestep": 0.001})
        sim.setState(pos)
        sim.initialise()
        sim.minimise(maxIterations=10)
        start = sim.readState()["positions"].astype(np.float64)
        sim.setState(start)
        sim.initialise()
        sim.run(10, blockSize=10)
        runs.append((start, sim.readState(), sim.diagnostics()))
        sim.release()
    (a0, a, da), (b0, b, db) = runs
    assert da["cluster_count"] == db["cluster_count"] > 0
    assert not any(d[k] for d in (da, db) for k in ("shake_hit_iteration_cap", "rattle_hit_iteration_cap"))
    assert abs(da["max_shake_iterations"] - db["max_shake_iterations"]) <= 1
    # the same arithmetic on turned differences, up to the contraction of multiply-adds: a few ulp of
    # a coordinate a step, and the tolerance's own slack where an iteration count differs
    bar = 10 * 20 * 2.0 ** -23 * np.max(np.abs(a["positions"])) + 10 * da["constraint_tolerance"] * 0.1
    assert np.max(np.abs(a0 - b0)) < bar
    assert np.max(np.abs(a["positions"] - b["positions"])) < bar
    pairs = system["constraints"]
    x = a["positions"].reshape(-1, 3).astype(np.float64)
    length = np.linalg.norm(x[pairs["atomA"]] - x[pairs["atomB"]], axis=1)
    # SHAKE's bound is relative to the squared length; the device's coordinates are 32-bit
    slack = da["constraint_tolerance"] * pairs["distance"] + 4 * 2.0 ** -24 * np.max(np.abs(x))
    assert np.all(np.abs(length - pairs["distance"]) <= slack)
