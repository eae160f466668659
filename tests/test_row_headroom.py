"""Group-pair rows hold a quarter more than the planned capacity: builds inside a block of steps that
pass it lose no pair before the block's check grows the lists. (A dropped pair changes the forces
of the step, and which pairs are dropped depends on timing, so runs would not repeat either.)
"""
import numpy as np
import pytest

from goldens import system_for
from rainmd_b200.simulation import GpuSimulation
from test_rebuild_on_demand import ALPHA, make

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("short", [0, 24])
def test_builds_past_the_capacity_inside_a_block_lose_no_pair(short):
    probe = make(skin=0.08)
    state = probe.readState()
    need = probe.diagnostics()["neighbour_required"]
    probe.release()
    s, _, _ = system_for("ala-wat")
    runs = []
    for capacity in (need, 4 * need):
        sim = GpuSimulation(s, {"alpha": ALPHA, "grid": [24, 24, 24], "temperature": 300, "seed": 11,
                                "dispersionCorrection": False, "skin": 0.08, "maxNeighbours": capacity - short})
        sim.setState(state["positions"].astype(np.float64), state["velocities"].astype(np.float64))
        sim.initialise()
        sim.run(100, blockSize=100)
        d = sim.diagnostics()
        assert d["worst_neighbour_required"] < 1.25 * (need - short)
        runs.append(sim.readState())
        sim.release()
    # no pair was lost: the run repeats, bit for bit, the one whose rows never filled
    for k in ("positions", "velocities", "forces"):
        assert np.array_equal(runs[0][k], runs[1][k]), k
