"""Group-pair rows hold a quarter more than the planned capacity: builds inside a block of steps that need up to
that much lose no pair before the block's check grows the lists. (A dropped pair changes the forces of the
step, and which pairs are dropped depends on timing, so runs would not repeat either.) A build that needs still more
is reported: the block's steps count as steps on lists that may lack pairs.
"""
import numpy as np
import pytest

from goldens import system_for
from rainmd_b200.simulation import GpuSimulation
from test_rebuild_on_demand import ALPHA, make

pytestmark = pytest.mark.gpu


def engine(state, skin, temperature, capacity):
    s, _, _ = system_for("ala-wat")
    sim = GpuSimulation(s, {"alpha": ALPHA, "grid": [24, 24, 24], "temperature": temperature, "seed": 11,
                            "dispersionCorrection": False, "skin": skin, "maxNeighbours": capacity})
    sim.setState(state["positions"].astype(np.float64), state["velocities"].astype(np.float64))
    sim.initialise()
    return sim


def tight_and_ample(skin, temperature, steps):
    """Two runs of one block: rows planned for the start alone, and rows that never fill."""
    probe = make(skin=skin)
    state = probe.readState()
    need = probe.diagnostics()["neighbour_required"]
    probe.release()
    out = []
    for capacity in (need, 4 * need):
        sim = engine(state, skin, temperature, capacity)
        before = sim.diagnostics()
        assert before["neighbour_growths"] == 0  # the rows hold the first build
        sim.run(steps, blockSize=steps)
        out.append((before["neighbour_capacity"], sim.diagnostics(), sim.readState()))
        sim.release()
    return out


@pytest.mark.parametrize("skin", [0.08, 0.15])
def test_builds_past_the_capacity_inside_a_block_lose_no_pair(skin):
    (capacity, tight, a), (_, ample, b) = tight_and_ample(skin, 300, 100)
    # builds of this block need more than the capacity, and no more than the headroom
    assert capacity < ample["worst_neighbour_required"] <= capacity + capacity // 4
    # the check after the block saw it
    assert tight["neighbour_growths"] == 1 and tight["worst_neighbour_required"] == ample["worst_neighbour_required"]
    assert tight["neighbour_capacity"] >= ample["worst_neighbour_required"]
    assert tight["steps_with_stale_list"] == ample["steps_with_stale_list"] == 0
    # no pair was lost: the run repeats, bit for bit, the one whose rows never filled
    for k in ("positions", "velocities", "forces"):
        assert np.array_equal(a[k], b[k]), k


def test_builds_past_the_headroom_are_reported():
    (capacity, tight, _), (_, ample, _) = tight_and_ample(0.02, 600, 400)
    assert ample["worst_neighbour_required"] > capacity + (capacity // 4 + 3) // 4 * 4
    assert tight["neighbour_growths"] == 1
    assert tight["steps_with_stale_list"] == 400 and ample["steps_with_stale_list"] == 0
