"""What the host reads back in one copy after a block of steps, an evaluation or an initialise agrees
with what the separate reads of the same handle give, for one system and for a batch; readState's
packed arrays agree with one another whichever are asked for.
"""
import ctypes as C

import numpy as np
import pytest

from rainmd_b200 import synthetic
from rainmd_b200.simulation import BatchSimulation
from rainmd_b200.topology import build_system

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count", [1, 3])
def test_packed_state_and_reports(count):
    made = synthetic.batch(count, low=1001, high=2500, seed=5)
    batch = BatchSimulation([build_system(t, cutoff=0.9) for t, _ in made],
                            {"pmeOrder": 4, "skin": 0.1, "seed": 3, "pressure": 1.0, "neighbourSlack": 3.0, "waterSolver": 1})
    for k, (_, pos) in enumerate(made):
        batch.setState(k, pos)
    batch.initialise()
    batch.minimise(maxIterations=20)
    batch.run(60, blockSize=25)
    for k in range(count):
        state = batch.readState(k)
        n = batch.atom_counts[k]
        # one array at a time: the same values
        for which, name in enumerate(("positions", "velocities", "forces")):
            out = np.zeros(3 * n, np.float32)
            ptr = out.ctypes.data_as(C.POINTER(C.c_float))
            args = [None, None, None]
            args[which] = ptr
            assert batch._lib.rmd_read_state_at(batch._h, k, *args, None, None) == 0
            assert np.array_equal(out, state[name]), name
        e = batch.energy(k)
        assert np.isfinite(e["potential"]) and abs(e["volume"] - state["volume"]) < 1e-12
        v = state["velocities"].reshape(-1, 3).astype(np.float64)
        m = np.asarray(batch.systems[k]["topology"]["masses"])
        assert abs(e["kinetic"] - 0.5 * np.sum(m[:, None] * v ** 2)) < 1e-6 * e["kinetic"]
        d = batch.diagnostics(k)
        assert d["barostat_attempts"] == 2 and d["neighbour_required"] > 0
        assert batch.lastVolumeMove(k)["attempted"] == 1
        _, fresh = batch.debugEvaluate(k)
        assert np.max(np.abs(fresh - state["forces"])) < 1e-5 * np.sqrt(np.mean(fresh ** 2)) + 1e-6 * np.max(np.abs(fresh))
