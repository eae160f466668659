"""A released handle gives its device memory back."""
import pytest
import torch

from rainmd_b200 import synthetic
from rainmd_b200.simulation import GpuSimulation
from rainmd_b200.topology import build_system

pytestmark = pytest.mark.gpu


def test_release_returns_the_device_memory():
    topology, pos = synthetic.water_box(9000, seed=2)
    system = build_system(topology, cutoff=0.9)

    def one():
        sim = GpuSimulation(system, {"pmeOrder": 4, "skin": 0.1, "neighbourSlack": 3.0, "pressure": 1.0, "waterSolver": 1})
        sim.setState(pos)
        sim.initialise()
        sim.minimise(maxIterations=5)
        sim.run(10, blockSize=5)
        sim.energy()
        sim.readState()
        held = sim.diagnostics()["device_bytes"]
        sim.release()
        return held

    one()  # (module loading, and what the driver keeps for graphs)
    free = torch.cuda.mem_get_info()[0]
    held = sum(one() for _ in range(8))
    torch.cuda.synchronize()
    lost = free - torch.cuda.mem_get_info()[0]
    assert lost < 0.25 * held, (lost, held)
