"""Every form of the group-pair search (one, four or eight warps a row, chosen by the number of group slots of the
handle) lists every pair of the oracle's rows once, for sizes on both sides of each line.
"""
import numpy as np
import pytest

from rainmd_b200.simulation import GpuSimulation
from test_bench_parity import assert_group_rows_cover, bench_options, water

pytestmark = pytest.mark.gpu


def slots(atoms, counts):
    return (atoms + 3) // 4 + int(np.prod(counts))


# lines at 1,184 slots (eight warps below) and at 4,736 (one from there on)
@pytest.mark.parametrize("atoms,skin,low,high", [(4200, 0.15, 1000, 1184), (4700, 0.15, 1184, 1400), (16000, 0.25, 3900, 4736),
                                                 (18900, 0.25, 4736, 5100)])
def test_every_form_lists_every_pair(atoms, skin, low, high):
    system, pos, grid = water(atoms, seed=3)
    sim = GpuSimulation(system, bench_options(grid, skin=skin))
    sim.setState(pos)
    sim.initialise()
    assert low <= slots(system["topology"]["atomCount"], sim.diagnostics()["cell_counts"]) < high
    assert assert_group_rows_cover(sim, system, skin=skin) > 0
    sim.release()
