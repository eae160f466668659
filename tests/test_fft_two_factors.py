"""The two-factor reciprocal-space transforms (csrc/fft.cuh): every DFT length they are built from,
on every axis, in planes of one block and of a cluster with even and ragged shares, with odd
planes (no 16-byte pairs), and beside axes without two factors, against the FP64 oracle; the
separate passes' line transforms against numpy.
"""
import math

import numpy as np
import pytest

from goldens import system_for
from rainmd_b200.simulation import BatchSimulation
from test_gpu_parity import ALPHA, engine_for, oracle_terms, relative

pytestmark = pytest.mark.gpu

# Factors: 4=2.2 5=1.5 6=2.3 8=2.4 9=3.3 10=2.5 12=3.4 15=3.5 16=4.4 18=3.6 20=4.5 25=5.5 27=3.9 32=4.8
# 36=6.6 45=5.9 50=5.10 54=6.9 60=6.10 64=8.8 72=8.9 75=5.15 80=8.10 81=9.9 96=8.12 100=10.10 108=9.12
# 125=5.25 128=8.16 135=9.15 144=12.12 150=10.15 160=10.16 162=9.18 200=10.20 225=15.15 240=15.16 250=10.25
# 288=16.18 320=16.20 324=18.18 400=20.20; none: 243 384 480
GRIDS = [
    (25, 27, 45), (27, 25, 5), (5, 5, 6), (6, 8, 10), (9, 10, 12), (15, 16, 18), (20, 36, 54),
    (45, 45, 50), (50, 50, 60), (64, 64, 64), (72, 75, 80), (81, 81, 15), (96, 100, 8),
    (108, 125, 10), (125, 108, 16), (128, 135, 9), (144, 144, 20), (150, 150, 6), (5, 400, 12),
    (320, 8, 25), (20, 20, 162), (16, 12, 225), (12, 16, 250), (10, 9, 400), (8, 240, 324), (18, 12, 243), (243, 10, 12),
    (12, 12, 480),
]


@pytest.mark.parametrize("grid", GRIDS)
def test_reciprocal_energy_and_forces(grid):
    s, pos, _ = system_for("ala-wat")
    sim = engine_for(s, pos, grid=list(grid))
    e, forces = sim.debugEvaluate()
    expect, fo = oracle_terms(s, pos, ALPHA, list(grid), 5)
    assert relative(e["coulomb_reciprocal"], expect["coulombReciprocal"]) < 2e-5
    assert np.max(np.abs(forces - fo)) / math.sqrt(np.mean(fo ** 2)) < 3e-3
    sim.release()


@pytest.mark.parametrize("grid", [(25, 27, 45), (6, 5, 8), (12, 10, 243), (7 + 1, 9, 400), (16, 18, 20)])
def test_z_passes_against_numpy(grid):
    """R2C and C2R z passes (the debug transform runs the separate y and x passes between them); the bar
    is an f32 FFT's error bound, 5 eps log2(N) of the spectrum's norm per point."""
    s, pos, _ = system_for("ala-wat")
    sim = engine_for(s, pos, grid=list(grid))
    data = np.random.default_rng(3).normal(size=grid)
    n = data.size
    half, back = sim.debugFft(data.reshape(-1), n // grid[2] * (grid[2] // 2 + 1))
    expect = np.fft.rfftn(data).reshape(-1)
    bar = 5 * 2 ** -24 * math.log2(n) * math.sqrt(n)
    assert np.max(np.abs(half - expect)) < bar
    assert np.max(np.abs(back / n - data.reshape(-1))) < 10 * 2 ** -24 * math.log2(n) * 4
    sim.release()


def test_a_batch_gives_each_grid_its_own_bits():
    """Axes of factors up to 12 and of longer ones take kernels built apart; which of them a system takes
    depends on its own axes alone, whatever shares its handle."""
    grids = [(64, 64, 64), (75, 75, 75), (24, 24, 24), (25, 75, 32), (160, 160, 8), (20, 24, 128), (125, 108, 16), (30, 30, 243)]
    s, pos, _ = system_for("ala-wat")
    options = [{"alpha": ALPHA, "grid": list(g), "skin": 0.1, "dispersionCorrection": False} for g in grids]
    batch = BatchSimulation([s] * len(grids), options)
    for k in range(len(grids)):
        batch.setState(k, pos)
    batch.initialise()
    for k, g in enumerate(grids):
        together, forces = batch.debugEvaluate(k)
        sim = engine_for(s, pos, grid=list(g))
        alone, expect = sim.debugEvaluate()
        for term in ("coulomb_reciprocal", "potential", "volume_derivative"):
            assert together[term] == alone[term], (g, term)
        assert np.array_equal(forces, expect), g
        sim.release()
    batch.release()
