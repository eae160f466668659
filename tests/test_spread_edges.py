"""Charge spreading and force gathering at the grid's edges: atoms on and a rounding step off the
faces of the cell and far outside it, on the smallest grids (an axis of exactly the spline's order,
where a spline covers the whole axis) and odd ones, against the FP64 oracle's reciprocal terms.
"""
import math

import numpy as np
import pytest

from goldens import system_for
from test_gpu_parity import ALPHA, engine_for, oracle_terms, relative

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order", [4, 5])
@pytest.mark.parametrize("grid", [(5, 24, 25), (24, 5, 27), (25, 27, 5), (6, 5, 8)])
def test_atoms_on_the_faces(order, grid):
    s, pos, _ = system_for("ala-wat")
    box = np.asarray(s["boxVectors"]).reshape(3, 3)
    pos = np.asarray(pos, dtype=np.float64).reshape(-1, 3).copy()
    # everything moved so that an atom sits on a corner of the cell (or a rounding step before one), then
    # whole molecules by whole cells, some far outside
    molecule = np.asarray(s["topology"]["moleculeOfAtom"])
    corner = np.array([1.0, 1 - 2.0 ** -24, 0.0]) @ box
    pos += corner - pos[30]
    cells = np.array([[0, 0, 0], [-3, 2, 0], [4, -2, 3], [0, 0, -1]])
    pos += (cells[molecule % 4] @ box)
    flat = pos.reshape(-1)
    sim = engine_for(s, flat, grid=list(grid), pmeOrder=order, neighbourSlack=4.0)
    e, _ = sim.debugEvaluate()
    got = sim.debugForceTerm("reciprocal")
    expect, _ = oracle_terms(s, flat, ALPHA, list(grid), order)
    assert relative(e["coulomb_reciprocal"], expect["coulombReciprocal"]) < 2e-5
    total = sim.debugChargeGrid(points=int(np.prod(grid))).sum()
    charge = float(np.sum(s["topology"]["charges"]))
    assert abs(total - charge) < pos.shape[0] * order ** 3 * 2.0 ** -24 * 0.2  # f32 weights of |q| < 1
    assert np.all(np.isfinite(got)) and math.isfinite(e["potential"])
    sim.release()
