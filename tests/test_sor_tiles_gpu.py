"""PCSOR's two forms on the GPU (systems up to 3,600 unknowns: the whole CG solve in one block;
larger ones: one warp per tile of 32 lines) where their tiles end inside the grid."""
import numpy as np
import pytest

from frehg_gb300.abi import SolverConfig

from tests.test_linear_seam_gpu import spd_stencil
from tests.test_sor_gpu import assemble_coo

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [
    (15, 15, 16), (60, 60, 1), (1, 3600, 1),  # 3,600 unknowns: the last size solved in one block
    (13, 277, 1), (1, 1, 3700),               # above it: one tile axis, none
    (61, 3, 40), (9, 33, 34), (34, 9, 33),    # tiles cut off along either axis, each line axis
    (5, 2, 700), (2, 1900, 2)])
def test_sor_tile_edges(gpu_lib, oracle_mod, shape):
    """The sweeps' tiles (32 lines along the longest axis) cut off by the grid, tiles of one or no
    axis, and both forms of the solve, against the oracle's sequential sweeps.  Both
    converge the same system to rtol 1e-12, so the solutions agree to that times the
    condition number (below 1e3 for these diagonally dominant systems): 1e-9 relative."""
    from frehg_gb300.linear import makeLinearSolver
    nx, ny, nz = shape
    coef, b = spd_stencil(nx, ny, nz, seed=nx * 100 + ny * 10 + nz)
    solver = makeLinearSolver("gb300", SolverConfig("cg", "sor", rtol=1e-12))
    A = solver.createSystem(nx, ny, nz)
    assemble_coo(A, coef, nx, ny, nz)
    x = solver.solve(A, b)
    xo, reason, its, _ = oracle_mod.ksp_solve_stencil(nx, ny, nz, coef.ravel(), b, "cg", "sor",
                                                      1e-12)
    assert reason > 0
    assert abs(solver.getIterationCount() - its) <= 1
    assert np.abs(x - xo).max() <= 1e-9 * max(1.0, np.abs(xo).max())
