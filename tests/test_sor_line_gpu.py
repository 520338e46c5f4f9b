"""PCSOR on one line of cells (the sweeps as a scan over 32 chunks) along each axis, with chunks empty,
of one cell and uneven."""
import numpy as np
import pytest

from frehg_gb300.abi import SolverConfig

from tests.test_linear_seam_gpu import spd_stencil
from tests.test_sor_gpu import assemble_coo

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(1, 1, 1), (2, 1, 1), (1, 31, 1), (1, 1, 32), (33, 1, 1), (1, 1, 100),
                                   (1, 1025, 1), (3599, 1, 1)])
def test_sor_line(gpu_lib, oracle_mod, shape):
    """Both converge the same system to rtol 1e-12, so the solutions agree to that times the
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
