"""The updated refinement residual (exact FP32 products) at the edges of its tiles and marches, with
both inner preconditioners: Picard steps solved to a true residual of 1e-13 against the FP64 solve."""
import numpy as np
import pytest

from frehg_gb300 import workloads as W
from frehg_gb300.abi import SolverConfig

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pc", ["line", "jacobi"])
@pytest.mark.parametrize("shape", [(1, 1, 5), (2, 1, 6), (33, 9, 4), (31, 7, 66), (64, 17, 33)])
def test_updated_residual(gpu_lib, shape, pc):
    """Systems solved to 1e-13 and 1e-12 of the right-hand side's norm: heads agree far below the
    parity bound of 1e-8 m per step, with equal Picard counts."""
    from frehg_gb300.re_solver import Grid, ReSolver
    nx, ny, nz = shape
    runs = []
    for solver in (SolverConfig("cg", pc, rtol=1e-12, max_it=20000, precision=1, ir_rtol=1e-13),
                   SolverConfig("cg", "jacobi", rtol=1e-12, max_it=20000)):
        w = W.config4(nx=nx, ny=ny, nz=nz)
        w.solver = solver
        g = ReSolver(Grid(nx, ny, nz, w.params.dx, w.params.dy, w.params.dz), w.params)
        w.apply(g)
        g.advance_step()
        runs.append((g.interior("h"), g.counters().last_picard_iterations))
    (ha, ia), (hb, ib) = runs
    assert np.abs(ha - hb).max() <= 1e-8
    assert ia == ib
