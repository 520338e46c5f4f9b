"""Preparation of the mixed solve where its two forms meet (65,536 columns, 190 levels) and where a
block's 32 columns or eight levels are partly filled: Picard steps with the mixed line solve against
the FP64 Jacobi solve."""
import numpy as np
import pytest

from frehg_gb300 import workloads as W
from frehg_gb300.abi import SolverConfig

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(1, 1, 9), (31, 1, 8), (33, 1, 7), (3, 2, 190), (3, 2, 191),
                                   (256, 256, 3), (257, 256, 3)])
def test_preparation_forms(gpu_lib, shape):
    """Both solve each Picard system to a true residual of 1e-12, so heads agree far below the
    parity bound of 1e-8 m per step, with equal Picard counts."""
    from frehg_gb300.re_solver import Grid, ReSolver
    nx, ny, nz = shape
    runs = []
    for solver in (SolverConfig("cg", "line", rtol=1e-12, max_it=20000, precision=1, ir_rtol=1e-12),
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
