"""The line preconditioner's kernels over the level counts where their split of a column changes
(2 to 16 levels per warp of 16, one thread per column beyond 256 levels), ragged rows and columns
fewer than a warp: Picard steps with the mixed line solve against the FP64 Jacobi solve."""
import numpy as np
import pytest

from frehg_gb300 import workloads as W
from frehg_gb300.abi import SolverConfig

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(5, 3, 31), (33, 7, 33), (32, 4, 64), (19, 9, 65), (12, 5, 97),
                                   (40, 3, 128), (7, 6, 129), (9, 4, 256), (6, 5, 257)])
def test_line_solve_level_counts(gpu_lib, shape):
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
        out = []
        for _ in range(2):
            g.advance_step()
            out.append((g.interior("h"), g.counters().last_picard_iterations))
        runs.append(out)
    for (ha, ia), (hb, ib) in zip(*runs):
        assert np.abs(ha - hb).max() <= 1e-8
        assert ia == ib
