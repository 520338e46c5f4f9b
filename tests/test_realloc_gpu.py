"""Reallocation of the PCA step on both sides of its change of form (2,048 columns in one block), and
where a column's 16-level groups are partly filled: steps against the oracle."""
import numpy as np
import pytest

from frehg_gb300 import workloads as W
from frehg_gb300.abi import SolverConfig

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(1, 1, 33), (5, 3, 16), (45, 45, 17), (46, 45, 17)])
def test_reallocation_forms(gpu_lib, oracle_mod, shape):
    """Heads and water contents within the parity bounds of the PCA step (1e-8 m, 1e-9)."""
    from frehg_gb300.re_solver import Grid, ReSolver
    nx, ny, nz = shape
    w = W.config1("pca", nx=nx, ny=ny, nz=nz, steps=3)
    w.solver = SolverConfig("cg", "jacobi", rtol=1e-13, max_it=5000)
    g = ReSolver(Grid(nx, ny, nz, w.params.dx, w.params.dy, w.params.dz), w.params)
    o = oracle_mod.OracleRe(nx, ny, nz, w.params)
    w.apply(g)
    w.apply(o)
    for _ in range(3):
        g.advance_step()
        o.advance_step()
    assert np.abs(g.interior("h") - o.interior("h")).max() <= 1e-8
    assert np.abs(g.interior("wc") - o.interior("wc")).max() <= 1e-9
    assert g.counters().realloc_sweeps >= 3
