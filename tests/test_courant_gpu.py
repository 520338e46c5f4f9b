"""The Courant bound of the adaptive step in its three forms (four lanes per cell up to 8,192 cells,
separate blocks, in the update's blocks) against the oracle, on both sides of their limits."""
import numpy as np
import pytest

from frehg_gb300 import workloads as W
from frehg_gb300.abi import SolverConfig

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(1, 1, 33), (5, 3, 16), (33, 9, 6), (64, 16, 8), (64, 16, 9),
                                   (1, 1, 311), (40, 70, 20)])
def test_courant_forms(gpu_lib, oracle_mod, shape):
    """A small Courant number makes the bound the new step.  dK/dtheta is evaluated below 0.9999
    theta_s, where its relative change with theta is 1e4 at most; theta agrees to 1e-12: 1e-8."""
    from frehg_gb300.re_solver import Grid, ReSolver
    nx, ny, nz = shape
    w = W.config1("pca", nx=nx, ny=ny, nz=nz, steps=2)
    w.solver = SolverConfig("cg", "jacobi", rtol=1e-14, max_it=5000)
    w.params.adaptive_dt = 1
    w.params.co_max = 1e-6
    w.params.dt_min = 1e-12
    w.h0 = -np.random.default_rng(nx + ny + nz).uniform(0.05, 0.5, (nz, ny, nx))
    g = ReSolver(Grid(nx, ny, nz, w.params.dx, w.params.dy, w.params.dz), w.params)
    o = oracle_mod.OracleRe(nx, ny, nz, w.params)
    w.apply(g)
    w.apply(o)
    for _ in range(2):
        before = o.dt()
        g.advance_step()
        o.advance_step()
        assert abs(g.dt() - o.dt()) <= 1e-8 * o.dt()
    assert w.params.dt_min < o.dt() and o.dt() != before
