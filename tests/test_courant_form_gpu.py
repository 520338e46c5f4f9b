"""The Courant bound of a small grid does not depend on how its cells lie in the kernel's blocks: the
same column of cells along x and along y, and modified van Genuchten cells among the others."""
import numpy as np
import pytest

from frehg_gb300 import workloads as W
from frehg_gb300.abi import SolverConfig
from frehg_gb300.re_solver import SoilMap

pytestmark = pytest.mark.gpu

N, NZ = 60, 40


def bound(shape, seed, mvg):
    """dt after a step too short to change the water content (1e-30 s), set by the bound"""
    from frehg_gb300.re_solver import Grid, ReSolver
    nx, ny, nz = shape
    w = W.config0("pca", nx=nx, ny=ny, nz=nz)
    p = w.params
    p.bc_type[5] = 0  # closed top: no saturated neighbour
    p.adaptive_dt, p.dt, p.dt_min, p.dt_max, p.co_max = 1, 1e-30, 1e-60, 1.0, 1e-40
    g = ReSolver(Grid(nx, ny, nz, p.dx, p.dy, p.dz), p)
    h = -np.random.default_rng(seed).uniform(0.2, 0.5, (nz, N))
    dry = np.arange(N) % 8 == 5  # one cell of eight neighbours: a hundred times the bound
    h[:, dry] = -50.0
    if mvg:
        other = p.soil.copy()
        other.use_mvg = 1
        m = SoilMap()
        m.setClasses([p.soil.copy(), other])
        m.setClassIndex3D(nx, ny, nz, np.broadcast_to(dry, (nz, N)).reshape(nz, ny, nx)
                          .astype(np.int32))
        g.set_soil_map(m)
    g.initialize_geometry()
    g.attach_solver(SolverConfig("cg", "jacobi", rtol=1e-12, max_it=1000))
    g.set_initial_head(h.reshape(nz, ny, nx))
    g.finalize_initial_state()
    wc = g.interior("wc").copy()
    g.advance_step()
    assert np.abs(g.interior("wc") - wc).max() <= 1e-15  # (a product and a quotient by the volume)
    assert p.dt_min < g.dt() < 1e-30
    return g.dt()


@pytest.mark.parametrize("shape,mvg", [((1, N, NZ), False), ((N, 1, NZ), True)])
def test_bound_in_any_block(gpu_lib, shape, mvg):
    for seed in range(24):  # (another form's last bit differs for one seed in six)
        assert bound(shape, seed, mvg) == bound((N, 1, NZ), seed, False)
