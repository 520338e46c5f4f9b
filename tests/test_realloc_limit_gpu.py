"""A reallocation that does not settle within its limit is reported, by both of its forms (one block up
to 2,048 columns; above, the host's loop), and a handle goes on afterwards."""
import ctypes as C

import numpy as np
import pytest

from frehg_gb300 import workloads as W
from frehg_gb300.abi import FREHG_ERR_STATE, SolverConfig, check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(3, 2, 40), (45, 45, 17), (46, 45, 17)])
def test_realloc_limit(gpu_lib, shape):
    """From a head of -0.03 m under a ponded top, the first step takes the top cells' head above the air
    entry while more water leaves them than enters: the first sweep fills each of them, so a limit of
    no further sweep is too low, and one of n + 1 is enough."""
    from frehg_gb300.re_solver import Grid, ReSolver
    nx, ny, nz = shape
    w = W.config0("pca", nx=nx, ny=ny, nz=nz)
    w.h0 = np.full((nz, ny, nx), -0.03)
    w.solver = SolverConfig("cg", "jacobi", rtol=1e-12, max_it=5000)
    status = C.c_int(-1)
    for limit, want in ((0, FREHG_ERR_STATE), (nx * ny * nz + 1, 0)):
        g = ReSolver(Grid(nx, ny, nz, w.params.dx, w.params.dy, w.params.dz), w.params)
        w.apply(g)
        check(g._lib.frehg_re_check_realloc_limit(g._h, limit, C.byref(status)), "check")
        assert status.value == want
        g.advance_step()
        g.sync()
        assert g.counters().realloc_sweeps >= 2
