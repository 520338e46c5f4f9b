"""The bounded waits of the one-launch FP64 solve and of the SOR sweeps: with a block (a tile) that never
delivers its values every wait for them runs out, the solve reports it and the handle goes on."""
import ctypes as C

import numpy as np
import pytest

from frehg_gb300.abi import FREHG_ERR_CUDA, SolverConfig, check, dptr

from tests.test_linear_seam_gpu import spd_stencil
from tests.test_sor_gpu import assemble_coo

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pc,shape,want", [
    ("jacobi", (8, 8, 16), FREHG_ERR_CUDA),      # words between a few blocks
    ("jacobi", (16, 16, 32), FREHG_ERR_CUDA),    # a counter before the words
    ("jacobi", (40, 50, 50), FREHG_ERR_CUDA),    # and the neighbours' words
    ("jacobi", (2, 2, 5), 0),                    # one block: no waits
    ("sor", (50, 1, 40), FREHG_ERR_CUDA),        # tiles of a one-block solve
    ("sor", (60, 1, 70), FREHG_ERR_CUDA),        # sweeps that round, sweeps that fuse
    ("sor", (20, 15, 17), FREHG_ERR_CUDA),
    ("sor", (5, 2, 700), 0)])                    # one tile
def test_waits_run_out(gpu_lib, pc, shape, want):
    from frehg_gb300.linear import makeLinearSolver
    coef, b = spd_stencil(*shape, seed=sum(shape))
    s = makeLinearSolver("gb300", SolverConfig("cg", pc, rtol=1e-12, max_it=2000))
    A = s.createSystem(*shape)
    assemble_coo(A, coef, *shape)
    before = s.solve(A, b).copy()
    status = C.c_int(-1)
    check(gpu_lib.frehg_cg_check_waits(s._h, A._h, dptr(b), 1 << 12, C.byref(status)), "check_waits")
    assert status.value == want
    assert np.array_equal(s.solve(A, b), before)
