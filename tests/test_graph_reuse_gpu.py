"""A solver handle's captured iterations are not replayed for a system they were not captured for:
buffers that a larger system had the handle allocate again, and a system made anew with the same
number of cells but another shape."""
import numpy as np
import pytest

from frehg_gb300.abi import SolverConfig

from tests.test_linear_seam_gpu import spd_stencil
from tests.test_sor_gpu import assemble_coo

pytestmark = pytest.mark.gpu


def solve(solver, A, shape):
    coef, b = spd_stencil(*shape, seed=sum(shape))
    assemble_coo(A, coef, *shape)
    return solver.solve(A, b).copy()


@pytest.mark.parametrize("pc", ["sor", "jacobi"])
def test_other_systems(gpu_lib, pc):
    from frehg_gb300.linear import makeLinearSolver

    def make():
        s = makeLinearSolver("gb300", SolverConfig("cg", pc, rtol=1e-12, max_it=2000))
        s.setFusedIteration(False)  # (of the Jacobi solve: captured kernels at this size)
        return s

    small, large, turned = (12, 20, 17), (20, 30, 25), (17, 12, 20)
    solver = make()
    A = solver.createSystem(*small)
    want = solve(solver, A, small)
    # a larger system that converges at its initial test: the handle's buffers move, nothing is captured
    B = solver.createSystem(*large)
    coef, b = spd_stencil(*large, seed=1)
    assemble_coo(B, coef, *large)
    assert not solver.solve(B, np.zeros_like(b)).any()
    assert np.array_equal(solve(solver, A, small), want)
    del A, B
    # the same number of cells in another shape, in what the first system freed
    C = solver.createSystem(*turned)
    got = solve(solver, C, turned)
    other = make()
    assert np.array_equal(got, solve(other, other.createSystem(*turned), turned))
