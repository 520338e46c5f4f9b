"""The refinement residual that the float-float Picard solve keeps from sweep to sweep, against b - A d
formed on the host in extended precision from the operator the solve used."""
import numpy as np
import pytest

from frehg_gb300 import workloads as W
from frehg_gb300.abi import SolverConfig, check, dptr

pytestmark = pytest.mark.gpu


def refine(shape, pc, rhs, solves=1):
    """(||b - A d||, as reported, ||b||, its terms, kept residual's error, sweeps, inner iterations)
    after two steps of ponded infiltration (None: the third step's own right-hand side, else
    rhs N(0, 1))"""
    from frehg_gb300.re_solver import Grid, ReSolver
    nx, ny, nz = shape
    w = W.config0("picard", nx=nx, ny=ny, nz=nz)
    w.solver = SolverConfig("cg", pc, rtol=1e-12, max_it=20000, precision=1, ir_rtol=1e-12)
    g = ReSolver(Grid(nx, ny, nz, w.params.dx, w.params.dy, w.params.dz), w.params)
    w.apply(g)
    for _ in range(2):
        g.advance_step()
    b = None if rhs is None else rhs * np.random.default_rng(7).standard_normal(nx * ny * nz)
    out = np.zeros(7)
    check(g._lib.frehg_re_check_refinement(g._h, None if b is None else dptr(b), solves, dptr(out)),
          "check_refinement")
    return out


def check_residual(out):
    """The reported norm is a compensated FP32 sum (1e-5) of the kept residual.  That residual's
    error per sweep: sums in three levels, 2^-57 of a power of two at most twice the largest term;
    and an ulp of x~ where an update crosses a power of two, in fewer than one cell in a hundred:
    together below 2^-55 of the norm of the terms' magnitudes."""
    true, reported, b, terms, error, sweeps, _ = out
    assert sweeps >= 2
    assert error <= sweeps * 2.0 ** -55 * terms
    assert abs(true - reported) <= 1e-5 * reported + error
    assert true <= 1e-12 * b * (1 + 1e-5) + error


@pytest.mark.parametrize("pc", ["line", "jacobi"])
@pytest.mark.parametrize("rhs", [None, 1.0, 1e-20])  # 1e-20: the preparation's scaling does not fit
@pytest.mark.parametrize("shape", [(40, 40, 100), (33, 9, 40), (5, 3, 31)])
def test_kept_residual(gpu_lib, shape, rhs, pc):
    check_residual(refine(shape, pc, rhs))


@pytest.mark.parametrize("pc", ["line", "jacobi"])
def test_second_solve(gpu_lib, pc):
    """The same operator solved again without a new assembly: what the preparation made serves it, so
    that it takes the first solve's iterations (one more or less in a sweep, whose right-hand side
    is scaled by another power of two)."""
    first, second = (refine((33, 9, 40), pc, 1.0, solves=n) for n in (1, 2))
    check_residual(second)
    assert abs(second[6] - first[6]) <= second[5]
