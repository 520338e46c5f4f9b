"""The FP64 Jacobi-PCG loop as one launch per solve (the default up to 622,592 unknowns) over the
shapes of its launch: one block, a few blocks that exchange words, many behind a counter, one to
eight cells per thread, neighbours' directions formed or waited for, the largest size it takes
and the first it does not; against the three-kernel form."""
import numpy as np
import pytest

from tests.test_fused_cg_gpu import solve, spd_coo

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [
    (1, 1, 1), (1, 1, 2), (127, 1, 1), (1, 1, 129),     # a block and its first remainder
    (5, 3, 137), (16, 16, 16),                         # up to 16 blocks
    (19, 7, 131), (37, 29, 19), (2, 3, 9001),          # behind the counter; long rows
    (41, 39, 101), (101, 77, 53), (90, 75, 60), (81, 53, 140), (19, 32768, 1),  # more per thread
    (152, 64, 64), (153, 64, 64)])                     # 622,592 unknowns and more
def test_one_launch_solve_matches_three_kernels(gpu_lib, shape):
    """Iteration counts within one (the dot products are summed over other partitions) and
    solutions to 1e-10 relative, as between the two iteration forms."""
    nx, ny, nz = shape
    rows, cols, vals, _, b = spd_coo(nx, ny, nz, seed=nx + 7 * ny + 13 * nz)
    xd, itd, rd = solve(nx, ny, nz, rows, cols, vals, b, None)
    x3, it3, r3 = solve(nx, ny, nz, rows, cols, vals, b, False)
    assert rd == r3 > 0
    assert abs(itd - it3) <= 1, (itd, it3)
    assert np.abs(xd - x3).max() <= 1e-10 * max(1.0, np.abs(x3).max())


def test_one_launch_solve_stops(gpu_lib):
    """max_it, a NaN right-hand side, a zero one, and an indefinite operator end the loop with the
    three-kernel form's reasons."""
    from frehg_gb300.abi import FrehgError, SolverConfig
    from frehg_gb300.linear import makeLinearSolver
    nx, ny, nz = 24, 20, 16
    rows, cols, vals, _, b = spd_coo(nx, ny, nz, seed=3)
    bad = b.copy()
    bad[11] = np.nan
    flipped = np.where((rows == cols) & (rows % 3 == 0), -vals, vals)
    for max_it, rhs, v in ((3, b, vals), (20000, bad, vals), (20000, 0.0 * b, vals),
                           (20000, b, flipped)):
        out = []
        for fused in (None, False):
            s = makeLinearSolver("gb300", SolverConfig("cg", "jacobi", rtol=1e-12, max_it=max_it))
            s.setFusedIteration(fused)
            A = s.createSystem(nx, ny, nz)
            A.zeroEntries()
            A.addCOO(rows, cols, v)
            A.endAssembly()
            try:
                s.solve(A, rhs)
                code = 0
            except FrehgError as e:
                code = e.code
            out.append((code, s.getConvergedReason(), s.getIterationCount()))
        assert out[0][:2] == out[1][:2], out
        assert abs(out[0][2] - out[1][2]) <= 1, out
