"""A triplet whose row is outside the system is refused also as the first one of a call, whatever its
column (row -1 with the neighbours' columns of a row before the first), and leaves the system as it
was."""
import numpy as np
import pytest

from frehg_gb300.abi import FREHG_ERR_BAD_ARG, FrehgError, SolverConfig

pytestmark = pytest.mark.gpu

NX, NY, NZ = 4, 3, 5
N = NX * NY * NZ


@pytest.mark.parametrize("row", [-1, -2, N, -2 ** 31, 2 ** 31 - 1])
@pytest.mark.parametrize("col", [0, NZ - 1, NZ * NX - 1, -1, N - 1])
def test_first_row_outside(gpu_lib, row, col):
    from frehg_gb300.linear import makeLinearSolver
    s = makeLinearSolver("gb300", SolverConfig("cg", "jacobi", rtol=1e-12, max_it=100))
    A = s.createSystem(NX, NY, NZ)
    A.zeroEntries()
    r = np.arange(N, dtype=np.int32)
    A.addCOO(r, r, np.full(N, 2.0))
    for call in (lambda: A.addCOO(np.array([row], np.int32), np.array([col], np.int32), np.ones(1)),
                 lambda: A.addRow(row, [col], [1.0])):
        with pytest.raises(FrehgError) as e:
            call()
        assert e.value.code == FREHG_ERR_BAD_ARG
    A.endAssembly()
    b = np.arange(1.0, N + 1.0)
    assert np.allclose(s.solve(A, b), 0.5 * b, rtol=1e-14, atol=0.0)
