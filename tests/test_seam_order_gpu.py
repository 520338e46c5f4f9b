"""COO triplets in row order, in reverse and shuffled, on grids with axes of length 1 and 2: the same
operator (each entry given as two exact halves), and a wrong neighbour after right ones is refused."""
import numpy as np
import pytest

from frehg_gb300.abi import FREHG_ERR_BAD_ARG, FrehgError, SolverConfig

pytestmark = pytest.mark.gpu


def triplets(nx, ny, nz):
    rng = np.random.default_rng(nx * 100 + ny * 10 + nz)
    n = nx * ny * nz
    r = np.arange(n)
    k, i, j = r % nz, (r // nz) % nx, r // (nz * nx)
    rows, cols, vals = [], [], []
    diag = rng.uniform(0.5, 1.0, n)
    for off, ok in ((1, k < nz - 1), (nz, i < nx - 1), (nz * nx, j < ny - 1)):
        q = r[ok]
        v = -rng.uniform(0.1, 2.0, q.size)
        np.add.at(diag, q, -v)
        np.add.at(diag, q + off, -v)
        rows += [q, q + off]
        cols += [q + off, q]
        vals += [v, v]
    rows, cols, vals = (np.concatenate(a) for a in (rows + [r], cols + [r], vals + [diag]))
    rows, cols, vals = np.tile(rows, 2), np.tile(cols, 2), np.tile(vals / 2, 2)
    return rows.astype(np.int32), cols.astype(np.int32), vals, rng.standard_normal(n)


@pytest.mark.parametrize("shape", [(1, 1, 1), (2, 1, 5), (1, 4, 2), (5, 4, 3), (3, 2, 1)])
def test_triplet_order(gpu_lib, shape):
    """The halves of an entry add to it exactly in either order, so all orders give the same bits."""
    from frehg_gb300.linear import makeLinearSolver
    rows, cols, vals, b = triplets(*shape)
    s = makeLinearSolver("gb300", SolverConfig("cg", "jacobi", rtol=1e-12, max_it=2000))
    out = []
    rng = np.random.default_rng(3)
    for order in (np.argsort(rows, kind="stable"), np.argsort(-rows, kind="stable"),
                  rng.permutation(rows.size)):
        A = s.createSystem(*shape)
        A.zeroEntries()
        A.addCOO(rows[order], cols[order], vals[order])
        A.endAssembly()
        out.append(s.solve(A, b).copy())
    assert np.array_equal(out[0], out[1]) and np.array_equal(out[0], out[2])
    A = s.createSystem(*shape)
    A.zeroEntries()
    n = rows.max() + 1
    for bad in ((0, n), (n, 0), (-1, 0)):
        with pytest.raises(FrehgError) as e:
            A.addCOO(np.array([0, bad[0]], np.int32), np.array([0, bad[1]], np.int32), np.ones(2))
        assert e.value.code == FREHG_ERR_BAD_ARG
    if shape == (5, 4, 3):  # the last level of a column and the first of the next are no neighbours
        with pytest.raises(FrehgError):
            A.addCOO(np.array([1, 2], np.int32), np.array([2, 3], np.int32), np.ones(2))
