"""PCSOR of a section (two axes) rounds as the sequential sweeps do at every size: in the one-block
solve (up to 3,600 cells) and above it, with its lines along either axis."""
from fractions import Fraction

import numpy as np
import pytest

from frehg_gb300.abi import SolverConfig

from tests.test_linear_seam_gpu import spd_stencil
from tests.test_sor_gpu import assemble_coo

pytestmark = pytest.mark.gpu


def fma(a, b, c):
    return float(Fraction(a) * Fraction(b) + Fraction(c))


def grid_dot(a, b):
    """a.b in blocks of 256 threads with up to four cells each, butterflies over the warps' lanes,
    the warps and the blocks"""
    n = len(a)
    blocks = -(-n // 1024)
    v = [0.0] * (blocks * 256)
    for c in range(n):
        t = c % (blocks * 256)
        v[t] = fma(a[c], b[c], v[t])

    def butterfly(x):
        x = np.array(x).reshape(-1, 32)
        for o in (16, 8, 4, 2, 1):
            x = x + x[:, np.arange(32) ^ o]
        return x[:, 0]

    def block(x):  # 256 threads
        w = butterfly(x)
        return butterfly(np.concatenate([w, np.zeros(24)]))[0]

    parts = [block(v[256 * q:256 * q + 256]) for q in range(blocks)]
    return block(parts + [0.0] * (256 - blocks))


@pytest.mark.parametrize("shape", [(50, 1, 30), (61, 1, 65), (65, 1, 61), (1, 60, 70), (70, 60, 1),
                                   (58, 66, 1), (1, 401, 10)])
def test_section_bits(gpu_lib, shape):
    """A solve that converges in its first iteration returns alpha z, z = M^-1 b; compared with the
    sequential sweeps (terms in column order, y / (1/d)) and the sums' order, bit for bit."""
    from frehg_gb300.linear import makeLinearSolver
    nx, ny, nz = shape
    n = nx * ny * nz
    coef, b = spd_stencil(nx, ny, nz, seed=nx * 100 + ny * 10 + nz)
    solver = makeLinearSolver("gb300", SolverConfig("cg", "sor", rtol=0.9))
    A = solver.createSystem(nx, ny, nz)
    assemble_coo(A, coef, nx, ny, nz)
    x = solver.solve(A, b)
    assert solver.getIterationCount() == 1
    a = coef.tolist()
    inv = (1.0 / coef[:, 0]).tolist()
    lower = ((3, -nz * nx), (1, -nz), (5, -1))
    upper = ((6, 1), (2, nz), (4, nz * nx))
    z = [0.0] * n
    for c in range(n):
        s = float(b[c])
        for q, off in lower:
            if a[c][q] != 0.0:
                s -= a[c][q] * z[c + off]
        z[c] = s * inv[c]
    for c in reversed(range(n)):
        s = z[c] / inv[c]
        for q, off in upper:
            if a[c][q] != 0.0:
                s -= a[c][q] * z[c + off]
        z[c] = s * inv[c]
    w = []
    for c in range(n):
        v = a[c][0] * z[c]
        for q, off in ((5, -1), (6, 1), (1, -nz), (2, nz), (3, -nz * nx), (4, nz * nx)):
            if a[c][q] != 0.0:
                v = fma(a[c][q], z[c + off], v)
        w.append(v)
    alpha = grid_dot(z, b.tolist()) / grid_dot(z, w)
    assert np.array_equal(x, alpha * np.array(z))
