"""The water content of an initial head on the GPU (table-driven powers for van Genuchten soils)
against the oracle's pow() forms, over dry to saturated heads and every soil model."""
import numpy as np
import pytest

from frehg_gb300 import workloads as W
from frehg_gb300.abi import ReParams

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("soil", ["loam", "sand", "clay", "mvg", "exponential"])
@pytest.mark.parametrize("cells", [1, 63, 65, 30000])
def test_initial_water_content(gpu_lib, oracle_mod, soil, cells):
    """theta = theta_r + (theta_s - theta_r) se: both forms of se are within about two ulps
    (2.2e-16 each), so theta agrees to 1e-15 relative."""
    from frehg_gb300.re_solver import Grid, ReSolver
    s = W.soil({"loam": W.LOAM, "sand": W.SAND, "clay": W.CLAY}.get(soil, W.LOAM))
    if soil == "mvg":
        s.use_mvg = 1
    if soil == "exponential":
        s.use_vg = 0
    rng = np.random.default_rng(cells)
    h = -(10.0 ** rng.uniform(-6.0, 3.0, cells))
    h[: min(cells, 6)] = [0.0, -1e-300, 0.5, -0.02, -1.0 / s.alpha, -1e5][: min(cells, 6)]
    p = ReParams(soil=s)
    out = []
    for r in (ReSolver(Grid(1, 1, cells), p), oracle_mod.OracleRe(1, 1, cells, p)):
        r.initialize_geometry()
        r.set_initial_head(h)
        r.finalize_initial_state()
        out.append(np.asarray(r.interior("wc")).ravel())
    assert np.abs(out[0] - out[1]).max() <= 1e-15 * out[1].max()
    assert (np.abs(out[0] - out[1]) <= 1e-15 * out[1]).all()
