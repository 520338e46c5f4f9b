"""The water content of dry soils without a residual content, where theta is the van Genuchten power's
own: both forms (the CUDA library's pow() up to 8,192 cells, the table-driven powers above) against
extended precision."""
import numpy as np
import pytest

from frehg_gb300 import workloads as W
from frehg_gb300.abi import ReParams

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("soil", ["loam", "sand", "clay"])
@pytest.mark.parametrize("cells", [8192, 30000])
def test_dry_water_content(gpu_lib, soil, cells):
    """In units of 2^-53: t = |alpha h|^n within 4 (a power within two ulps) + n < 2.7 (its argument's
    rounding), 1 + t within 7.7, its power with m < 0.63 within 4.9 + 4, the product 1 more: 10."""
    from frehg_gb300.re_solver import Grid, ReSolver
    s = W.soil({"loam": W.LOAM, "sand": W.SAND, "clay": W.CLAY}[soil])
    s.theta_r = 0.0
    h = -(10.0 ** np.random.default_rng(3).uniform(-1.0, 5.0, cells))
    g = ReSolver(Grid(1, 1, cells), ReParams(soil=s))
    g.initialize_geometry()
    g.set_initial_head(h)
    g.finalize_initial_state()
    wc = g.interior("wc").ravel()
    m = 1.0 - 1.0 / s.n
    t = np.abs(np.longdouble(s.alpha) * h) ** np.longdouble(s.n)
    exact = np.longdouble(s.theta_s) * (1 + t) ** np.longdouble(-m)
    assert (h < s.air_entry).all()
    assert float((np.abs(wc - exact) / exact).max()) <= 10 * 2.0 ** -53
