"""The projections on both sides of the line between their two forms (4,864 cells on a GPU of 152
SMs), at the smallest grid and on narrow ones, with empty cells: a step's projected fields, residual
and sub-grid changes against the oracle."""
import numpy as np
import pytest

from fvmic2d_gb300 import gpu, workloads as W
from fvmic2d_gb300.mic_types import PROJECTED_FIELDS
from oracle import oraclepy
from tests.helpers import close

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,nm", [(2, 2, 3), (3, 40, 2), (76, 64, 2), (77, 64, 2), (130, 41, 1)])
def test_step_projections_match_oracle(nx, ny, nm):
    wl = W.vep_slab_box(nx_cells=nx, ny_cells=ny, nm=nm, seed=nx)
    m = wl.markers
    if len(m) > 100:  # a block of empty cells
        gone = (m["X"] > 0.5 * wl.grid.LX) & (m["X"] < 0.6 * wl.grid.LX) & (m["Y"] < 0.5 * wl.grid.LY)
        m["X"][gone] = -1.0
    G = gpu.MicProblem(wl)
    O = oraclepy.OracleProblem(wl)
    for _ in range(2):
        _, rg = G.step(wl.dt, wl.dt_thermal)
        eo, ro = O.step(wl.dt, wl.dt_thermal)
        assert abs(rg - ro) <= 1e-12 * abs(ro)
        for f in PROJECTED_FIELDS + ["srr", "dsxx", "dsyy", "dsxy"]:
            ok, msg = close(G.get_nodal(f), O.get_nodal(f), 1e-12)
            assert ok, (f, msg)
    a, b = G.markers, O.markers
    for f in ("X", "Y", "T", "sxx", "syy", "sxy", "eta", "srr"):
        ok, msg = close(a[f], b[f], 1e-12)
        assert ok, (f, msg)
    G.close()
