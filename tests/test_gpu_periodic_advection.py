"""advectMarkersRK on grids periodic in x: the product build's coefficient forms against the FMA-free
build's own divisions, at the smallest and at odd sizes, with a free-slip and a moving top wall, for
a time step that carries markers over the seam and more than a cell."""
import numpy as np
import pytest

from fvmic2d_gb300 import gpu, workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,top", [(4, 3, 1), (17, 5, 0), (33, 8, 1), (130, 9, 0)])
def test_product_matches_exact_build(nx, ny, top):
    """Bilinear interpolation in the two forms differs by a few roundings of the corner values, RK4
    by a few of those: 1e-13 of a field's largest value, 1e-12 with the rotation's products."""
    out = []
    for exact in (True, False):
        wl = W.periodic_box(nx_cells=nx, ny_cells=ny, nm=4, seed=nx)
        wl.bcs.mechBCTop.type[0] = top
        wl.bcs.mechBCTop.value[0] = 4e-10 if top == 0 else 0.0
        P = gpu.MicProblem(wl, exact=exact)
        P.findMarkerCells()
        P.advectMarkersRK(2.5 * wl.dt)
        out.append(P.markers)
        P.close()
    a, b = out
    moved = np.abs(a["X"] - W.periodic_box(nx_cells=nx, ny_cells=ny, nm=4, seed=nx).markers["X"])
    assert np.count_nonzero(moved > 0.5 * wl.grid.LX) > 0  # some crossed the seam
    for f in ("X", "Y", "VX", "VY", "wxy", "sxx", "syy", "sxy", "Eii"):
        assert np.max(np.abs(a[f] - b[f])) <= 1e-12 * np.max(np.abs(a[f])), f
