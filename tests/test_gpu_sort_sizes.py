"""The stable sort by cell at the edges of its tiles and passes: marker counts around one tile, many
tiles and the change of tile size; one, two and three digits; markers spread out, in one cell, and
all outside the domain -- the permutation and the cell offsets against NumPy's stable sort."""
import numpy as np
import pytest

from fvmic2d_gb300 import gpu, workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("where", ["spread", "one_cell", "outside", "mixed"])
@pytest.mark.parametrize("ncell,n", [(7, 1), (7, 1023), (64, 1024), (64, 1025), (64, 33 * 1024 + 7), (150, 524288),
                                     (150, 524289), (150, 3 * 4096 * 64 + 1)])
def test_sort_matches_stable_argsort(ncell, n, where):
    wl = W.convection_member(ncell, ncell, 1, 1, 1e4, 10.0, 1)
    rng = np.random.default_rng(n)
    X, Y = rng.random(n), rng.random(n)
    if where == "one_cell":
        X, Y = 0.3 + 1e-4 * X / ncell, 0.6 + 1e-4 * Y / ncell
    elif where == "outside":
        X = X + 2.0
    elif where == "mixed":
        X[::3] = -1.0
        Y[1::7] = np.nan
    mk = np.zeros(n, dtype=gpu.MARKER_DTYPE)
    mk["X"], mk["Y"] = X, Y
    P = gpu.MicProblem(wl, markers=mk)
    out = P.findMarkerCells()
    ids, cs = P.sorted_ids(), P.cell_start()
    got = P.markers
    g = wl.grid
    inside = (X >= 0) & (Y >= 0) & (X <= g.LX) & (Y <= g.LY)
    cx = np.clip(np.searchsorted(g.x, X, side="right") - 1, 0, g.NX - 2)
    cy = np.clip(np.searchsorted(g.y, Y, side="right") - 1, 0, g.NY - 2)
    qx, qy = X >= g.xc[cx + 1], Y >= g.yc[cy + 1]
    key = np.where(inside, 4 * (cy * (g.NX - 1) + cx) + 2 * qy + qx, 4 * g.ncells)
    assert out == np.count_nonzero(~inside)
    assert np.array_equal(got["cellX"], np.where(inside, cx, -1))
    assert np.array_equal(ids, np.argsort(key, kind="stable"))
    per = np.bincount(key // 4, minlength=g.ncells + 1)
    assert np.array_equal(cs, np.concatenate([[0], np.cumsum(per)]))
    # again from the sorted order, with the cells as hints: the same order
    P.findMarkerCells()
    assert np.array_equal(P.sorted_ids(), np.argsort(key, kind="stable"))
    P.close()
