"""Pressure cells cut off between slab and plate, groups of two to hundreds: the Stokes matrix is
singular, with no empty row or column.  The solve goes on with the group's free pressure at zero."""
import numpy as np
import pytest

from fvmic2d_gb300 import gpu
from fvmic2d_gb300 import workloads as W
from fvmic2d_gb300.mic_types import SubductionOptions

pytestmark = pytest.mark.gpu


def _free_groups(rp, c, ncells):
    """groups of pressure cells linked by the equations that hold two pressures, without those that an
    equation holds alone"""
    p = [c[rp[r]:rp[r + 1]] for r in range(len(rp) - 1)]
    p = [q[q % 3 == 2] // 3 for q in p]
    parent = list(range(ncells))

    def root(a):
        while parent[a] != a:
            a = parent[a]
        return a

    held = set()
    for q in p:
        for b in q[1:]:
            parent[max(root(q[0]), root(b))] = min(root(q[0]), root(b))
        if len(q) == 1:
            held.add(int(q[0]))
    held = {root(a) for a in held}
    groups = {}
    for a in range(ncells):
        groups.setdefault(root(a), []).append(a)
    return [np.array(g) for r, g in groups.items() if r not in held and len(g) > 1]


def _check(P, sizes):
    rp, c, v, b = P.system(P.STOKES)
    x = P.solution(P.STOKES)
    groups = _free_groups(rp, c, len(b) // 3)
    assert sorted(len(g) for g in groups) == sorted(sizes)
    assert np.all(np.isfinite(x))
    for g in groups:  # the free constant is near zero beside the pressures' differences, which are not free
        p = x[2::3][g]
        assert np.max(np.abs(p)) <= 2.0 * (np.max(p) - np.min(p))
    # every equation, row by row, but the one of a group that holds its pressure in the solve
    r = np.abs(np.add.reduceat(v * x[c], rp[:-1]) - b)
    scale = np.add.reduceat(np.abs(v) * np.abs(x)[c], rp[:-1]) + np.abs(b)
    row = np.maximum.reduceat(np.abs(v), rp[:-1]) * np.max(np.abs(x).reshape(-1, 3), axis=0)[np.arange(len(b)) % 3]
    off = np.flatnonzero(r > len(b) * np.finfo(float).eps * np.maximum(scale, row))
    assert len(off) <= len(groups)
    assert all(q % 3 == 2 and any(q // 3 in g for g in groups) for q in off)


@pytest.mark.parametrize("k", [4, 6])
def test_pairs_in_a_time_step(k):
    wl, topt = W.subduction_box(nx_cells=128, ny_cells=32, nm=4, seed=10 + k)
    topt.sub.slabAngle = 0.6 + 0.02 * k
    P = gpu.MicProblem(wl)
    P.subductionTimestep(topt, 0.0)
    _check(P, [2])
    assert np.max(np.abs(P.markers["p"])) < 1e12
    P.close()


@pytest.mark.parametrize("nx,ny,width,sizes", [(128, 32, 0.1, [40]), (256, 64, 0.05, [325]), (256, 64, 0.1, [2, 143]),
                                               (400, 100, 0.1, [324])])
def test_large_groups_below_a_thick_root(nx, ny, width, sizes):
    """a plate root half the box deep beside the slab encloses a pocket of mantle"""
    wl, topt = W.subduction_box(nx_cells=nx, ny_cells=ny, nm=2, seed=4)
    g = wl.grid
    so = topt.sub
    so.rootThickness, so.rootCenter, so.rootWidth = 0.5 * g.LY, 0.2 * g.LX, width * g.LX
    P = gpu.MicProblem(wl)
    P.findMarkerCells()
    P.projectMarkersNodesAll2()
    P.formVEPSystem(so, 3.0e11)
    P.linear_solve(P.STOKES)
    _check(P, sizes)
    P.close()
