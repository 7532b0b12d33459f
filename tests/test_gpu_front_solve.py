"""The direct solver (mic_front_lu.cu) at the edges of its tree: grids of one leaf, grids one or
two cells wide, odd sizes whose fronts differ within a level, sizes that use shared-memory fronts
only and sizes that use panels -- against a dense host solve of the same matrix."""
import numpy as np
import pytest

from fvmic2d_gb300 import gpu
from fvmic2d_gb300 import workloads as W
from fvmic2d_gb300.mic_types import SubductionOptions

pytestmark = pytest.mark.gpu

SIZES = [(2, 2), (3, 2), (2, 19), (41, 2), (7, 5), (13, 30), (33, 9), (26, 24)]


def _problem(nx, ny, top_type=0):
    """the refined box with viscosities over four decades; a slab that covers the first node column
    alone and a plate thinner than the first cell, so that every other node has its full stencil
    and no pressure cell is cut off"""
    wl = W.vep_slab_box(nx_cells=nx, ny_cells=ny, nm=1, seed=5)
    g = wl.grid
    u = W.splitmix64_uniform(100 * nx + ny, 9 * g.NX * g.NY).reshape(9, g.NY, g.NX)
    wl.nodal.update({"etaN": 10 ** (19 + 4 * u[0]), "etaS": 10 ** (19 + 4 * u[1]), "muN": 1e10 * (0.5 + u[2]),
                     "muS": 1e10 * (0.5 + u[3]), "rho": 30 * (u[4] - 0.5), "rhodot": 0 * u[5],
                     "kThermal": 2.0 + 2.0 * u[6], "Cp": 1000.0 + 250.0 * u[7], "lastT": 273.0 + 1300.0 * u[8]})
    so = SubductionOptions(gx=0.0, gy=10.0, slabVelocity=1e-9, slabAngle=1.55, slabAge=50.0,
                           overridingPlateThickness=0.01 * g.y[1], rootThickness=0.0, rootCenter=-g.LX, rootWidth=0.1 * g.LX,
                           thermalBCTopType=top_type, thermalBCTopValue=273.0)
    return gpu.MicProblem(wl), so


def _dense(P, which):
    rp, c, v, b = P.system(which)
    A = np.zeros((len(b), len(b)))
    A[np.repeat(np.arange(len(b)), np.diff(rp)), c] = v
    return A, b


@pytest.mark.parametrize("nx,ny", SIZES)
def test_solve_matches_dense(nx, ny):
    """Both solves against LAPACK's dense LU.  Residual: partial pivoting keeps it at rounding level
    times the matrix and the solution (n eps, a few 1e-13 at these sizes; bound 1e-12).  Solution:
    within that residual times the matrix's condition after its rows are scaled, which is what
    separates two backward-stable solves."""
    P, so = _problem(nx, ny)
    P.formVEPSystem(so, 3.0e11)
    P.enforceThermalBCs1(so)
    P.formThermalSystem(so, 3.0e11)
    for which in (P.STOKES, P.THERMAL):
        P.linear_solve(which)
        x = P.solution(which)
        A, b = _dense(P, which)
        assert np.all(np.isfinite(x))
        assert np.max(np.abs(A @ x - b)) <= 1e-12 * np.max(np.abs(A).sum(axis=1)) * np.max(np.abs(x)), which
        s = 1.0 / np.abs(A).max(axis=1)
        ref = np.linalg.solve(A * s[:, None], b * s)
        cond = np.linalg.cond(A * s[:, None])
        assert cond < 1e12  # the case itself is not degenerate
        eps = np.finfo(float).eps
        assert np.linalg.norm(x - ref) <= 10 * len(b) * eps * cond * np.linalg.norm(ref), which
    P.close()


def test_zero_column_is_refused_and_the_context_stays_usable():
    """a top boundary type the assembly leaves without an entry (an empty row): the solve reports
    it, and the same context then solves a proper system"""
    P, so = _problem(13, 30, top_type=2)
    P.enforceThermalBCs1(so)
    P.formThermalSystem(so, 3.0e11)
    with pytest.raises(gpu.MicError) as e:
        P.linear_solve(P.THERMAL)
    assert e.value.code == 12  # MIC_ERR_SOLVE
    so.thermalBCTopType = 0
    P.formThermalSystem(so, 3.0e11)
    P.linear_solve(P.THERMAL)
    A, b = _dense(P, P.THERMAL)
    x = P.solution(P.THERMAL)
    assert np.max(np.abs(A @ x - b)) <= 1e-12 * np.max(np.abs(A).sum(axis=1)) * np.max(np.abs(x))
    P.close()


@pytest.mark.parametrize("nx,ny", [(260, 90), (430, 430), (770, 760)])
def test_tall_fronts_residual(nx, ny):
    """Temperatures on grids whose panels are factored by one, two, four and eight blocks (180, 860
    and 1,520 rows at the top), and whose updates take every tile size: the residual stays at
    rounding level (a diagonally dominant matrix, no growth: n eps at most, 2e-10 at the largest, in
    practice a few eps; bound 1e-12)."""
    P, so = _problem(nx, ny)
    P.enforceThermalBCs1(so)
    P.formThermalSystem(so, 3.0e11)
    P.linear_solve(P.THERMAL)
    x = P.solution(P.THERMAL)
    rp, c, v, b = P.system(P.THERMAL)
    assert np.all(np.isfinite(x))
    r = np.add.reduceat(v * x[c], rp[:-1]) - b
    a = np.add.reduceat(np.abs(v), rp[:-1])
    assert np.max(np.abs(r)) <= 1e-12 * np.max(a) * np.max(np.abs(x))
    P.close()


@pytest.mark.parametrize("nx,ny", [(61, 61), (129, 33), (220, 64)])
def test_tall_stokes_fronts_residual(nx, ny):
    """Stokes systems with panels on clusters of blocks, whose pivots wander between the blocks:
    the residual within n eps of the matrix and the solution."""
    P, so = _problem(nx, ny)
    P.formVEPSystem(so, 3.0e11)
    P.linear_solve(P.STOKES)
    x = P.solution(P.STOKES)
    rp, c, v, b = P.system(P.STOKES)
    assert np.all(np.isfinite(x))
    r = np.add.reduceat(v * x[c], rp[:-1]) - b
    a = np.add.reduceat(np.abs(v), rp[:-1])
    assert np.max(np.abs(r)) <= len(b) * np.finfo(float).eps * np.max(a) * np.max(np.abs(x))
    P.close()


@pytest.mark.parametrize("nx,ny", [(260, 90), (300, 300)])
def test_zero_columns_in_tall_fronts(nx, ny):
    """empty rows on a grid whose top panels are factored by clusters: no block has a pivot, the
    solve reports it, and a proper system is solved after it"""
    P, so = _problem(nx, ny, top_type=2)
    P.enforceThermalBCs1(so)
    P.formThermalSystem(so, 3.0e11)
    with pytest.raises(gpu.MicError) as e:
        P.linear_solve(P.THERMAL)
    assert e.value.code == 12  # MIC_ERR_SOLVE
    so.thermalBCTopType = 0
    P.formThermalSystem(so, 3.0e11)
    P.linear_solve(P.THERMAL)
    x = P.solution(P.THERMAL)
    rp, c, v, b = P.system(P.THERMAL)
    r = np.add.reduceat(v * x[c], rp[:-1]) - b
    assert np.max(np.abs(r)) <= len(b) * np.finfo(float).eps * np.max(np.add.reduceat(np.abs(v), rp[:-1])) * np.max(np.abs(x))
    P.close()


@pytest.mark.parametrize("k", [4, 6])
def test_cut_off_pressure_cells_do_not_refuse_the_solve(k):
    """A pair of pressure cells cut off between slab and plate: the matrix is singular, with no empty
    row or column.  The solve goes on with the free pressure at zero: every equation but the one
    that was dropped for it holds to rounding (n eps of the matrix and the solution)."""
    wl, topt = W.subduction_box(nx_cells=128, ny_cells=32, nm=4, seed=10 + k)
    topt.sub.slabAngle = 0.6 + 0.02 * k
    P = gpu.MicProblem(wl)
    P.subductionTimestep(topt, 0.0)
    x = P.solution(P.STOKES)
    rp, c, v, b = P.system(P.STOKES)
    assert np.all(np.isfinite(x))
    r = np.abs(np.add.reduceat(v * x[c], rp[:-1]) - b)
    bound = len(b) * np.finfo(float).eps * np.max(np.add.reduceat(np.abs(v), rp[:-1])) * np.max(np.abs(x))
    assert 0 < np.count_nonzero(r > bound) <= 1 or np.max(r) <= bound
    assert np.all(np.isfinite(P.markers["p"]))
    P.close()
