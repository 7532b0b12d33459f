"""Bounded waits between blocks, made to run out at once: the call reports it, nothing is lost, and
the context goes on."""
import ctypes

import numpy as np
import pytest

from fvmic2d_gb300 import gpu
from fvmic2d_gb300 import workloads as W
from tests.test_gpu_front_solve import _problem

pytestmark = pytest.mark.gpu

ERR_CELL, ERR_SOLVE = 4, 12
LOOK_BACK = POLLS = 1 << 22  # the defaults


def _refused(f, *a):
    with pytest.raises(gpu.MicError) as e:
        f(*a)
    assert e.value.code == ERR_CELL


@pytest.mark.parametrize("ncell,nm", [(12, 3), (24, 3), (182, 4)])  # one tile; small tiles; large ones
def test_sort_that_gives_up_keeps_the_markers(ncell, nm):
    """The order is the identity, no cell holds a marker, and every later call that waits says so until
    the markers are replaced (one tile waits for none: nothing to give up)."""
    wl = W.convection_box(ncell=ncell, nm=nm, seed=3)
    P = gpu.MicProblem(wl)
    n = P.n
    P.debug_set_wait_limit(P.WAIT_SORT, 0)
    if n <= 1024:
        P.findMarkerCells()
        P.close()
        return
    _refused(P.findMarkerCells)
    assert P.status().bad_cell == n
    assert np.array_equal(P.sorted_ids(), np.arange(n))
    assert not P.cell_start().any()
    P.debug_set_wait_limit(P.WAIT_SORT, LOOK_BACK)
    _refused(P.findMarkerCells)  # sorted now, but what was computed before may not be used
    assert P.status().bad_cell == 0
    got = np.empty(n, dtype=gpu.MARKER_DTYPE)
    assert P.L.mic_markers_download(P.h, got.ctypes.data, n) == ERR_CELL
    for f in ("X", "Y", "T", "Mat", "eta"):  # every marker is still there, in the caller's order
        assert np.array_equal(got[f], wl.markers[f]), f
    P.upload_markers(wl.markers)
    P.findMarkerCells()
    Q = gpu.MicProblem(wl)
    Q.findMarkerCells()
    assert np.array_equal(P.sorted_ids(), Q.sorted_ids())
    P.close()
    Q.close()


def test_step_after_a_sort_that_gave_up_is_refused():
    wl = W.convection_box(ncell=24, nm=3, seed=3)
    P = gpu.MicProblem(wl)
    z, y = ctypes.c_double(0.0), ctypes.c_int(0)
    P.debug_set_wait_limit(P.WAIT_SORT, 0)
    assert P.L.mic_step(P.h, wl.dt, wl.dt_thermal, 1, None) == 0  # asynchronous
    P.debug_set_wait_limit(P.WAIT_SORT, LOOK_BACK)
    assert P.L.mic_step(P.h, wl.dt, wl.dt_thermal, 1, None) == 0  # its binning succeeds
    assert P.L.mic_synchronize(P.h) == ERR_CELL
    assert P.L.mic_step(P.h, wl.dt, wl.dt_thermal, 1, ctypes.byref(z)) == ERR_CELL
    assert P.L.mic_step_pre_stokes(P.h, wl.dt, ctypes.byref(y), ctypes.byref(z)) == ERR_CELL
    assert P.L.mic_step_post_stokes(P.h, wl.dt, 1, ctypes.byref(z)) == ERR_CELL
    assert P.L.mic_step_post_thermal(P.h, wl.dt_thermal, ctypes.byref(z)) == ERR_CELL
    assert P.L.mic_max_abs_sxx(P.h, ctypes.byref(z)) == ERR_CELL
    assert P.L.mic_save_markers_binary(P.h, b"/dev/null", 0.0) == ERR_CELL
    P.upload_markers(wl.markers)
    assert P.L.mic_step(P.h, wl.dt, wl.dt_thermal, 1, ctypes.byref(z)) == 0
    P.close()


@pytest.mark.parametrize("graph", [False, True])
def test_ensemble_reports_a_member_whose_sort_gave_up(graph):
    wls = [W.convection_box(ncell=24, nm=3, seed=s) for s in (1, 2)]
    Ps = [gpu.MicProblem(w) for w in wls]
    E = gpu.MicEnsemble(Ps)
    E.step(graph=graph)
    E.synchronize()
    Ps[1].debug_set_wait_limit(gpu.MicProblem.WAIT_SORT, 0)
    E.step(graph=graph)  # the captured step is taken again with the new limit
    E.step(graph=graph)
    _refused(E.synchronize)
    assert Ps[0].L.mic_synchronize(Ps[0].h) == 0
    assert Ps[1].L.mic_synchronize(Ps[1].h) == ERR_CELL


@pytest.mark.parametrize("nx,ny,which", [(260, 90, 1), (61, 61, 0), (129, 33, 0), (300, 300, 1)])
@pytest.mark.parametrize("polls", [0, 3])
def test_panel_exchange_that_gives_up_fails_the_solve(nx, ny, which, polls):
    """Panels on clusters of two to eight blocks; no poll (every block gives up at its first exchange) and
    a few (some exchanges arrive): the solve fails or is right, and the next one is the undisturbed one's
    equal, bit for bit."""
    P, so = _problem(nx, ny)
    if which == P.STOKES:
        P.formVEPSystem(so, 3.0e11)
    else:
        P.enforceThermalBCs1(so)
        P.formThermalSystem(so, 3.0e11)
    P.linear_solve(which)
    x = P.solution(which)
    P.debug_set_wait_limit(P.WAIT_SOLVE, polls)
    for _ in range(2):  # the launches as they are captured, and the captured graph
        code = P.L.mic_linear_solve(P.h, which)
        assert code == ERR_SOLVE if polls == 0 else code in (0, ERR_SOLVE)
        assert code == ERR_SOLVE or np.array_equal(P.solution(which), x)
    P.debug_set_wait_limit(P.WAIT_SOLVE, POLLS)
    P.linear_solve(which)
    assert np.array_equal(P.solution(which), x)
    P.close()
