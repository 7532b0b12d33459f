"""retrieveSolutions returns with its fields in place: a caller may read them on another stream."""
import ctypes

import pytest

from fvmic2d_gb300 import gpu
from fvmic2d_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def test_retrieve_of_the_device_solution_waits():
    wl, topt = W.subduction_box(nx_cells=128, ny_cells=32, nm=16, seed=4)  # 1,048,576 markers: a step of milliseconds
    P = gpu.MicProblem(wl)
    P.findMarkerCells()
    P.projectMarkersNodesAll2()
    _, kcont = P.formVEPSystem(topt.sub, topt.dtMax)
    P.linear_solve(P.STOKES)
    P.synchronize()
    rt = ctypes.CDLL("libcudart.so.13")
    stream, nan = ctypes.c_void_p(P.stream()), ctypes.c_int(-1)
    for _ in range(8):
        P.L.mic_step(P.h, wl.dt, wl.dt, 1, None)  # queued, not waited for
    assert rt.cudaStreamQuery(stream) == 600  # cudaErrorNotReady: there is something to wait for
    assert P.L.mic_retrieve_solutions(P.h, None, kcont, ctypes.byref(nan)) == 0
    assert rt.cudaStreamQuery(stream) == 0 and nan.value == 0
    P.close()
