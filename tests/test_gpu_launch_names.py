"""A profile names the form of a kernel that ran: the rules that choose between forms show in it."""
import pytest

from fvmic2d_gb300 import gpu
from fvmic2d_gb300 import workloads as W
from tests.test_gpu_front_solve import _problem

pytestmark = pytest.mark.gpu


def _names(P, f):
    P.profile_enable(8192)
    f()
    names = set(P.profile_read())
    P.profile_enable(0)
    return names


@pytest.mark.parametrize("ncell,form", [(24, "k_corners"), (80, "k_partials")])  # 32 cells an SM and fewer; more
def test_projection_forms(ncell, form):
    wl = W.convection_box(ncell=ncell, nm=2, seed=1)
    P = gpu.MicProblem(wl)
    names = _names(P, lambda: P.step(wl.dt, wl.dt_thermal))
    assert {form + "_basic<first>", form + "_basic<visc>", form + "_centre", "k_corners_centre<scalar>"} <= names
    other = "k_partials" if form == "k_corners" else "k_corners_basic<"
    assert not [n for n in names if n.startswith(other)]
    P.close()


def test_solver_forms():
    P, so = _problem(128, 32)
    P.formVEPSystem(so, 3.0e11)
    names = _names(P, lambda: P.linear_solve(P.STOKES))
    panels = {n for n in names if n.startswith("k_front_panel")}
    assert panels and all(n.endswith((">",)) and "<16" in n for n in panels)
    assert any("_cluster<16," in n for n in panels)
    assert any(n.startswith("k_front_update<16,") for n in names)
    assert {"k_front_small<256>", "k_front_back", "k_front_back_small"} <= names
    P.close()
