"""The direct solver's host logic when a launch is refused, over a CUDA runtime without a device
(tests/probe/fakecudart.c): the solve fails, no graph without that launch is kept or run, and the next
solve captures again."""
import os
import subprocess
import sys

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)

CHILD = """
import ctypes, sys
sys.path.insert(0, %r)
from fvmic2d_gb300 import gpu
from tests.test_gpu_front_solve import _problem
F = ctypes.CDLL(None)
P, so = _problem(%d, %d)
P.enforceThermalBCs1(so)
P.formThermalSystem(so, 3.0e11)
profile = %d
if profile:  # launches timed one by one: no graph
    P.profile_enable(4096)
F.fake_refuse(b"%s")
code = P.L.mic_linear_solve(P.h, P.THERMAL)
assert F.fake_refused() == 1, F.fake_refused()  # nothing was launched behind it
assert code == 2, code  # MIC_ERR_CUDA
assert F.fake_graph_launches() == 0
F.fake_refuse(b"")
code = P.L.mic_linear_solve(P.h, P.THERMAL)
assert code == 0, code
if not profile:
    assert F.fake_captures() == 2 and F.fake_graph_launches() == 1, (F.fake_captures(), F.fake_graph_launches())
    assert P.L.mic_linear_solve(P.h, P.THERMAL) == 0
    assert F.fake_captures() == 2 and F.fake_graph_launches() == 2
print("done")
"""


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    from fvmic2d_gb300 import build

    if not os.path.exists(build.lib_path()):
        build.build(variants=["libmic_gb300.so"])
    out = str(tmp_path_factory.mktemp("fake") / "libfakecudart.so")
    subprocess.run([os.environ.get("CC", "gcc"), "-O1", "-fPIC", "-shared", "-Wall", "-o", out,
                    os.path.join(HERE, "probe", "fakecudart.c")], check=True)
    return out


@pytest.mark.parametrize("profile", [0, 1])
@pytest.mark.parametrize("nx,ny,kernel", [(33, 9, "k_front_small"), (200, 120, "k_front_gather"), (200, 120, "k_front_panelILi"),
                                          (200, 120, "k_front_panel_cluster"), (200, 120, "k_front_update"),
                                          (513, 129, "k_front_solve"), (200, 120, "k_front_border"),
                                          (33, 9, "k_front_back_small"), (200, 120, "k_front_backE"), (33, 9, "k_band_width")])
def test_refused_launch_fails_the_solve_and_keeps_no_graph(fake, nx, ny, kernel, profile):
    env = dict(os.environ, LD_PRELOAD=fake)
    r = subprocess.run([sys.executable, "-c", CHILD % (ROOT, nx, ny, profile, kernel)], env=env, capture_output=True,
                       text=True, timeout=120)
    assert r.returncode == 0 and r.stdout.strip().endswith("done"), r.stderr[-2000:]
