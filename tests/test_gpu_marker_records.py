"""Marker records to device columns and back, around the edges of a block's records: after the
columns were sorted every field that the cell search does not write comes back in upload order,
padding as zeros."""
import numpy as np
import pytest

from fvmic2d_gb300 import gpu, workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 127, 128, 129, 20011, 90001])
def test_records_round_trip(n):
    wl = W.convection_member(40, 40, 1, 1, 1e4, 10.0, 1)
    rng = np.random.default_rng(n)
    raw = rng.integers(0, 256, size=(n, gpu.MARKER_DTYPE.itemsize), dtype=np.uint8)
    mk = raw.reshape(-1).view(gpu.MARKER_DTYPE).copy()
    mk["X"], mk["Y"] = rng.random(n), rng.random(n)
    mk["Mat"] = 0
    P = gpu.MicProblem(wl, markers=mk, capacity=n)
    P.findMarkerCells()
    got = P.markers
    assert np.all(got["cellX"] >= 0) and len(np.unique(got["cellX"])) > min(n, 30) // 2
    seen = np.zeros(gpu.MARKER_DTYPE.itemsize, bool)
    for name in gpu.MARKER_DTYPE.names:
        dt, off = gpu.MARKER_DTYPE.fields[name][:2]
        seen[off:off + dt.itemsize] = True
        if name not in ("cellX", "cellY", "cpu"):  # what the cell search writes
            assert got[name].tobytes() == mk[name].tobytes(), name
    assert not got.view(np.uint8).reshape(n, -1)[:, ~seen].any()
    P.close()
