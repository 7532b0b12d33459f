"""The direct solver's error against a refined solution: no larger than that of an elimination of the
band from one end, whose updates sum a panel's products before they subtract them."""
import numpy as np
import pytest
import scipy.sparse as sp
import scipy.sparse.linalg as sl

from tests.test_gpu_front_solve import _problem

pytestmark = pytest.mark.gpu

# |x - x*| / |x*| (2-norms) of such a band solver with partial pivoting, geometric mean over the four
# systems of each set
BAND = {"thermal, 4,000 cells": (1, [(128, 32), (120, 36), (140, 30), (100, 44)], 2.44e-16),
        "thermal, 17,000 cells": (1, [(256, 64), (240, 70), (280, 60), (200, 88)], 2.88e-16),
        "Stokes, 4,000 cells": (0, [(128, 32), (120, 36), (140, 30), (100, 44)], 4.53e-13)}


def _refined(rp, c, v, b):
    """the host's LU and refinement with residuals in long double until nothing changes"""
    L, n = np.longdouble, len(b)
    rows = np.repeat(np.arange(n), np.diff(rp))
    s = 1.0 / np.maximum.reduceat(np.abs(v), rp[:-1])
    lu = sl.splu(sp.csc_matrix((v * s[rows], (rows, c)), shape=(n, n)))
    x, vl, bl = lu.solve(b * s).astype(L), v.astype(L), b.astype(L)
    for _ in range(8):
        d = lu.solve(((bl - np.add.reduceat(vl * x[c], rp[:-1])) * s).astype(np.float64))
        x = x + d.astype(L)
    assert np.linalg.norm(d) <= 1e-18 * np.linalg.norm(x.astype(np.float64))
    return x


@pytest.mark.parametrize("kind", sorted(BAND))
def test_error_is_no_larger_than_a_band_elimination_s(kind):
    which, sizes, band = BAND[kind]
    errs = []
    for nx, ny in sizes:
        P, so = _problem(nx, ny)
        if which == P.STOKES:
            P.formVEPSystem(so, 3.0e11)
        else:
            P.enforceThermalBCs1(so)
            P.formThermalSystem(so, 3.0e11)
        P.linear_solve(which)
        y = P.solution(which).astype(np.longdouble)
        x = _refined(*P.system(which))
        errs.append(float(np.sqrt(((y - x) ** 2).sum() / (x * x).sum())))
        P.close()
    assert np.exp(np.mean(np.log(errs))) <= band
