"""The direct solver's pivot search (mic_pivot.cuh): the largest of a warp's values to the last bit,
the first of equal ones; and its reciprocal."""
import ctypes
import os
import subprocess
from fractions import Fraction

import numpy as np
import pytest

from fvmic2d_gb300 import build

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def probe(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("probe") / "libpivot.so")
    cmd = [build.nvcc(), *build.ARCH, "-O3", "-std=c++17", "-Xcompiler", "-fPIC", "-shared",
           "-I" + os.path.join(build.ROOT, "include"), "-I" + build.CSRC, os.path.join(HERE, "probe", "pivot_probe.cu"),
           "-o", out]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    L = ctypes.CDLL(out)

    def run(a, p):
        a, p = np.ascontiguousarray(a, dtype=np.float64), np.ascontiguousarray(p, dtype=np.float64)
        best, r = np.zeros(len(a), dtype=np.int32), np.zeros(len(p))
        ptr = lambda v: v.ctypes.data_as(ctypes.c_void_p)
        assert L.pivot_probe(ptr(a), len(a), ptr(best), ptr(p), len(p), ptr(r)) == 0
        return best, r

    return run


def test_search_finds_the_largest_value_to_the_last_bit(probe):
    rng = np.random.default_rng(5)
    sets = [rng.standard_normal((64, 32)) * 10.0 ** rng.integers(-300, 300, (64, 32))]
    one = rng.uniform(1.0, 2.0, (192, 1))
    for ulps in (2 ** 20, 2 ** 33, 2 ** 43):  # values that agree in 32, 19 and 9 bits of the mantissa
        sets.append(one + rng.integers(0, ulps, (192, 32)) * np.spacing(1.0))
    sets.append(rng.integers(-1, 2, (64, 32)).astype(float))  # many equal ones
    tiny = rng.integers(0, 4, (64, 32)) * 5e-324
    sets.append(tiny)
    odd = rng.standard_normal((64, 32))
    odd[rng.random(odd.shape) < 0.5] = np.nan
    odd[::3, 7] = -np.inf
    sets.append(odd)
    a = np.concatenate(sets) * np.where(rng.random((sum(map(len, sets)), 32)) < 0.5, -1.0, 1.0)
    best, _ = probe(a, np.ones(1))
    want = np.argmax(np.where(np.isnan(a), -1.0, np.abs(a)), axis=1)
    assert np.array_equal(best, want)


def test_reciprocal_is_accurate_to_rounding(probe):
    """|r p - 1|: half a unit in the last place of r, at most 2^-53 of it, and the iteration's 2^-66."""
    rng = np.random.default_rng(6)
    p = np.concatenate([rng.uniform(1.0, 2.0, 4000), 2.0 ** np.arange(-1000.0, 1000.0, 7), 1.0 + np.arange(64) * 2.0 ** -52,
                        2.0 - np.arange(1, 65) * 2.0 ** -52, rng.uniform(1, 2, 500) * 2.0 ** rng.integers(-1020, 1020, 500)])
    p[::2] *= -1.0
    _, r = probe(np.zeros((1, 32)), p)
    worst = max(abs(Fraction(float(x)) * Fraction(float(y)) - 1) for x, y in zip(p, r))
    assert worst <= Fraction(1, 2 ** 53) * (1 + Fraction(1, 2 ** 12))
    _, z = probe(np.zeros((1, 32)), np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 5e-324]))
    assert z[0] == 0.0 and z[1] == 0.0 and z[2] == 0.0 and z[3] == 0.0 and np.isnan(z[4]) and z[5] == np.inf
