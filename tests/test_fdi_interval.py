"""The interval arithmetic of the Fermi-Dirac family's kernel (fd_interval of
csrc/bnsn_fx.cuh), compiled by g++, against exact rationals.

The argument is held in units of 2^-56 (truncated below |x| = 1/8); the position is twice
the offset over the width, its difference from the exact one at most that unit over half
the narrower width plus two roundings.
"""

import ctypes
import os
import subprocess
from fractions import Fraction

import numpy as np
import pytest

from bns_nurates_gb300 import fdi_tables as ft

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "bns_nurates_gb300", "csrc")
SRC = """
#include "bnsn_fx.cuh"
extern "C" void positions(const double* x, double* v, int* i, long n)
{
    for (long k = 0; k < n; ++k)
        v[k] = bnsn::fx::fd_interval(x[k], i + k);
}
"""
TOL = Fraction(1, 2 ** 56) * Fraction(32, 11) + Fraction(2, 2 ** 53)


@pytest.fixture(scope="module")
def positions(tmp_path_factory):
    d = tmp_path_factory.mktemp("fdi")
    (d / "t.cpp").write_text(SRC)
    so = str(d / "t.so")
    subprocess.check_call(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-I", CSRC,
                           str(d / "t.cpp"), "-o", so])
    lib = ctypes.CDLL(so)

    def f(x):
        x = np.ascontiguousarray(x, dtype=np.float64)
        v, i = np.empty(x.size), np.empty(x.size, dtype=np.int32)
        ptr = ctypes.c_void_p
        lib.positions(ptr(x.ctypes.data), ptr(v.ctypes.data), ptr(i.ctypes.data),
                      ctypes.c_long(x.size))
        return v, i
    return f


def exact(x):
    """Interval and position of x as rationals."""
    x = Fraction(float(x))
    wide = x >= ft.X_MID
    lo, w = (Fraction(ft.X_MID), Fraction(ft.WIDE)) if wide else (Fraction(ft.X_LO),
                                                                 Fraction(ft.WIDTH))
    i = (x - lo) // w
    return int(i) + (ft.NARROW if wide else 0), 2 * (x - lo - i * w) / w - 1


def test_interval_and_position(positions):
    edges = np.array([ft.piece(i)[0] - ft.piece(i)[1] for i in range(ft.PIECES)])
    tiny = np.concatenate([10. ** np.arange(-320., 0.), [5e-324, 0.125, 1. / 16., 0.1249999]])
    x = np.concatenate([edges, np.nextafter(edges, 200.), np.nextafter(edges[1:], -200.),
                        np.random.default_rng(1).uniform(-4., 100., 4000), tiny, -tiny,
                        [0., -0., np.nextafter(100., 0.)]])
    v, i = positions(x)
    for k in range(x.size):
        n, pos = exact(x[k])
        if i[k] != n:  # a negative argument truncated to the interval's edge
            assert -0.125 < x[k] < 0. and i[k] == n + 1
            continue
        assert abs(Fraction(float(v[k])) - pos) <= TOL, (x[k], v[k])
        assert -1. <= v[k] <= 1.
