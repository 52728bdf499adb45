"""The fixed-point elementary functions and Fermi integrals of
csrc/bnsn_fx.cuh: the same source compiled by g++ against mpmath.

Tolerances follow from the number formats: the 64-bit results are rounded to a
double once (2^-53) after truncations of a few 2^-62; Fermi integrals add the
rounding of table entries that keep at least 57 bits; x^p adds |p| ln 2 times
the 2^-56 of log2 x; the polynomial branch above y = 36 has up to four
roundings.
"""

import ctypes
import os
import subprocess

import numpy as np
import pytest

mpmath = pytest.importorskip("mpmath")
mp = mpmath.mp
CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "bns_nurates_gb300", "csrc")
SRC = """
#include "bnsn_fx.cuh"
using namespace bnsn;
extern "C" {
void t_exp(const double* x, const double*, double* o, long n) { for (long i = 0; i < n; ++i) o[i] = fx::exp(x[i]); }
void t_pow(const double* x, const double* p, double* o, long n) { for (long i = 0; i < n; ++i) o[i] = fx::pow(x[i], p[i]); }
void t_fd(const double* x, const double*, double* o, long n) { for (long i = 0; i < n; ++i) fx::fd_orders<0, 5>(x[i], o + 6 * i); }
void t_phi(const double* x, const double*, double* o, long n) { for (long i = 0; i < n; ++i) fx::fd_orders<0, 5, true>(x[i], o + 6 * i); }
void t_log(const double* x, const double*, double* o, long n) { for (long i = 0; i < n; ++i) o[i] = fx::log(x[i]); }
void t_log2(const double* x, const double*, double* o, long n) { for (long i = 0; i < n; ++i) o[i] = fx::log2(x[i]); }
void t_quot(const double* x, const double* p, double* o, long n) { for (long i = 0; i < n; ++i) o[i] = fx::quot(x[i], p[i]); }
void t_div(const double* x, const double* p, double* o, long n) { for (long i = 0; i < n; ++i) o[i] = fx::div(x[i], p[i]); }
}
"""


@pytest.fixture(scope="module")
def call(tmp_path_factory):
    d = tmp_path_factory.mktemp("fx")
    (d / "t.cpp").write_text(SRC)
    so = str(d / "t.so")
    subprocess.check_call(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-I", CSRC,
                           str(d / "t.cpp"), "-o", so])
    lib = ctypes.CDLL(so)

    def f(name, x, p=None, width=1):
        x = np.ascontiguousarray(x, dtype=np.float64)
        p = x if p is None else np.ascontiguousarray(p, dtype=np.float64)
        out = np.empty(x.size * width)
        ptr = ctypes.c_void_p
        getattr(lib, name)(ptr(x.ctypes.data), ptr(p.ctypes.data), ptr(out.ctypes.data),
                           ctypes.c_long(x.size))
        return out.reshape(-1, width) if width > 1 else out
    return f


def worst(got, want):
    return max(abs(float(mp.mpf(float(g)) / w - 1)) for g, w in zip(got, want))


def fermi(k, y):
    """F_k(y) from the polylogarithm below 0 and the reflection above."""
    a = abs(y)
    r = mp.log1p(mp.exp(-a)) if k == 0 else -mp.re(mp.polylog(k + 1, -mp.exp(-a)))
    if y > 0:
        eta = [mp.mpf(1) / 2] + [mp.altzeta(2 * n) for n in (1, 2, 3)]
        r = (-1) ** k * r + sum(2 * eta[n] * a ** (k + 1 - 2 * n) / mp.factorial(k + 1 - 2 * n)
                                for n in range(4) if k + 1 - 2 * n >= 0)
    return mp.factorial(k) * r


@pytest.mark.parametrize("lo,hi", [(-1., 1.), (-45., 45.), (-707.9, 707.9)])
def test_exp(call, lo, hi):
    mp.dps = 40
    x = np.concatenate([np.random.default_rng(1).uniform(lo, hi, 1500), [0., -0., 1e-18, -1e-18]])
    assert worst(call("t_exp", x), [mp.exp(mp.mpf(float(v))) for v in x]) <= 2. ** -52


def test_exp_outside_the_fixed_point_range(call):
    x = np.array([-800., -np.inf, 800., np.inf, np.nan, -745., 709.5])
    with np.errstate(over="ignore"):
        np.testing.assert_allclose(call("t_exp", x), np.exp(x), rtol=4e-16)


@pytest.mark.parametrize("p", [-4., -1.45, 0.4, 0.93, 1.1, 2.8, 3.6])
def test_pow(call, p):
    mp.dps = 40
    rng = np.random.default_rng(2)
    x = np.concatenate([np.exp(rng.uniform(-40., 40., 600)), rng.uniform(0.99, 1.01, 100), [1.]])
    want = [mp.mpf(float(v)) ** mp.mpf(p) for v in x]
    assert worst(call("t_pow", x, np.full_like(x, p)), want) <= 2. ** -52 + abs(p) * 2. ** -55


@pytest.mark.parametrize("name,base", [("t_log", None), ("t_log2", 2)])
def test_log(call, name, base):
    """Absolute error 2^-56 (the fixed-point unit) plus the result's rounding."""
    mp.dps = 40
    x = np.concatenate([np.exp(np.random.default_rng(5).uniform(-80., 80., 500)),
                        np.linspace(0.98, 1.02, 101), [1e-300, 1e300]])
    for g, v in zip(call(name, x), x):
        want = mp.log(mp.mpf(float(v))) / (mp.log(base) if base else 1)
        assert abs(mp.mpf(float(g)) - want) <= 2. ** -56 + 3. * 2. ** -53 * abs(want)


def test_pow_outside_the_fixed_point_range(call):
    x = np.array([0., 1e-300, 5e-324, np.inf, 1e200, -2., np.nan, 2.])
    p = np.array([0.6, 0.6, 0.5, 1.5, 0.6, 2., 1., 1500.])
    with np.errstate(over="ignore"):
        np.testing.assert_allclose(call("t_pow", x, p), np.power(x, p), rtol=4e-16)


@pytest.mark.parametrize("name", ["t_fd", "t_phi"])
def test_fermi_integrals(call, name):
    mp.dps = 60
    rng = np.random.default_rng(3)
    edge = np.arange(-288, 289, 7) / 8.
    y = np.concatenate([rng.uniform(-36., 36., 150), rng.uniform(-2., 2., 80), edge,
                        np.nextafter(edge, -100.), [-36., 35.9999, 36., 36.1, 250., -37., -690.]])
    got = call(name, y, width=6)
    for k in range(6):
        want = [fermi(k, mp.mpf(float(v))) / (mp.factorial(k) if name == "t_phi" else 1)
                for v in y]
        assert worst(got[:, k], want) <= 2. ** -51, k


def test_fermi_integrals_of_non_finite_arguments(call):
    got = call("t_fd", np.array([np.nan, -np.inf, np.inf]), width=6)
    assert (got[0] == 0.).all() and (got[1] == 0.).all() and (got[2] == np.inf).all()


def test_quotient(call):
    rng = np.random.default_rng(4)
    a, b = np.exp(rng.uniform(-50., 50., (2, 2000)))
    assert np.abs(call("t_quot", a, b) / (a / b) - 1.).max() <= 2. ** -51


def test_division_outside_the_quotient_range(call):
    v = np.array([0., 1., 3e-320, 1e-130, 1e130, 1e-300, 1e300, np.inf, np.nan, -7.])
    a, b = (w.ravel() for w in np.meshgrid(v, v))
    with np.errstate(all="ignore"):
        want = a / b
    got = call("t_div", a, b)
    near = np.isfinite(want) & (np.abs(want) > 1e-290)
    assert np.abs(got[near] / want[near] - 1.).max() <= 2. ** -51
    np.testing.assert_array_equal(got[~near], want[~near])
