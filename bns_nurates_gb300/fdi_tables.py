"""Coefficient tables of the Fermi-Dirac integral family F_j, j = -9/2 ... 21/2.

F_j(x) = integral_0^inf t^j / (exp(t - x) + 1) dt for j > -1, without the
1 / Gamma(j + 1) normalisation (the convention of functions.hpp:442-4375),
continued to j < -1 by dF_{j+1}/dx = (j + 1) F_j; for every j,
F_j(x) = -Gamma(j + 1) Li_{j+1}(-e^x).

The integer orders 0..5 are evaluated by the library's fixed-point Taylor
tables (fx_tables.py).  Every other member of the family the reference defines
(FDI_m92 .. FDI_m12, FDI_p12 .. FDI_p212 and FDI_p6 .. FDI_p10) is a factor
times one polynomial of degree 15, f * sum_m c_m v^m, whose row of coefficients
depends on the interval of x:

  x < -4        : f = e^x, v = -e^x, c_m = Gamma(j+1) (m+1)^{-(j+1)} (the
                  alternating series in e^x)
  -4 <= x < 100 : f = 1, v in [-1, 1] the position in one of 70 intervals,
                  of width 11/16 below 40 and 10 above
                  (the only singularities of F_j are at x = +-i pi, +-3i pi, ...,
                  so a Chebyshev expansion falls by >= 18 per degree)
  x >= 100      : f = x^{j+1} / (j+1), v = x^{-2} (the Sommerfeld expansion),
                  c_0 = 1, c_k = 2 eta(2k) (j+1) j ... (j+2-2k); the truncation and
                  the exponentially small remainder are below 1e-20 of the
                  leading term

One degree for every interval keeps the threads of a warp, whose arguments lie
in any of them, in one instruction stream.

``generate()`` computes the coefficients with mpmath at 34 digits and writes
csrc/bnsn_fdi_tab.h (checked in; mpmath is only needed to regenerate it).
``load_header()`` and ``evaluate()`` are the same evaluation in numpy (FP64),
used by the CPU tests to check the tables without a GPU.

Regenerate with:  python bns_nurates_gb300/fdi_tables.py
"""

import os
import re

import numpy as np

HERE = os.path.dirname(os.path.abspath(__file__))
HEADER = os.path.join(HERE, "csrc", "bnsn_fdi_tab.h")

# Twice the order of each table slot: the half-integers -9/2 .. 21/2 and the
# integers 6 .. 10 (0 .. 5 have the Taylor tables of fx_tables.py).
ORDERS2 = (-9, -7, -5, -3, -1, 1, 3, 5, 7, 9, 11, 12, 13, 14, 15, 16, 17, 18, 19, 20, 21)
# Every twice-order of the family (functions.hpp:442-4375).
FAMILY2 = (-9, -7, -5, -3, -1) + tuple(range(0, 22))

DEGREE = 15
X_LO, X_MID, X_HI = -4.0, 40.0, 100.0
WIDTH, WIDE = 0.6875, 10.0  # no interval ends within 0.1 of a zero of F_j
NARROW = int((X_MID - X_LO) / WIDTH)
PIECES = NARROW + int((X_HI - X_MID) / WIDE)
ROWS = PIECES + 2  # the series, the intervals, the Sommerfeld expansion
CHEB_NODES = 32
DPS = 34


def _mp():
    import mpmath

    mpmath.mp.dps = DPS
    return mpmath


def f_mp(j, x):
    """F_j(x) in mpmath (the unnormalised convention): the alternating series
    in e^x for x < -1 (mpmath's polylog loses the tiny values of order 1 to
    its log(1 - z) form), the Sommerfeld series for x > 200 (its remainder is
    of order e^-x) and -Gamma(j+1) Li_{j+1}(-e^x) in between."""
    mp = _mp()
    j = mp.mpf(j)
    x = mp.mpf(x)
    if x < -1:
        e, s, n = mp.exp(x), mp.mpf(0), 1
        while True:
            t = mp.power(e, n) * mp.power(n, -(j + 1))
            s += t if n % 2 else -t
            if abs(t) < abs(s) * mp.mpf(10) ** (-DPS - 2):
                break
            n += 1
        return mp.gamma(j + 1) * s
    if x > 200:
        u, s, fall = 1 / (x * x), mp.mpf(1), mp.mpf(1)
        for k in range(1, 60):
            fall *= (j + 1 - (2 * k - 2)) * (j + 1 - (2 * k - 1))
            t = 2 * mp.altzeta(2 * k) * fall * mp.power(u, k)
            s += t
            if abs(t) < mp.mpf(10) ** (-DPS - 2):
                break
        return mp.power(x, j + 1) / (j + 1) * s
    return mp.re(-mp.gamma(j + 1) * mp.polylog(j + 1, -mp.exp(x)))


def _series(j):
    mp = _mp()
    g = mp.gamma(mp.mpf(j) + 1)
    return [float(g * mp.power(n, -(mp.mpf(j) + 1))) for n in range(1, DEGREE + 2)]


def _piece_row(args):
    """Monomial coefficients in v of the Chebyshev expansion of degree DEGREE."""
    j, i = args
    mp = _mp()
    centre, half = (mp.mpf(c) for c in piece(i))
    th = [mp.pi * (k + mp.mpf(0.5)) / CHEB_NODES for k in range(CHEB_NODES)]
    fv = [f_mp(j, centre + half * mp.cos(t)) for t in th]
    out = [mp.mpf(0)] * (DEGREE + 1)
    t0, t1 = [mp.mpf(1)], [mp.mpf(0), mp.mpf(1)]  # T_0, T_1 in powers of v
    for m in range(DEGREE + 1):
        c = 2 * mp.fsum(fv[k] * mp.cos(m * th[k]) for k in range(CHEB_NODES)) / CHEB_NODES
        for k, a in enumerate(t0):
            out[k] += a * (c / 2 if m == 0 else c)
        t2 = [mp.mpf(0)] + [2 * a for a in t1]
        for k, a in enumerate(t0):
            t2[k] -= a
        t0, t1 = t1, t2
    return j, i, [float(c) for c in out]


def piece(i):
    """Centre and half-width of interval i."""
    if i < NARROW:
        return X_LO + WIDTH * i + WIDTH / 2, WIDTH / 2
    return X_MID + WIDE * (i - NARROW) + WIDE / 2, WIDE / 2


def _asym(j):
    """1 and 2 eta(2k) (j+1) j ... (j+2-2k), k = 1..DEGREE (eta: Dirichlet eta)."""
    mp = _mp()
    j1 = mp.mpf(j) + 1
    out, fall = [1.0], mp.mpf(1)
    for k in range(1, DEGREE + 1):
        fall *= (j1 - (2 * k - 2)) * (j1 - (2 * k - 1))
        out.append(float(2 * mp.altzeta(2 * k) * fall))
    return out


def _hex_rows(rows, indent):
    return (",\n" + indent).join("{" + ", ".join(float(v).hex() for v in r) + "}" for r in rows)


def generate(path=HEADER, workers=None):
    import multiprocessing as mproc

    mp = _mp()
    jobs = [(k2 / 2, i) for k2 in ORDERS2 for i in range(PIECES)]
    ctx = mproc.get_context("spawn")
    with ctx.Pool(workers or os.cpu_count()) as pool:
        res = pool.map(_piece_row, jobs, chunksize=4)
    rows = {(j, i): c for j, i, c in res}
    lines = [
        "// Generated by bns_nurates_gb300/fdi_tables.py (mpmath %s, %d digits); do not edit."
        % (mp.__version__, DPS),
        "// Tables of the Fermi-Dirac integral family evaluated by fdi.cu: polynomials",
        "// of the alternating series (x < -4), of the intervals of [-4, 100) and of",
        "// the Sommerfeld expansion (x >= 100).",
        "#pragma once",
        "",
        "namespace bnsn {",
        "namespace fdit {",
        "",
        "constexpr int kNumOrders   = %d;" % len(ORDERS2),
        "constexpr int kDegree      = %d;" % DEGREE,
        "constexpr int kPieces      = %d;" % PIECES,
        "constexpr int kNarrow      = %d;" % NARROW,
        "constexpr int kRows        = kPieces + 2;",
        "constexpr double kXlo = %r, kXmid = %r, kXhi = %r;" % (X_LO, X_MID, X_HI),
        "constexpr double kWidth = %r, kWide = %r;" % (WIDTH, WIDE),
        "",
        "// twice the order of each slot",
        "constexpr int kTwice[kNumOrders] = {%s};" % ", ".join(str(k) for k in ORDERS2),
        "",
        "// c_0 .. c_15 of the series (row 0), the intervals (rows 1 .. kPieces) and",
        "// the Sommerfeld expansion (row kPieces + 1)",
        "__device__ const double kPoly[kNumOrders][kRows][kDegree + 1] = {",
    ]
    for n, k2 in enumerate(ORDERS2):
        j = k2 / 2
        r = [_series(j)] + [rows[(j, i)] for i in range(PIECES)] + [_asym(j)]
        lines.append("    {" + _hex_rows(r, "     ") + "}" + ("," if n + 1 < len(ORDERS2) else ""))
    lines += [
        "};",
        "",
        "} // namespace fdit",
        "} // namespace bnsn",
        "",
    ]
    with open(path, "w") as f:
        f.write("\n".join(lines))


def load_header(path=HEADER):
    """The table of csrc/bnsn_fdi_tab.h as a numpy array (exact, hex literals)."""
    with open(path) as f:
        text = f.read()

    def block(name):
        m = re.search(r"%s\[[^=]*=\s*\{(.*?)\};" % name, text, re.S)
        vals = re.findall(r"-?0x[0-9a-fA-Fp.+-]+|-?inf|nan", m.group(1))
        return np.array([float.fromhex(v) for v in vals])

    n = len(ORDERS2)
    return block("kPoly").reshape(n, ROWS, DEGREE + 1)


def pow_half(x, h):
    """x^(h/2): an integer power by repeated squaring, times sqrt(x) for odd h,
    inverted for negative h."""
    a = abs(h)
    q = a >> 1
    v = np.ones_like(x)
    b = x.copy()
    while q:
        if q & 1:
            v = v * b
        q >>= 1
        if q:
            b = b * b
    if a & 1:
        v = v * np.sqrt(x)
    return 1.0 / v if h < 0 else v


def evaluate(k2, x, tabs):
    """F_{k2/2}(x) for a table order, in FP64 from the kernel's tables.  The kernel finds
    the interval and the position in it in fixed point (fd_interval of bnsn_fx.cuh)
    and takes its exponentials and powers from there; here they are numpy's."""
    slot = ORDERS2.index(k2)
    x = np.asarray(x, dtype=np.float64)
    j1 = 0.5 * k2 + 1.0
    nan = np.isnan(x)
    lo = x < X_LO
    hi = x >= X_HI
    row = np.where(lo, 0, PIECES + 1)
    v = np.zeros_like(x)
    f = np.ones_like(x)
    with np.errstate(over="ignore", invalid="ignore", divide="ignore", under="ignore"):
        e = np.exp(x[lo])
        v[lo], f[lo] = -e, e
        v[hi], f[hi] = 1.0 / (x[hi] * x[hi]), pow_half(x[hi], k2 + 2) / j1
        mid = ~(lo | hi | nan)
        xm = x[mid]
        i = np.where(xm < X_MID, np.floor((xm - X_LO) * (1.0 / WIDTH)),
                     NARROW + np.floor((xm - X_MID) * (1.0 / WIDE)))
        i = np.clip(i.astype(np.int64), 0, PIECES - 1)
        narrow = i < NARROW
        cen = np.where(narrow, X_LO + WIDTH * i + WIDTH / 2,
                       X_MID + WIDE * (i - NARROW) + WIDE / 2)
        v[mid] = (xm - cen) * np.where(narrow, 2.0 / WIDTH, 2.0 / WIDE)
        row[mid] = i + 1
        c = tabs[slot][row]
        p = c[..., DEGREE]
        for m in range(DEGREE - 1, -1, -1):
            p = p * v + c[..., m]
        out = f * p
    out[nan] = 0.0 if k2 % 2 == 0 else np.nan
    return out


if __name__ == "__main__":
    generate()
    print("wrote", HEADER)
