"""Generates csrc/bnsn_fx_tab.h: the tables of the fixed-point functions.

``python -m bns_nurates_gb300.fx_tables`` writes the header (needs mpmath).

kFdRows: the normalised Fermi-Dirac integrals phi_m = F_m / m! and their
derivatives (d phi_m / dx = phi_{m-1}, down to m = -10) at x = i / 8,
i = -288 .. 287, as integers round(phi_m 2^(s + (5 - m) d)) with the scale s
and the step d of the row chosen so that the largest entry stays below 2^62
and phi_0 .. phi_5 keep as many bits as possible.  kExp2: 2^(j/128) in units
of 2^-63.  kLog: per 7-bit interval of [1, 2) the 12-bit reciprocal c_j of its
centre and -log2(c_j / 2^11) in units of 2^-63.
"""

import os

HERE = os.path.dirname(os.path.abspath(__file__))
LIMIT = 288  # rows x = i / 8, i in [-LIMIT, LIMIT)
TOP, BOTTOM = 5, -10
WIDE = 11    # entries m = 5 .. -5 in 64 bits, the rest in 32


def fd_derivatives(mp, x):
    """phi_5 .. phi_-10 at x (mpmath)."""
    out = {}
    a = abs(x)
    z = [mp.mpf(1)] + [(1 - mp.mpf(2) ** (1 - 2 * n)) * mp.zeta(2 * n) for n in range(1, 4)]
    for m in range(0, TOP + 1):
        # phi_m(-a), and phi_m(a) = (-1)^m phi_m(-a) + 2 sum_n eta(2n) a^(m+1-2n) / (m+1-2n)!
        # (eta(0) = 1/2) above zero
        low = mp.log1p(mp.exp(-a)) if m == 0 else -mp.re(mp.polylog(m + 1, -mp.exp(-a)))
        if x > 0:
            low = (-1) ** m * low + sum(
                (1 if n == 0 else 2) * z[n] * a ** (m + 1 - 2 * n) / mp.factorial(m + 1 - 2 * n)
                for n in range(0, 4) if m + 1 - 2 * n >= 0)
        out[m] = low
    # derivatives of the logistic f as polynomials in f: P -> P' f (1 - f)
    f = 1 / (1 + mp.exp(-x))
    poly = [0, 1]
    for m in range(-1, BOTTOM - 1, -1):
        out[m] = sum(c * f ** k for k, c in enumerate(poly))
        d = [k * c for k, c in enumerate(poly)][1:]
        new = [0] * (len(d) + 2)
        for k, c in enumerate(d):
            new[k + 1] += c
            new[k + 2] -= c
        poly = new
    return out


def row(mp, x):
    phi = fd_derivatives(mp, x)
    best = None
    for d in range(0, 8):
        top = max(abs(phi[m]) * 2 ** ((TOP - m) * d) for m in phi)
        s = 62 - int(mp.ceil(mp.log(top, 2)))
        bits = min(mp.log(phi[m] * mp.mpf(2) ** (s + (TOP - m) * d), 2) for m in range(0, 6))
        if best is None or bits > best[0]:
            best = (bits, s, d)
    bits, s, d = best
    c = [int(mp.nint(phi[m] * mp.mpf(2) ** (s + (TOP - m) * d)))
         for m in range(TOP, BOTTOM - 1, -1)]
    assert max(abs(v) for v in c) <= 2 ** 62 and bits > 56.9, (x, bits, s, d)
    wide, rest = c[:WIDE], [(v + 2 ** 31) >> 32 for v in c[WIDE:]]
    return wide, rest, s, d


def main():
    from mpmath import mp
    mp.dps = 60
    L = ["// Tables of the fixed-point functions of bnsn_fx.cuh, written by fx_tables.py",
         "// (mpmath).  kFdRows: normalised Fermi-Dirac integrals phi_5 .. phi_-5 (64 bits) and",
         "// phi_-6 .. phi_-10 (32 bits) at x = i / 8, i = -288 .. 287, scaled by 2^(s + (5 - m) d);",
         "// meta = s << 8 | d.  kExp2: 2^(j/128) in 2^-63.  kLog: 12-bit reciprocals c_j of the",
         "// centres of 128 intervals of [1, 2) and -log2(c_j / 2^11) in 2^-63.",
         "#pragma once", "", "#include <stdint.h>", "", "namespace bnsn {", "namespace fx {", "",
         "constexpr int kFdLimit = %d;" % LIMIT, "",
         "struct alignas(16) FdRow", "{", "    int64_t c[%d];" % WIDE,
         "    int32_t t[%d];" % (TOP - BOTTOM + 1 - WIDE), "    int32_t meta;", "};", "",
         "struct alignas(16) LogRow", "{", "    uint64_t l;", "    uint64_t c;", "};", "",
         "BNSN_FX_TABLE FdRow kFdRows[%d] = {" % (2 * LIMIT)]
    for i in range(-LIMIT, LIMIT):
        wide, rest, s, d = row(mp, mp.mpf(i) / 8)
        L.append("{{%s}, {%s}, %d}," % (", ".join("%dLL" % v for v in wide),
                                       ", ".join(str(v) for v in rest), s << 8 | d))
    L += ["};", "", "BNSN_FX_TABLE uint64_t kExp2[128] = {"]
    v = [int(mp.nint(mp.mpf(2) ** (mp.mpf(j) / 128 + 63))) for j in range(128)]
    L += ["".join("%dull, " % u for u in v[k:k + 4]).rstrip() for k in range(0, 128, 4)]
    L += ["};", "", "BNSN_FX_TABLE LogRow kLog[128] = {"]
    for j in range(128):
        c = int(mp.nint(2048 / (1 + (mp.mpf(j) + mp.mpf(1) / 2) / 128)))
        L.append("{%dull, %dull}," % (int(mp.nint(-mp.log(mp.mpf(c) / 2048, 2) * mp.mpf(2) ** 63)), c))
    L += ["};", "", "} // namespace fx", "} // namespace bnsn", ""]
    with open(os.path.join(HERE, "csrc", "bnsn_fx_tab.h"), "w") as f:
        f.write("\n".join(L))


if __name__ == "__main__":
    main()
