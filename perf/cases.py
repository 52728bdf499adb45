"""Workloads of the opacity library and their values in plain 64-bit torch.

``listed()`` are the calls a radiation-hydrodynamics code makes: single points
through the per-point drop-in, small and ragged batches, whole patches and
slabs in both precisions, AMR blocks, host-buffer batches, spectral opacities,
and the auxiliary Fermi-integral, distribution and equilibrium calls.
``draw(rng)`` gives more of the same ranges.  ``run(state)`` is one call (or
the few calls of one step) through the public entry points.  ``exact(case,
seed)`` evaluates the same integrals in 64 bits from the formulas of the
reference, with Fermi integrals from an accelerated alternating series.
"""

import math

import numpy as np
import torch

import bns_nurates_gb300 as bn

FIELDS = ("eta_0", "kappa_0_a", "eta", "kappa_a", "kappa_s")
SPECTRAL = ("j", "kappa", "j_s", "kappa_s")
DISTR = ("w_t", "temp_t", "eta_t", "w_f", "temp_f", "c_f", "beta_f")
EOS = ("nb", "temp", "ye", "yp", "yn", "mu_p", "mu_n", "mu_e", "mu_mu", "dU", "dm_eff")
HR98, BRT06, GP19 = 0, 1, 2


# ---------------------------------------------------------------------------
# cases
# ---------------------------------------------------------------------------

def _grey(name, call, n, nquad, brem, precision, abs_em=1, pair=1, use_brem=1, nes=1, iso=1,
          stim=1):
    case = dict(call=call, n=n, nquad=nquad, brem=brem, precision=precision, abs_em=abs_em,
                pair=pair, use_brem=use_brem, nes=nes, iso=iso, stim=stim)
    return dict(case, name=name) if name else case


def _spectral(name, n, energies, nquad, brem, precision, nes, stim=1):
    case = dict(call="spectral", n=n, energies=energies, nquad=nquad, brem=brem,
                precision=precision, abs_em=1, pair=1, use_brem=1, nes=nes, iso=1, stim=stim)
    return dict(case, name=name) if name else case


def listed():
    return [
        # host code that has not been batched yet: ComputeM1Opacities once per
        # cell, a host struct in and a host struct out
        _grey("point_fp64", "point", 1, 10, HR98, "fp64"),
        # the smallest batch: a boundary strip, or the zones a solver revisits
        _grey("batch_256_fp64", "batch", 256, 10, HR98, "fp64"),
        # leftover zones in the fast precision, the third brem variant, no
        # stimulated absorption, a coarse quadrature (GaussLegendre(6))
        _grey("batch_1001_mixed", "batch", 1001, 6, BRT06, "mixed", stim=0),
        # the usual patch call in the default precision: no inelastic
        # scattering, the reference's largest quadrature
        _grey("patch_fp64", "batch", 100003, 10, HR98, "fp64", nes=0),
        # all reactions with the finest quadrature in the default precision
        _grey("slab_fp64", "batch", 20011, 20, GP19, "fp64"),
        # the same in mixed precision at slab size (a 256 x 256 x 4 slab)
        _grey("slab_mixed", "batch", 262144, 20, GP19, "mixed"),
        # a host code that keeps its grid in host memory
        _grey("host_mixed", "host", 300001, 10, HR98, "mixed", nes=0),
        # AMR blocks of uneven size with their own reactions and quadrature
        dict(name="blocks_mixed", call="blocks", blocks=96, precision="mixed"),
        # spectral opacities of a patch at the configurations' 24 energies
        _spectral("spectral_fp64", 8191, 24, 10, HR98, "fp64", 0),
        # and with every reaction and the finest quadrature
        _spectral("spectral_mixed", 16384, 24, 20, GP19, "mixed", 1),
        # electron densities and pressures from half-integer Fermi integrals
        dict(name="fdi_half", call="fdi", twice_order=1, n=4000037),
        # equilibrium distributions and the M1 reconstruction of a large grid
        dict(name="equilibrium", call="equilibrium", n=1000003),
    ]


def _cost(case):
    """Rough work of a case in reference operations."""
    if case["call"] == "blocks":
        return sum(b["count"] * _ops_per_point(b) for b in _block_list(case, 0))
    if case["call"] == "fdi":
        return 60. * case["n"]
    if case["call"] == "equilibrium":
        return 1500. * case["n"]
    per = _ops_per_point(case)
    return case["n"] * per


def _ops_per_point(c):
    """Operations of the reference algorithm per point: the counts of its
    instrumented build (profiles/op_counts.json) over nodes or node pairs."""
    q = c["nquad"]
    brem = {HR98: 1670., BRT06: 300., GP19: 632.}[c["brem"]]
    if c["call"] == "spectral":
        pairs = 2. * q * c["energies"]  # one integral over 2n nodes per energy
        return pairs * (1700. * c["pair"] + 1.6 * brem * c["use_brem"] + 3300. * c["nes"]) + \
            900. * c["energies"]
    return 2700. * q + q * q * (2130. * c["pair"] + brem * c["use_brem"] + 5250. * c["nes"])


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    largest = _cost(listed()[5])
    kind = rng.choice(["batch", "batch", "batch", "batch", "host", "boxes", "blocks", "spectral",
                       "spectral", "fdi", "equilibrium", "point"])
    precision = rng.choice(["fp64", "mixed"])
    brem = rng.choice([HR98, BRT06, GP19])
    nquad = rng.randint(4, 20)
    if kind == "fdi":
        return dict(call="fdi", twice_order=rng.choice([0, 1, 3, 4, 5, 7, 10, 11, 12, 15, 21]),
                    n=size(1000, 8000000))
    if kind == "equilibrium":
        return dict(call="equilibrium", n=size(1000, 2000000))
    if kind == "blocks":
        return dict(call="blocks", blocks=rng.randint(3, 90 if precision == "mixed" else 24),
                    precision=precision)
    if kind == "spectral":
        ne = rng.randint(1, 40)
        case = _spectral(None, 1, ne, nquad, brem, precision, rng.randint(0, 1),
                         rng.randint(0, 1))
        top = largest / _cost(case) / (6. if precision == "fp64" else 4.)
        return dict(case, n=size(16, max(64., min(65536., top))))
    case = _grey(None, kind, 1, nquad, brem, "fp64" if kind == "point" else precision,
                 abs_em=int(rng.random() < 0.9), pair=int(rng.random() < 0.9),
                 use_brem=int(rng.random() < 0.9), nes=int(rng.random() < 0.6),
                 iso=int(rng.random() < 0.9), stim=int(rng.random() < 0.7))
    if kind == "point":
        return case
    top = largest / _cost(case) / (6. if precision == "fp64" else 1.5)
    return dict(case, n=size(64, min(300000., top)))


def work(case):
    """Each input read once, each output written once, and the reference
    algorithm's operations."""
    call = case["call"]
    if call == "fdi":
        return {"bytes": 16 * case["n"], "flops": _cost(case)}
    if call == "equilibrium":
        # T, mu_p, mu_n, mu_e in; 28 + 12 out; the 12 moments in again; 28 out
        return {"bytes": 8 * case["n"] * (4 + 28 + 12 + 12 + 28), "flops": _cost(case)}
    if call == "blocks":
        n = sum(b["count"] for b in _block_list(case, 0))
        return {"bytes": n * 8 * (22 + 20), "flops": _cost(case)}
    if call == "spectral":
        return {"bytes": case["n"] * 8 * (22 + 16 * case["energies"]), "flops": _cost(case)}
    if call == "point":
        return {"bytes": 8 * (22 + 28 + 20), "flops": _cost(case)}
    return {"bytes": case["n"] * 8 * (22 + 20), "flops": _cost(case)}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------

def _points(n, seed):
    """Matter and radiation states over the densities, temperatures and
    electron fractions of a merger: (eos [11, n], m1 [12, n]) host arrays."""
    return bn.synthetic_points((seed * 0x9E3779B1 + 12345) & 0xffffffff, n)


def _block_list(case, seed):
    """Blocks as bench.py's AMR workload draws them, with fewer cells: the
    largest block has 24^3.  The layout does not depend on the seed (a grid
    hierarchy outlives many time steps)."""
    rng = np.random.default_rng(20261203 + case["blocks"])
    blocks, first = [], 0
    for _ in range(case["blocks"]):
        count = int(rng.choice((8, 12, 16, 24), p=(0.55, 0.28, 0.12, 0.05))) ** 3
        blocks.append(dict(call="blocks", first=first, count=count, brem=int(rng.integers(0, 3)),
                           nes=int(rng.integers(0, 2)), nquad=int(rng.choice((10, 20))),
                           abs_em=1, pair=1, use_brem=1, iso=1, stim=1))
        first += count
    return blocks


def _boxes(case):
    """Interior extent of one grid box with case["n"] cells and 3 ghost zones."""
    edge = max(1, int(round(case["n"] ** (1. / 3.))))
    return (edge, edge + 1, max(1, case["n"] // (edge * (edge + 1))))


def _flags(c):
    return bn.opacity_flags(c["abs_em"], c["pair"], c["use_brem"], c["nes"], c["iso"])


def _params(c):
    return bn.opacity_params(brem_implementation=c["brem"])


def _fdi_arguments(case, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed + 17)
    # degeneracies from the dilute gas to neutron-star matter
    return torch.rand(case["n"], generator=g, device="cuda", dtype=torch.float64) * 200. - 50.


def _energies(c):
    return np.logspace(0., math.log10(300.), c["energies"])


def prepare(case, seed):
    call = case["call"]
    if call == "fdi":
        x = _fdi_arguments(case, seed)
        return dict(case=case, x=x, out=torch.empty_like(x))
    if call == "blocks":
        blocks = _block_list(case, seed)
        n = blocks[-1]["first"] + blocks[-1]["count"]
    elif call == "boxes":
        nx, ny, nz = _boxes(case)
        n = nx * ny * nz
    else:
        n = case["n"]
    eos_h, m1_h = _points(n, seed)
    if call == "equilibrium":
        return dict(case=case, eos=torch.from_numpy(eos_h).cuda())
    if call == "blocks" or case["brem"] == GP19:
        from bns_nurates_gb300 import gp19_synthetic
        bn.set_gp19_table(gp19_synthetic.table())
    if call == "host":
        return dict(case=case, eos=torch.from_numpy(eos_h).pin_memory(),
                    m1=torch.from_numpy(m1_h).pin_memory(),
                    out=torch.empty((20, n), dtype=torch.float64).pin_memory(),
                    flags=_flags(case), params=_params(case),
                    quad=bn.gauss_legendre(case["nquad"]))
    eos, m1 = torch.from_numpy(eos_h).cuda(), torch.from_numpy(m1_h).cuda()
    if call == "point":
        gp = bn.GreyOpacityParams()
        for k, name in enumerate(EOS):
            setattr(gp.eos_pars, name, float(eos_h[k, 0]))
        d = bn.distr_from_m1(m1).cpu().numpy()
        for s in range(4):
            gp.m1_pars.n[s], gp.m1_pars.J[s] = m1_h[s, 0], m1_h[4 + s, 0]
            gp.m1_pars.chi[s] = m1_h[8 + s, 0]
            for q, name in enumerate(DISTR):
                getattr(gp.distr_pars, name)[s] = d[4 * q + s, 0]
        gp.opacity_flags, gp.opacity_pars = _flags(case), _params(case)
        return dict(case=case, gp=gp, quad=bn.gauss_legendre(case["nquad"]))
    if call == "blocks":
        out = torch.empty((20, n), dtype=torch.float64, device="cuda")
        plan = bn.BlocksPlan([(b["first"], b["count"], (b["abs_em"], b["pair"], b["use_brem"],
                                                        b["nes"], b["iso"]), b["brem"], b["nquad"])
                              for b in blocks], eos, m1, out, precision=case["precision"])
        return dict(case=case, plan=plan, eos=eos, m1=m1, out=out)
    state = dict(case=case, eos=eos, m1=m1, flags=_flags(case), params=_params(case),
                 quad=bn.gauss_legendre(case["nquad"]))
    if call == "boxes":
        g = 3  # ghost zones
        box = {}
        for name, src in (("eos", eos), ("m1", m1)):
            t = torch.zeros((src.shape[0], nz + 2 * g, ny + 2 * g, nx + 2 * g),
                            dtype=torch.float64, device="cuda")
            t[:, g:g + nz, g:g + ny, g:g + nx] = src.reshape(-1, nz, ny, nx)
            box[name] = t
        box["out"] = torch.zeros((20,) + tuple(box["eos"].shape[1:]), dtype=torch.float64,
                                 device="cuda")
        box["lo"], box["hi"] = (g, g, g), (g + nx, g + ny, g + nz)
        return dict(state, box=box)
    if call == "spectral":
        out = torch.empty((16, n, case["energies"]), dtype=torch.float64, device="cuda")
        return dict(state, energies=_energies(case), out=out)
    return dict(state, out=torch.empty((20, n), dtype=torch.float64, device="cuda"))


def run(state):
    case = state["case"]
    call = case["call"]
    if call == "point":
        f = bn.ComputeM1Opacities if case["stim"] else bn.ComputeM1OpacitiesNotStimulated
        return f(state["quad"], state["quad"], state["gp"])
    if call == "fdi":
        return {"F": bn.fdi(case["twice_order"] / 2., state["x"], out=state["out"])}
    if call == "equilibrium":
        distr, m1 = bn.nu_equilibrium(state["eos"])
        back = bn.distr_from_m1(m1)
        return {"distr": distr, "n": m1[0:4], "J": m1[4:8], "chi": m1[8:12],
                "eta_t": back[8:12], "temp_t": back[4:8], "temp_f": back[16:20],
                "weights": torch.stack([back[0:4], back[12:16], back[20:24]]),
                "beta_f": back[24:28]}
    if call == "blocks":
        return _fields(state["plan"].run(state["eos"], state["m1"], state["out"]))
    if call == "host":
        bn.m1_opacities_host(state["eos"], state["m1"], state["flags"], state["params"],
                             state["quad"], stim_abs=case["stim"], precision=case["precision"],
                             out=state["out"])
        return _fields(state["out"])
    if call == "boxes":
        bn.m1_opacities_grid_boxes([state["box"]], state["flags"], state["params"],
                                   state["quad"], stim_abs=case["stim"],
                                   precision=case["precision"])
        return _fields(state["box"]["out"])
    if call == "spectral":
        out = bn.spectral_opacities(state["eos"], state["m1"], state["flags"], state["params"],
                                    state["quad"], state["energies"], stimulated=case["stim"],
                                    precision=case["precision"], out=state["out"])
        return {name: out[4 * k:4 * k + 4] for k, name in enumerate(SPECTRAL)}
    return _fields(bn.m1_opacities(state["eos"], state["m1"], state["flags"], state["params"],
                                   state["quad"], stim_abs=case["stim"],
                                   precision=case["precision"], out=state["out"]))


def _fields(out):
    return {name: out[4 * k:4 * k + 4] for k, name in enumerate(FIELDS)}


# ---------------------------------------------------------------------------
# the same in 64 bits, in torch
# ---------------------------------------------------------------------------

MEV = 1.6021766341182763e+8
ME, MN, MP, DELTA = 0.51099895069, 939.56542194, 938.27208943, 1.29333251
MB = 1.6737747126723517e-24
H, CLIGHT, GF0 = 4.135667696e-21, 2.99792458e+17, 1.1663787e-11
HBAR = 0.5 * H / math.pi
GF = GF0 * (HBAR * CLIGHT) ** 3
GA, SW2 = 1.23, 0.2325
FPHC3 = 4. * math.pi / (H * CLIGHT) ** 3
BETA = CLIGHT ** 3 * (GF0 * HBAR) ** 2 * (1. + 3. * GA ** 2) / math.pi
ISO = 2. * math.pi * GF ** 2 / HBAR / (H * CLIGHT) ** 3
BREM = 0.63 ** 2 * GF ** 2 / HBAR
NEPS = 2. * GF0 ** 2 * CLIGHT * (HBAR * CLIGHT) ** 2 / (3. * math.pi)
T2D = 0.5 * 4.364


def _alternating_weights(n=26):
    """Weights of Cohen, Rodriguez Villegas and Zagier's acceleration of
    alternating series (algorithm 1): sum (-1)^k a_k ~ sum w_k a_k."""
    d = (3. + math.sqrt(8.)) ** n
    d = (d + 1. / d) / 2.
    b, c, w = -1., -d, []
    for k in range(n):
        c = b - c
        w.append(c / d)
        b *= (k + n) * (k - n) / ((k + 0.5) * (k + 1.))
    return w


WEIGHTS = _alternating_weights()


def _fermi(y, lo, hi):
    """Complete Fermi integrals F_lo .. F_hi (integer orders) of y."""
    z = torch.exp(-y.abs())
    out = [torch.zeros_like(y) for _ in range(lo, hi + 1)]
    p = torch.ones_like(y)
    for m, w in enumerate(WEIGHTS):
        p = p * z
        for k in range(lo, hi + 1):
            out[k - lo].add_(p, alpha=w * math.factorial(k) / float(m + 1) ** (k + 1))
    pos = y > 0.
    y2 = y * y
    a2, a4, a6 = math.pi ** 2 / 6., 7. * math.pi ** 4 / 360., 31. * math.pi ** 6 / 15120.
    for k in range(lo, hi + 1):
        poly = (y, 0.5 * y2 + a2, y * (y2 / 3. + 2. * a2),
                6. * a4 + y2 * (3. * a2 + y2 / 4.),
                y * (24. * a4 + y2 * (4. * a2 + y2 / 5.)),
                120. * a6 + y2 * (60. * a4 + y2 * (5. * a2 + y2 / 6.)))[k]
        f = out[k - lo]
        out[k - lo] = torch.where(pos, poly + f if k % 2 == 0 else poly - f, f)
    return out


def _safe_exp(x):
    return torch.exp(x.clamp(-700., 700.))


def _occ(arg):
    """1 / (e^arg + 1)."""
    t = _safe_exp(-arg.abs())
    return torch.where(arg > 0., t, torch.ones_like(t)) / (1. + t)


def _poly(y, c):
    p = torch.full_like(y, c[0])
    for v in c[1:]:
        p = p * y + v
    return p


def _distribution(m1):
    """Thick (equilibrium) and thin parts of each species from n, J, chi:
    seven tensors [4, P]."""
    n, J, chi = m1[0:4].clamp(min=1e-100), m1[4:8].clamp(min=1e-100), m1[8:12]
    y = n * (n / J) ** 3 / FPHC3
    low = torch.log(_poly(y, [1., 0.19926987701997, 38865.0149220478, 14364.6331099737,
                              5750.1878570758, 1120.71610972194, 1.60356108438235e-8]) /
                    _poly(y, [1., 1., 38840.0743174942, -99.9009680656931, -171.874844843596,
                              75.7101579899442, 83.0160130941424]))
    mid = _poly(y, [41.3836568203438, 32.5515666786612, -157.774993512235, 66.5726772426253,
                    14.4883415579211, 0.315360380575709, 0.000660414331285249]) / \
        _poly(y, [1., 1.8888797407042, -5.35488690539183, 1.94673781342617, 0.483128792035557,
                  0.0113386564109086, 2.64160073447322e-5]) - 30.
    high = torch.exp(_poly(y, [3852.81416018959, -5316.18895799799, 1102.91561586553,
                               1.54082262710661e-6, 1732.89925128741, -1769.59868329086,
                               586.406885304906]) /
                     _poly(y, [1., 255.936658313629, 9.42360945627147e-5, -81.2467063138386,
                               -180.100197053091, -89.0343496217014, 143.849128123195]))
    eta = torch.where(y < 0.005, low,
                      torch.where(y <= 0.7, mid,
                                  torch.where(y < 0.7901234567745267, high,
                                              torch.full_like(y, 20.)))).clamp(max=20.)
    f2, f3 = _fermi(eta, 2, 3)
    Tf = J / (n * 3.6)
    g36 = math.sqrt(2. * math.pi / 3.6) * (3.6 / math.e) ** 3.6
    return dict(w_t=1.5 * (1. - chi), temp_t=f2 * J / (f3 * n), eta_t=eta,
                w_f=0.5 * (3. * chi - 1.), temp_f=Tf, c_f=torch.full_like(Tf, 0.6),
                beta_f=n / (FPHC3 * g36 * Tf ** 3.6))


def _g(d, s, nu):
    """Occupation of species s at energies nu [P, ...]."""
    v = [d[k][s].reshape((-1,) + (1,) * (nu.dim() - 1)) for k in DISTR]
    w_t, T_t, eta, w_f, T_f, c, b = v
    return w_t * _occ(nu / T_t - eta) + w_f * b * nu ** c * torch.exp(-nu / T_f)


def _form_factors(E, reac):
    e = E * (MEV / (MB * CLIGHT ** 2))
    tau = 0.5 * e * e / (1. + e)
    eta = 1. / (1. + 5.6 * tau)
    G = 1. / ((1. + 4.97 * tau) ** 2 * (1. + tau))
    lp, ln = 1.793, -1.913
    p1, p2 = (1. + tau * (1. + lp)) * G, lp * G
    n1, n2 = tau * ln * (5.6 * tau * eta) * G, ln * (1. + tau * eta) * G
    d = (1. + 3.53 * tau) ** 2
    cw = 0.5 - 2. * SW2
    if reac == 1:
        return e, cw * p1 - 0.5 * n1, 0.5 * GA / d, cw * p2 - 0.5 * n2
    if reac == 2:
        return e, cw * n1 - 0.5 * p1, -0.5 * GA / d, cw * n2 - 0.5 * p2
    return e, p1 - n1, GA / d, p2 - n2


def _beta(E, nu, anti):
    """(absorption, emission) of nu_e (anti = 0) or anti-nu_e at nu [P, K]."""
    e, cv, ca, F2 = _form_factors(nu, 3)
    t1 = cv ** 2 * (1. + 4. * e + 16. / 3. * e * e) + 3. * ca ** 2 * (1. + 4. / 3. * e) ** 2 + \
        8. / 3. * cv * F2 * e * e + 5. / 3. * e * e * (1. + 0.4 * e) * F2 ** 2
    t2 = 4. * (cv + F2) * ca * e * (1. + 4. / 3. * e)
    R = (t1 - t2 if anti else t1 + t2) / ((1. + 3. * GA ** 2) * (1. + 2. * e) ** 3)
    T, dU = E["temp"], E["dU"]
    nn, np_ = E["nb"] * E["yn"], E["nb"] * E["yp"]
    mu_hat = E["mu_n"] - E["mu_p"] - DELTA - dU

    def eta_nn(a, b, mu):
        v = (b - a) / (_safe_exp(-mu / T) - 1.)
        return torch.where((mu.abs() < 0.01) | (v < 0.), a, v)

    pref = eta_nn(nn, np_, mu_hat) if anti else eta_nn(np_, nn, -mu_hat)
    Q = DELTA + dU
    El = nu - Q if anti else nu + Q  # energy of the captured lepton
    sgn = -1. if anti else 1.
    root = torch.sqrt((1. - (ME / El) ** 2).clamp(min=0.)) * El * El
    cap = torch.where(El - ME >= 0., root * R, torch.zeros_like(R))
    dec = torch.where(-El - ME >= 0., root, torch.zeros_like(R))
    fl = _occ((El - sgn * E["mu_e"]) / T)
    fa = _occ((-El + sgn * E["mu_e"]) / T)
    em = BETA * pref * (cap * fl + dec * (1. - fa))
    mu = E["mu_p"] + E["mu_e"] - E["mu_n"]
    return em * _safe_exp((nu - (-mu if anti else mu)) / T), em


def _iso(E, nu, total):
    """Iso-energetic scattering kernel: l = 0 minus a third of l = 1, or l = 0."""
    out = 0.
    for reac, y in ((1, E["yp"]), (2, E["yn"])):
        n = y * E["nb"]
        eF = 4.785390000313652 * HBAR ** 2 / MB * MEV * n ** (2. / 3.)
        a = 1.5 * E["temp"] / eF
        eta = torch.where(n > 0., n * a / torch.sqrt(1. + a * a), torch.zeros_like(n))
        e, cv, ca, F2 = _form_factors(nu, reac)
        s = cv ** 2 + 3. * ca ** 2 + 1.5 * (e * F2) ** 2 + 2. * e * e * cv * F2
        if total:
            s = s - (cv ** 2 - ca ** 2 - 2. * (e * F2) ** 2 - 4. * e * e * cv * F2) / 3.
        out = out + eta * ISO * s
    return out


def _psi(eta, y, z):
    """Psi_0(y, z) of the pair kernel."""
    fam, fap = _fermi(eta - y, 1, 5), _fermi(eta + y, 1, 5)
    fbm, fbp = _fermi(eta - z, 1, 5), _fermi(eta + z, 1, 5)
    fm, fp = _fermi(eta - y - z, 3, 5), _fermi(eta + y + z, 3, 5)
    f3, f4 = _fermi(eta, 3, 4)
    c0, c1 = 20. * fam[3], 20. * fbp[3]
    c2, c3 = 120. * (fam[1] - fbp[1]), -40. * fam[2] + 40. * fbp[2]
    c5, c7 = 40. * fm[0] - 40. * f3, 20. * fm[1] - 20. * f4
    c8, c9 = -40. * fp[0] + 40. * f3, 20. * fp[1] - 20. * f4
    c10 = 4. * (-fam[4] + fm[2] - fbm[4] + fap[4] - fp[2] + fbp[4])
    p = c10 + y * (c1 - c0 + c7 + y * (c3 + c5 + z * (c2 + 120. * z * (fbp[0] - fam[0]))) +
                   z * (80. * (fam[2] - fbp[2]) - c2 * z)) + \
        z * (c0 - c1 + c9 + z * (c3 + c8))
    return torch.where(eta - y - z > 200., torch.zeros_like(p), p / (15. * (y * z) ** 2))


def _pair(E, nu, nub):
    """Pair emission and absorption kernels of the four species."""
    T = E["temp"]
    eta = E["mu_e"] / T
    y, z = torch.broadcast_tensors(nu / T, nub / T)
    p0, p1 = _psi(eta, y, z), _psi(eta, z, y)
    aux = 0.5 * 1.55e-12 / math.pi * T * T / (1. - _safe_exp(y + z))
    ex = _safe_exp(y + z)
    em = []
    for a in (1. + 2. * SW2, -1. + 2. * SW2):
        a1, a2 = a * a, (2. * SW2) ** 2
        em += [(a1 * p0 + a2 * p1) * aux, (a1 * p1 + a2 * p0) * aux]
    return em, [ex * v for v in em]


def _hr98(E, w):
    T, nb = E["temp"], E["nb"]
    x = w / T
    xs = x.clamp(min=1e-10)
    y = (19.4 / T).clamp(min=1e-10)
    snd = 2. * math.sqrt(math.pi) * (xs + 2. - _safe_exp(-y / 12.)) ** 1.5 * \
        (xs * xs + 2. * xs * y + 5. * y * y / 3. + 1.) / \
        (math.sqrt(math.pi) + (math.pi ** 0.125 + xs + y) ** 4)
    p = 0.67 + 0.18 * y ** 0.4
    total = 0.
    for weight, n_nuc, m in (
            (1., nb * E["yn"], MN * MEV / CLIGHT ** 2), (1., nb * E["yp"], MP * MEV / CLIGHT ** 2),
            (28. / 3., nb * torch.sqrt(E["yn"] * E["yp"]),
             MEV / CLIGHT ** 2 * 938.918532994116257276238085018813)):
        es = (3. * math.pi ** 2 * n_nuc) ** (2. / 3.) * 0.25 * H * H * MEV / math.pi ** 2 / \
            (2. * m * T)
        gamma = 1.63 * es ** 1.5 * T * 0.1
        e = es.clamp(min=1e-10)
        u = torch.sqrt(y / (2. * e)) + 1e-10
        ua = u * u / (2. * torch.sqrt(2. * u * u + 4.))
        fu = 1. - 5. * u * torch.atan(2. / u) / 6. + u * u / (3. * (u * u + 4.)) + \
            torch.atan(1. / ua) * ua / 3.
        fu = torch.where(fu.abs() < 1e-14, torch.full_like(fu, 1e-14), fu)
        sd = 3. * (math.pi / 2.) ** 2.5 * e ** -2.5 * (xs * xs + 4. * math.pi ** 2) * xs * fu / \
            (4. * math.pi ** 2 * -torch.expm1(-xs))
        F = 1. + 1. / ((3. + (xs - 1.2) ** 2 + xs ** -4.) * (1. + e * e) * (1. + y ** 4))
        G = 1. - 0.0044 * xs ** 1.1 * y / (0.8 + 0.06 * y ** 1.05) * torch.sqrt(e) / (e + 0.2)
        h = 0.1 * e / (2.39 + 0.1 * e ** 1.1)
        C = 1.1 * xs ** 1.1 * h / (2.3 + h * xs ** 0.93 + 0.0001 * xs ** 1.2) * 30. / \
            (30. + 0.005 * xs ** 2.8)
        s = (snd ** -p + sd ** -p) ** (-1. / p) * F * (1. + C * G)
        den = 25. * y * y + 1.
        a1 = (0.5 + 1. / e) / (1. + 1. / e) / den + (0.5 + e / 15.6) * 25. * y * y / den
        a2 = (0.63 + 0.04 * e ** 1.45) / (1. + 0.02 * e ** 2.5)
        a3 = 1.2 * _safe_exp(0.6 * e - 0.4 * e ** 1.5)
        p1 = (1.8 + 0.45 * e) / (1. + 0.15 * e ** 1.5)
        p2 = 2.3 - 0.05 * e / (1. + 0.025 * e)
        g = (a1 + a2 * y ** p1) / (1. + a3 * y ** p2 + a2 * y ** (p1 + 2.) / 13.75)
        total = total + weight * n_nuc * gamma / (x * x + (0.5 * gamma * g) ** 2) * s / T
    mc = (1. + (nb / 0.15e+18) ** (1. / 3.) / 3.) ** 6
    ab = 3. * BREM * total / mc
    return ab * _safe_exp(-x), ab


def _bessel_k1(x):
    t = (x / 3.75) ** 2
    i1 = x * _poly(t, [0.32411e-3, 0.301532e-2, 0.2658733e-1, 0.15084934, 0.51498869, 0.87890594,
                       0.5])
    y = x * x / 4.
    low = torch.log(x / 2.) * i1 + _poly(y, [-0.4686e-4, -0.110404e-2, -0.1919402e-1, -0.18156897,
                                             -0.67278579, 0.15443144, 1.]) / x
    high = torch.exp(-x) / torch.sqrt(x) * \
        _poly(2. / x, [-0.68245e-3, 0.325614e-2, -0.780353e-2, 0.1504268e-1, -0.3655620e-1,
                       0.23498619, 1.25331414])
    return torch.where(x <= 2., low, high)


def _brt06(E, w):
    T, yn, yp = E["temp"], E["yn"], E["yp"]
    q = 2.0778e+02 * 0.5 * MEV * (yn * yn + yp * yp + 28. / 3. * yn * yp) * \
        (E["nb"] * MB) ** 2 * T ** 5.5
    pre = (H * CLIGHT) ** 6 / (16. * math.pi ** 2) * 0.1409912109375 * q / T ** 7
    x = 0.5 * w / T
    k1 = pre * _bessel_k1(x) / x
    return k1 * _safe_exp(-x), k1 * _safe_exp(x)


def _gp19(E, w0, tab):
    """Quadrilinear interpolation of the response table with the reference's
    extrapolations below its densities and outside its temperatures."""
    dev = w0.device
    ax = {k: torch.as_tensor(tab[k], dtype=torch.float64, device=dev)
          for k in ("nb", "ye", "t", "w", "lognb", "logw")}
    data = torch.as_tensor(tab["data"], dtype=torch.float64, device=dev)
    D = tab["dims"]
    P = w0.shape[0]
    flat = w0.reshape(P, -1)
    w = flat.clamp(float(tab["w"][0]), float(tab["w"][-1]))
    T = E["temp"].reshape(P, 1)
    nb0 = E["nb"].reshape(P, 1) * 1e-18
    nbmin = float(tab["nb"][0])
    nb = nb0.clamp(nbmin, float(tab["nb"][-1]))
    ye = E["ye"].reshape(P, 1).clamp(max=float(tab["ye"][-1]))

    def bracket(v, a):
        i = (torch.searchsorted(a, v.contiguous()) - 1).clamp(0, a.numel() - 2)
        return i, (v - a[i]) / (a[i + 1] - a[i])

    i, tx = bracket(torch.log(nb), ax["lognb"])
    j, ty = bracket(ye, ax["ye"])
    l, tw = bracket(torch.log(w), ax["logw"])

    def at(temp):
        k, tz = bracket(temp, ax["t"])
        v = 0.
        for di, fi in ((0, 1. - tx), (1, tx)):
            for dj, fj in ((0, 1. - ty), (1, ty)):
                for dk, fk in ((0, 1. - tz), (1, tz)):
                    base = (((i + di) * D[1] + j + dj) * D[2] + k + dk) * D[3]
                    v = v + (data[base + l] * (1. - tw) + data[base + l + 1] * tw) * fi * fj * fk
        return BREM * nb * 1e18 * v

    scale = torch.where(nb0 < nbmin, (nb0 / nbmin) ** 2, torch.ones_like(nb0))
    full = torch.full_like(T, 0.)
    inside = at(T.clamp(float(tab["t"][0]), float(tab["t"][-1]))) * scale
    k2, k4 = at(full + 2.) * scale, at(full + 4.) * scale
    cold = k2 * (T * 0.5) ** (torch.log(k4 / k2) / math.log(2.))
    R48, R50 = at(full + 48.), at(full + 50.)
    n2 = (nb * 1e18) ** 2
    K = 4. * BREM * n2
    s50 = 7.0710678118654755
    A, B, m = 1. / R50, 1. / (K * s50), (R50 - R48) / 2.
    beta = 8. * w * w * K * B * B / (2. * m * A * A * s50 + A * K * B)
    gam = (A * beta - 4. * B * w * w) / (B * n2 * 50.)
    hot = BREM * nb * 1e18 * beta * nb * 1e18 / (T * torch.sqrt(T)) / \
        ((w / T) ** 2 + n2 / (4. * T) * gam) * scale
    s = torch.where(T < float(tab["t"][0]), cold, torch.where(T > float(tab["t"][-1]), hot, inside))
    s = (3. * s).abs().reshape(w0.shape)
    return s * _safe_exp(-w0 / E["temp"]), s


def _brem(E, w, impl, tab):
    if impl == HR98:
        return _hr98(E, w)
    return _brt06(E, w) if impl == BRT06 else _gp19(E, w, tab)


def _nes(E, w, wp):
    """Inelastic scattering kernels R_em, R_ab (four species each) at
    dimensionless energies w -> wp [1 or P, K], one direction."""
    T = E["temp"]
    w, wp = torch.broadcast_tensors(w + 0. * T, wp + 0. * T)
    x, y = torch.maximum(w, wp), torch.minimum(w, wp)
    d = wp - w
    sign = torch.where(d < 0., torch.ones_like(d), -torch.ones_like(d))
    em, ab = [0.] * 4, [0.] * 4
    ex = _safe_exp(-d.abs())
    den = -torch.expm1(-d.abs())
    efa = torch.where(d < 0., torch.ones_like(d), -ex) / den
    efb = torch.where(d < 0., -ex, torch.ones_like(d)) / den
    bz = 4. * SW2 ** 2
    for lepton, eta in ((0, E["mu_e"] / T), (1, -E["mu_e"] / T)):
        fw, fp = _fermi(eta - w, 1, 5), _fermi(eta - wp, 1, 5)
        fa, fe = _fermi(eta - d.abs(), 3, 5), _fermi(eta, 0, 5)
        dw = [a - b for a, b in zip(fp, fw)]
        da = [a - b for a, b in zip(fe[3:], fa)]
        S, wwp = w + wp, w * wp
        near = wwp * wwp
        a_out = ((sign * da[2] - dw[4]) * 0.2 -
                 S * (dw[3] + 2. * (S * dw[2] + 3. * wwp * dw[1])) +
                 sign * (x * da[1] + 2. * x * x * da[0])) / near - 6. * dw[0]
        b_out = ((sign * da[2] - dw[4]) * 0.2 +
                 sign * (-y * da[1] + 2. * y * y * da[0])) / near
        fx = _fermi(eta - x, 0, 2)
        fd0 = _occ(-eta)
        f = [fx[2] - fe[2], fx[1], fe[1], fx[0] + y * _occ(x - eta) / 6., fe[0] - y * fd0 / 6.]
        c = -sign * y / (x * x)
        a_one = c * (2. * f[0] + (y + 4. * x) * f[1] + (3. * y - 4. * x) * f[2] +
                     (0.2 * y * y + x * y + 2. * x * x) * f[3] -
                     (1.2 * y * y - 3. * x * y + 2. * x * x) * f[4])
        b_one = c * (2. * f[0] + 3. * y * f[1] + y * f[2] + 1.2 * y * y * f[3] -
                     0.2 * y * y * f[4])
        c = y * (w - wp) / (x * x)
        u = 4. * fe[1] + fd0 * (11. * y * y - 25. * x * y + 20. * x * x) / 30.
        v = (2. * x - y) * fe[0]
        out, one = y > eta * 1e-3, x > eta * 1e-3
        A = torch.where(out, a_out, torch.where(one, a_one, c * (u + v)))
        B = torch.where(out, b_out, torch.where(one, b_one, c * (u - v)))
        for s in range(4):
            bo = (2. * SW2 + 1.) ** 2 if s < 2 else (2. * SW2 - 1.) ** 2
            first = (s % 2 == 0) != (lepton == 1)
            r = NEPS * T * T * (A * bo + B * bz if first else A * bz + B * bo)
            em[s] = em[s] - r * efb
            ab[s] = ab[s] + r * efa
    return em, ab


def _nodes(n, dev):
    """The quadrature the calls are given (its nodes are an input, good to 1e-10)."""
    x, w = bn.quad_arrays(bn.gauss_legendre(n))
    return torch.as_tensor(x, device=dev), torch.as_tensor(w, device=dev)


def _grey_points(eos, m1, c, tab):
    """[20, P] grey opacities."""
    E = {k: eos[q].reshape(-1, 1) for q, k in enumerate(EOS)}
    T, n, J = E["temp"], m1[0:4], m1[4:8]
    d = _distribution(m1)
    x, w = _nodes(c["nquad"], eos.device)
    xs = torch.cat([x, 1. / x])
    ws = torch.cat([w, w / (x * x)])  # weights of the two half-intervals
    zero = torch.zeros_like(T[:, 0])
    S = {k: [zero] * 4 for k in ("n_em", "n_ab", "j_em", "j_ab", "iso")}
    stim = c["stim"]
    if c["abs_em"]:
        eta = (E["mu_e"] / T)
        for s in range(2):
            f4, f5 = _fermi(eta if s == 0 else -eta, 4, 5)
            inside = (eta > -30.) & (eta < 30.)
            t = torch.where(inside, T * f5 / f4,
                            torch.where((eta > 30.) == (s == 0), T * eta * 0.8333333333333333,
                                        T * 5.))
            nu = t * xs
            ab, em = _beta(E, nu, s)
            if stim:
                ab = ab + em
            g = _g(d, s, nu)
            for key, v in (("em", em), ("ab", g * ab)):
                base = ws * nu * nu * v
                S["n_" + key][s] = S["n_" + key][s] + FPHC3 * (t[:, 0] * base.sum(1))
                S["j_" + key][s] = S["j_" + key][s] + FPHC3 * (t[:, 0] * (base * nu).sum(1))
    if c["iso"]:
        for s in range(4):
            t = torch.where(n[s] > 1e-21, J[s] / n[s], 1.5 * T[:, 0]).reshape(-1, 1)
            nu = t * xs
            S["iso"][s] = (t * ws * _g(d, s, nu) * 4. * math.pi * nu ** 5 *
                           _iso(E, nu, True)).sum(1)
    if c["pair"] or c["use_brem"]:
        t2 = T2D * T
        nu = t2 * xs
        E3 = {k: v.reshape(-1, 1, 1) for k, v in E.items()}
        a, b = nu.unsqueeze(2), nu.unsqueeze(1)
        em, ab = [0.] * 4, [0.] * 4
        if c["pair"]:
            em, ab = _pair(E3, a, b)
        if c["use_brem"]:
            e, k = _brem(E3, a + b, c["brem"], tab)
            em, ab = [v + e for v in em], [v + k for v in ab]
        W = ws.reshape(1, -1, 1) * ws.reshape(1, 1, -1) * a * a * b * b
        g = [_g(d, s, nu) for s in range(4)]
        for s in range(4):
            ga, gb = g[s].unsqueeze(2), g[s ^ 1].unsqueeze(1)
            ke, ka = em[s] * (1. - gb), ab[s] * gb
            ka, ke = (ga * (ke + ka), ke) if stim else (ga * ka, ke * (1. - ga))
            for key, v in (("em", ke), ("ab", ka)):
                v = W * v
                u = FPHC3 ** 2 * t2[:, 0] ** 2
                S["n_" + key][s] = S["n_" + key][s] + u * v.sum((1, 2))
                S["j_" + key][s] = S["j_" + key][s] + u * (v * a).sum((1, 2))
    if c["nes"]:
        xi, xj, wi, wj = x.reshape(-1, 1), x.reshape(1, -1), w.reshape(-1, 1), w.reshape(1, -1)
        r0, r1 = 2. * T2D * xi, 2. * T2D / xi
        u = torch.cat([(r0 * (1. - xj)).reshape(1, -1), (r1 * (1. - xj)).reshape(1, -1)], 1)
        v = torch.cat([(r0 * (1. + xj)).reshape(1, -1), (r1 * (1. + xj)).reshape(1, -1)], 1)
        W = torch.cat([(wi * xi * wj).reshape(1, -1), (wi / xi ** 3 * wj).reshape(1, -1)], 1)
        e1, a1 = _nes(E, u, v)
        e2, a2 = _nes(E, v, u)
        nu, nub = u * T, v * T
        W = W * (nu * nub) ** 2
        unit = FPHC3 ** 2 * 0.5 * (4. * T2D * T[:, 0]) ** 2
        for s in range(4):
            g, gb = _g(d, s, nu), _g(d, s, nub)
            ke1, ka1, ke2, ka2 = e1[s] * gb, a1[s] * (1. - gb), e2[s] * g, a2[s] * (1. - g)
            if stim:
                ka1, ka2 = g * (ke1 + ka1), gb * (ke2 + ka2)
            else:
                ka1, ka2, ke1, ke2 = g * ka1, gb * ka2, ke1 * (1. - g), ke2 * (1. - gb)
            for key, p, q in (("em", ke1, ke2), ("ab", ka1, ka2)):
                S["n_" + key][s] = S["n_" + key][s] + unit * (W * (p + q)).sum(1)
                S["j_" + key][s] = S["j_" + key][s] + unit * (W * (p * nu + q * nub)).sum(1)
    out = torch.zeros((20, eos.shape[1]), dtype=torch.float64, device=eos.device)
    for s in range(4):
        cn, cj = CLIGHT * n[s], CLIGHT * J[s]
        okn, okj = n[s] > 1e-21, J[s] > 1e-25
        out[s], out[8 + s] = S["n_em"][s], S["j_em"][s]
        out[4 + s] = torch.where(okn, S["n_ab"][s] / cn, zero)
        out[12 + s] = torch.where(okj, S["j_ab"][s] / cj, zero)
        out[16 + s] = torch.where(okj, FPHC3 * S["iso"][s] / cj, zero)
    return out


def _spectral_points(eos, m1, c, tab):
    """[16, P, energies] spectral opacities."""
    E = {k: eos[q].reshape(-1, 1) for q, k in enumerate(EOS)}
    E3 = {k: v.reshape(-1, 1, 1) for k, v in E.items()}
    T = E["temp"]
    d = _distribution(m1)
    x, w = _nodes(c["nquad"], eos.device)
    xs, ws = torch.cat([x, 1. / x]), torch.cat([w, w / (x * x)])
    en = torch.as_tensor(_energies(c), device=eos.device).reshape(1, -1)
    nu = en + 0. * T
    j, k = [torch.zeros_like(nu) for _ in range(4)], [torch.zeros_like(nu) for _ in range(4)]
    if c["abs_em"]:
        for s in range(2):
            k[s], j[s] = _beta(E, nu, s)
    if c["pair"] or c["use_brem"]:
        t = T2D * T
        nub = t * xs
        a, b = nu.unsqueeze(2), nub.unsqueeze(1)
        em, ab = [0.] * 4, [0.] * 4
        if c["pair"]:
            em, ab = _pair(E3, a, b)
        if c["use_brem"]:
            e, q = _brem(E3, a + b, c["brem"], tab)
            em, ab = [v + e for v in em], [v + q for v in ab]
        W = FPHC3 * t.unsqueeze(2) * ws.reshape(1, 1, -1) * b * b
        for s in range(4):
            g = _g(d, s ^ 1, nub).unsqueeze(1)
            j[s] = j[s] + (W * em[s] * (1. - g)).sum(2)
            k[s] = k[s] + (W * ab[s] * g).sum(2)
    if c["nes"]:
        nub = nu.unsqueeze(2) * xs.reshape(1, 1, -1)
        em, ab = _nes(E3, nu.unsqueeze(2) / E3["temp"], nub / E3["temp"])
        W = FPHC3 * nu.unsqueeze(2) * ws.reshape(1, 1, -1) * nub * nub
        for s in range(4):
            g = _g(d, s, nub)
            j[s] = j[s] + (W * em[s] * g).sum(2)
            k[s] = k[s] + (W * ab[s] * (1. - g)).sum(2)
    iso = 4. * math.pi * nu * nu * _iso(E, nu, False) if c["iso"] else 0. * nu
    out = []
    for s in range(4):
        g = _g(d, s, nu)
        js, ks, ka = iso * g, iso * (1. - g) / CLIGHT, k[s] / CLIGHT
        if c["stim"]:
            ka, ks = ka + j[s] / CLIGHT, ks + js / CLIGHT
        out.append((j[s], ka, js, ks))
    return torch.stack([out[s][q] for q in range(4) for s in range(4)])


def _in_chunks(f, eos, m1, per_point):
    """f over slices of points whose largest arrays have about 4M entries."""
    step = max(1, int(4e6 // per_point))
    return torch.cat([f(eos[:, p:p + step], m1[:, p:p + step])
                      for p in range(0, eos.shape[1], step)], 1)


def _fermi_quadrature(x, j):
    """F_j(x) for j >= 0 with t = u^2 (smooth for half-integer orders):
    Gauss-Legendre panels around the Fermi edge u^2 = x."""
    node, weight = np.polynomial.legendre.leggauss(16)
    out = torch.empty_like(x)
    for p in range(0, x.numel(), 1 << 21):
        v = x[p:p + (1 << 21)]
        top = v.clamp(min=0.)
        cuts = [torch.sqrt((top + s).clamp(min=0.))
                for s in (-40., -25., -16., -9., -4.5, -1.5, 1.5, 4.5, 9., 16., 25., 40., 60.,
                          90., 130.)]
        # below the edge zone the occupation is 1 to 4e-18
        acc = cuts[0] ** (2. * j + 2.) / (j + 1.)
        for lo, hi in zip(cuts[:-1], cuts[1:]):
            h, m = 0.5 * (hi - lo), 0.5 * (hi + lo)
            for t, w in zip(node, weight):
                u = m + h * float(t)
                acc = acc + float(w) * h * 2. * u ** (2. * j + 1.) * _occ(u * u - v)
        out[p:p + (1 << 21)] = acc
    return out


def exact(case, seed):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    call = case["call"]
    if call == "fdi":
        if case["twice_order"] < 0:
            return None
        x = _fdi_arguments(case, seed)
        if case["twice_order"] in (0, 2, 4, 6, 8, 10):
            k = case["twice_order"] // 2
            return {"F": _fermi(x, k, k)[0]}
        return {"F": _fermi_quadrature(x, case["twice_order"] / 2.)}
    blocks = _block_list(case, seed) if call == "blocks" else None
    if blocks:
        n = blocks[-1]["first"] + blocks[-1]["count"]
    elif call == "boxes":
        nx, ny, nz = _boxes(case)
        n = nx * ny * nz
    else:
        n = case["n"]
    eos_h, m1_h = _points(n, seed)
    eos, m1 = torch.from_numpy(eos_h).to(dev), torch.from_numpy(m1_h).to(dev)
    if call == "equilibrium":
        return _exact_equilibrium(eos)
    from bns_nurates_gb300 import gp19_synthetic
    tab = gp19_synthetic.table()
    if call == "spectral":
        M = 2 * case["nquad"] * case["energies"]
        out = _in_chunks(lambda e, m: _spectral_points(e, m, case, tab), eos, m1, M)
        return {name: out[4 * k:4 * k + 4] for k, name in enumerate(SPECTRAL)}
    if blocks:
        out = torch.empty((20, n), dtype=torch.float64, device=dev)
        groups = {}
        for b in blocks:
            groups.setdefault((b["brem"], b["nes"], b["nquad"]), []).append(b)
        for members in groups.values():
            at = torch.cat([torch.arange(b["first"], b["first"] + b["count"], device=dev)
                            for b in members])
            out[:, at] = _in_chunks(lambda e, m: _grey_points(e, m, members[0], tab), eos[:, at],
                                    m1[:, at], 4 * members[0]["nquad"] ** 2)
        return _fields(out)
    out = _in_chunks(lambda e, m: _grey_points(e, m, case, tab), eos, m1, 4 * case["nquad"] ** 2)
    if call == "point":
        return {name: out[4 * k:4 * k + 4, 0].cpu().tolist() for k, name in enumerate(FIELDS)}
    if call == "boxes":
        g = 3
        full = torch.zeros((20, nz + 2 * g, ny + 2 * g, nx + 2 * g), dtype=torch.float64,
                           device=dev)
        full[:, g:g + nz, g:g + ny, g:g + nx] = out.reshape(20, nz, ny, nx)
        return _fields(full)
    return _fields(out)


def _exact_equilibrium(eos):
    T = eos[1]
    eta = (eos[7] - eos[6] + eos[5]) / T
    one, zero = torch.ones_like(T), torch.zeros_like(T)
    etas = torch.stack([eta, -eta, zero, zero])
    Ts = T.expand(4, -1)
    distr = torch.cat([one.expand(4, -1), Ts, etas, zero.expand(4, -1), Ts,
                       (0.6 * one).expand(4, -1), one.expand(4, -1)])
    f2, f3 = _fermi(etas, 2, 3)
    n, J = FPHC3 * T ** 3 * f2, FPHC3 * T ** 4 * f3
    chi = (one / 3.).expand(4, -1)
    d = _distribution(torch.cat([n, J, chi]))
    return {"distr": distr, "n": n, "J": J, "chi": chi, "eta_t": d["eta_t"],
            "temp_t": d["temp_t"], "temp_f": d["temp_f"],
            "weights": torch.stack([d["w_t"], d["w_f"], d["c_f"]]), "beta_f": d["beta_f"]}
