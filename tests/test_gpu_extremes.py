"""States at the ends of the number range against the CPU oracle: temperatures of 0 and
next to it, infinite chemical potentials and energy densities.  What the reference makes of
them is an accident of its clamped exponentials, but it is finite in many outputs, and
the FP64 path follows it.  Tolerance: the plain path's 1e-12.
"""

import numpy as np
import pytest

import bns_nurates_gb300 as bn
from test_gpu_mixed import _check, _spec_oracle_with_sens
from test_gpu_parity import (DEFAULT, F, P, assert_close, gpu_grey, oracle_grey,
                             port_fma)  # noqa: F401

pytestmark = pytest.mark.gpu

ENERGIES = np.array([0.1, 1., 7., 30., 100., 300.])
MU_P, MU_N, MU_E, TEMP = 5, 6, 7, 1


def spectral_both(torch, port, eos, m1, flags, pars, precision="fp64", stim=1, energies=ENERGIES,
                  nq=6):
    got = bn.spectral_opacities(torch.from_numpy(eos).cuda(), torch.from_numpy(m1).cuda(), F(flags),
                                P(*pars), bn.gauss_legendre(nq), energies, stimulated=stim,
                                precision=precision).cpu().numpy()
    return got, port.spectral(eos, m1, flags, pars, port.gauss_legendre(nq), energies,
                              stimulated=stim)


def states(row, values):
    eos, m1 = bn.synthetic_points(3, 3 * len(values))
    eos[row] = np.tile(values, 3)
    return eos, m1


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("stim", [0, 1])
@pytest.mark.parametrize("row,values", [
    (TEMP, [0., 1e-310, 1e-200, 1e-20, 1e-4]), (MU_E, [np.inf, -np.inf]),
    (MU_P, [np.inf, -np.inf]), (MU_N, [np.inf, -np.inf]),
])
def test_spectral_beta_rates(cuda, port, row, values, stim, precision):
    eos, m1 = states(row, values)
    got, want = spectral_both(cuda, port, eos, m1, (1, 0, 0, 0, 0), DEFAULT, precision, stim)
    assert_close(got, want, what="beta rates")


@pytest.mark.parametrize("row,values", [
    (TEMP, [1e-310, 1e-200, 1e-20]), (MU_E, [np.inf, -np.inf]), (MU_P, [np.inf, -np.inf]),
    (MU_N, [np.inf, -np.inf]),
])
def test_grey_beta_rates(cuda, port, row, values):
    eos, m1 = states(row, values)
    args = (m1, (1, 0, 0, 0, 0), DEFAULT, 6)
    assert_close(gpu_grey(cuda, eos, *args), oracle_grey(port, eos, *args), what="beta rates")


@pytest.mark.parametrize("flags", [(1, 0, 0, 0, 0), (0, 0, 1, 0, 0), (0, 0, 0, 1, 0)])
def test_grey_infinite_energy_density(cuda, port, flags):
    eos, m1 = bn.synthetic_points(5, 8)
    m1[4:8] = np.inf
    args = (m1, flags, DEFAULT, 6)
    assert_close(gpu_grey(cuda, eos, *args), oracle_grey(port, eos, *args), what="J = inf")


@pytest.mark.parametrize("nq", [6, 20])
@pytest.mark.parametrize("flags,brem", [((0, 1, 0, 0, 0), 0), ((0, 0, 1, 0, 0), 2)])
def test_spectral_pair_and_brem_next_to_zero_temperature(cuda, port, flags, brem, nq):
    """Energies far above e^700 T, nodes whose weight underflows."""
    eos, m1 = states(TEMP, [1e-310, 1e-200, 1e-100, 1e-30])
    got, want = spectral_both(cuda, port, eos, m1, flags, DEFAULT[:5] + (brem,) + DEFAULT[6:], nq=nq)
    assert_close(got, want, what="T next to 0")


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_spectral_brt06_emission_far_above_the_temperature(cuda, port, precision):
    """K_1(x/2) e^{-x/2} at x = (nu + nubar) / T beyond 700, where a clamped e^{-x} would stay at
    e^-700.  Densities far above nuclear ones lift the difference over the smallest doubles."""
    eos, m1 = bn.synthetic_points(5, 4)
    eos[0], eos[TEMP] = 1e39, [1., 1.4, 1.2, 0.7]
    got, want = spectral_both(cuda, port, eos, m1, (0, 0, 1, 0, 0),
                              DEFAULT[:5] + (1,) + DEFAULT[6:], precision, 0,
                              np.array([400., 900., 960., 1100., 1400.]))
    assert_close(got[:4], want[:4], what="BRT06 emission")


@pytest.mark.parametrize("nq", [6, 20])
def test_mixed_spectral_energies_at_the_fermi_edge_of_cold_electrons(cuda, port, port_fma, nq):
    """eta_e of thousands and energies just below mu_e: the FP32 pair integral's scale
    e^{(nu + nubar - mu_e) / T} is a product of two numbers outside the double range there."""
    eos, m1 = bn.synthetic_points(23, 8)
    eos[TEMP] = np.tile([0.05, 0.07, 0.1, 0.12], 2)
    eos[MU_E] = np.repeat([170., 140.], 4)
    energies = np.array([128., 131., 136., 139.5, 150., 161., 166., 169.5])
    flags, pars = (1, 1, 1, 1, 1), DEFAULT
    got, _ = spectral_both(cuda, port, eos, m1, flags, pars, "mixed", 1, energies, nq)
    want, sens = _spec_oracle_with_sens(port, port_fma, eos, m1, flags, pars, nq, energies)
    _check(got, want, sens, "cold electrons")
