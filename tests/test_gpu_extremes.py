"""States at the ends of the number range against the CPU oracle: temperatures of 0 and
next to it, infinite chemical potentials and energy densities.  What the reference makes of
them is an accident of its clamped exponentials, but it is finite in many outputs, and
the FP64 path follows it.  Tolerance: the plain path's 1e-12.
"""

import numpy as np
import pytest

import bns_nurates_gb300 as bn
from test_gpu_parity import DEFAULT, F, P, assert_close, gpu_grey, oracle_grey

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
