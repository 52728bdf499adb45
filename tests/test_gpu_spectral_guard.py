"""Mixed spectral opacities whose FP32 pair sums the NES sums cancel at points where NES
runs in FP64 from the start (an occupation outside the FP32 range): the error bound of
the pair sums is compared with the total that holds the FP64 NES sums.

The states: the antineutrino occupation exceeds 1, so that the pair emissivity of nu_e
(1 - g < 0) is negative, and nu_e's own occupation is scaled until its NES emissivity
cancels all but a thousandth of it at one energy per point.  The contract is
test_gpu_mixed.py's: 1e-6 where the FP64 result moves by at most 1e-9 under two ulps in T
or mu_e.
"""

import numpy as np
import pytest

import bns_nurates_gb300 as bn
from conftest import rel_err
from test_gpu_mixed import MIXED_TOL, WELL_CONDITIONED

pytestmark = pytest.mark.gpu

W_T, TEMP_T, ETA_T, W_F, TEMP_F, C_F, BETA_F = (4 * k for k in range(7))


def cancelling_states(port, nq, npts=24):
    """eos, m1, distr and an energy per point (about 2 T) of the states above."""
    eos, m1 = bn.synthetic_points(4711, 400)
    sel = np.flatnonzero((eos[1] > 3.) & (eos[1] < 40.) & (eos[7] < 2. * eos[1]))[:npts]
    eos, m1 = np.ascontiguousarray(eos[:, sel]), np.ascontiguousarray(m1[:, sel])
    T, n = eos[1], len(sel)
    d = np.zeros((28, n))
    d[TEMP_T:TEMP_T + 4] = d[TEMP_F:TEMP_F + 4] = T
    d[C_F:C_F + 4] = 0.6
    d[W_F:W_F + 4] = 1.
    d[BETA_F] = 1. / T ** 0.6           # nu_e
    d[BETA_F + 1] = 60. / T ** 0.6      # anti-nu_e: above 1 for E between T / 100 and 6 T
    d[BETA_F + 2:BETA_F + 4] = 1e-31    # outside the FP32 range
    energies = 2. * T
    pars, q = (1, 0, 1, 1, 1, 0, 1, 0), port.gauss_legendre(nq)
    for k in range(n):
        one = [np.ascontiguousarray(a[:, k:k + 1]) for a in (eos, m1, d)]
        pair, nes = (port.spectral(one[0], one[1], fl, pars, q, energies[k:k + 1], distr=one[2],
                                   stimulated=0)[0, 0, 0]
                     for fl in ((0, 1, 0, 0, 0), (0, 0, 0, 1, 0)))
        assert pair < 0. < nes
        d[BETA_F, k] *= -pair / nes * 1.001
    return eos, m1, d, energies, pars


@pytest.mark.parametrize("nq", [6, 20])
def test_pair_sums_cancelled_by_fp64_nes_are_recomputed(cuda, port, nq):
    torch = cuda
    eos, m1, d, energies, pars = cancelling_states(port, nq)
    fl, pa, q = (bn.opacity_flags(0, 1, 0, 1, 0), bn.opacity_params(brem_implementation=0),
                 bn.gauss_legendre(nq))

    def run(e, precision):
        t = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (e, m1, d)]
        out = bn.spectral_opacities(t[0], t[1], fl, pa, q, energies, distr=t[2], stimulated=0,
                                    precision=precision).cpu().numpy()
        return np.stack([out[:, k, k] for k in range(len(energies))], axis=1)

    bn.spectral_mixed_stats(reset=True)
    mixed = run(eos, "mixed")
    assert bn.spectral_mixed_stats()["pb_fp64"] >= len(energies)
    ref = run(eos, "fp64")
    sens = np.zeros_like(ref)
    for row in (1, 7):
        e2 = eos.copy()
        e2[row] *= 1. + 2. ** -51
        sens = np.maximum(sens, rel_err(run(e2, "fp64"), ref, floor=1e-300))
    r, well = rel_err(mixed, ref, floor=1e-300), sens <= WELL_CONDITIONED
    assert well[0].mean() > 0.9
    assert r[well].max() <= MIXED_TOL, float(r[well].max())
