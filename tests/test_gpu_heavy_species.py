"""Heavy-lepton neutrinos and antineutrinos evolved separately (species 3 differs from
species 2, so none of the kernels may take one's occupation for the other's): every form
of the grey kernels and both spectral paths against the oracle, with the tolerances of
test_gpu_parity.py and test_gpu_mixed.py."""

import numpy as np
import pytest

import bns_nurates_gb300 as bn
from test_gpu_mixed import _check, _gpu, _oracle_with_sens, _params, _spec_oracle_with_sens
from test_gpu_parity import (COND_SPEC, F, P, assert_close, gpu_grey, grey_probes, oracle_grey,
                             port_fma, probes)  # noqa: F401

pytestmark = pytest.mark.gpu

ALL = (1, 1, 1, 1, 1)
PARS = (1, 0, 1, 1, 1, 2, 1, 0)
NREF = 24


def points(n):
    eos, m1 = bn.synthetic_points(91, n)
    m1[3] *= 1.7
    m1[7] *= 1.3
    m1[11] = np.minimum(1., 1.05 * m1[11])
    return eos, m1


def head(a):
    return np.ascontiguousarray(a[:, :NREF])


def large_batch(torch):
    """More points than take the one-point-per-CTA forms (5 per SM in FP64)."""
    return 6 * torch.cuda.get_device_properties(0).multi_processor_count


@pytest.mark.parametrize("large", [0, 1])
@pytest.mark.parametrize("nq,stim", [(6, 0), (12, 1), (20, 1)])
def test_grey_fp64(cuda, port, port_fma, nq, stim, large):
    eos, m1 = points(large_batch(cuda) if large else NREF)
    got = gpu_grey(cuda, eos, m1, ALL, PARS, nq, stim=stim)[:, :NREF]
    args = (head(m1), ALL, PARS, nq)
    want = oracle_grey(port, head(eos), *args, stim=stim)
    assert (want[3] != want[2]).any()
    assert_close(got, want, grey_probes(port, port_fma, head(eos), *args, stim=stim),
                 what=f"nq {nq} large {large}")


@pytest.mark.parametrize("large", [0, 1])
@pytest.mark.parametrize("nq,stim", [(6, 0), (20, 1)])
def test_grey_mixed(cuda, port, port_fma, nq, stim, large):
    eos, m1 = points(large_batch(cuda) if large else NREF)
    got = _gpu(cuda, eos, m1, ALL, PARS, nq, "mixed", stim=stim)[:, :NREF]
    want, sens = _oracle_with_sens(port, port_fma, head(eos), head(m1), ALL, PARS, nq, stim=stim)
    _check(got, want, sens, f"nq {nq} large {large}")


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("nq,stim", [(6, 0), (20, 1)])
def test_spectral(cuda, port, port_fma, nq, stim, precision):
    eos, m1 = points(NREF)
    energies = np.logspace(0., np.log10(300.), 24)
    got = bn.spectral_opacities(cuda.from_numpy(eos).cuda(), cuda.from_numpy(m1).cuda(), F(ALL),
                                P(*PARS), bn.gauss_legendre(nq), energies, stimulated=stim,
                                precision=precision).cpu().numpy()
    if precision == "mixed":
        want, sens = _spec_oracle_with_sens(port, port_fma, eos, m1, ALL, PARS, nq, energies,
                                            stim=stim)
        _check(got, want, sens, f"nq {nq}")
    else:
        q = port.gauss_legendre(nq)
        args = (eos, m1, ALL, PARS, q, energies)
        assert_close(got, port.spectral(*args, stimulated=stim),
                     probes(port.spectral, port_fma.spectral, *args, stimulated=stim),
                     what=f"nq {nq}", cond=COND_SPEC)
