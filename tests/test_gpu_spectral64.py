"""Spectral opacities at the edges of the FP64 kernels' work: quadratures from one node
to the largest, energy counts around a pass over the cells (16 at n = 20, 32 below
n = 11) and a chunk of energies (32, 64), and energies from nu/T ~ 10^-3, where the pair
kernel takes its low-energy pass, to nu/T ~ 10^3, where the reference clamps e^x.

Against the oracle with the tolerance of the spectral parity tests: 1e-12, or 64 times
what an ulp in the inputs or Fermi integrals moves the oracle itself.
"""

import numpy as np
import pytest

import bns_nurates_gb300 as bn
from test_gpu_parity import (COND_SPEC, DEFAULT, F, P, assert_close, port_fma,  # noqa: F401
                             probes)

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nq,ne,brem,nes", [
    (1, 1, 0, 1), (2, 33, 1, 1), (4, 65, 0, 1), (10, 32, 2, 0), (11, 31, 0, 1), (20, 17, 2, 1),
    (20, 16, 1, 0),
])
def test_spectral_vs_oracle_at_edges(cuda, port, port_fma, nq, ne, brem, nes):
    eos, m1 = bn.synthetic_points(17 * nq, 5)
    flags, pars = (1, 1, 1, nes, 1), DEFAULT[:5] + (brem,) + DEFAULT[6:]
    energies = np.logspace(-1., 3., ne)
    out = bn.spectral_opacities(cuda.from_numpy(eos).cuda(), cuda.from_numpy(m1).cuda(), F(flags),
                                P(*pars), bn.gauss_legendre(nq), energies)
    cuda.cuda.synchronize()
    q = port.gauss_legendre(nq)
    want = port.spectral(eos, m1, flags, pars, q, energies)
    pr = probes(port.spectral, port_fma.spectral, eos, m1, flags, pars, q, energies)
    assert_close(out.cpu().numpy(), want, pr, what="spectral", cond=COND_SPEC)
