"""A point's spectral opacities do not depend on the size of the call: small mixed calls share
a point's energies between warps, for energy counts below, at and above a pass (32) and a
launch (64), and quadratures whose lane groups differ."""

import numpy as np
import pytest

import bns_nurates_gb300 as bn

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("brem", [0, 1, 2])
@pytest.mark.parametrize("nq,ne", [(1, 3), (4, 24), (10, 1), (10, 40), (12, 33), (20, 65)])
def test_small_calls_agree_bitwise(cuda, nq, ne, brem, precision):
    torch = cuda
    large = 5 * torch.cuda.get_device_properties(0).multi_processor_count
    eos, m1 = bn.synthetic_points(61, large)
    e, m = torch.from_numpy(eos).cuda(), torch.from_numpy(m1).cuda()
    args = (bn.opacity_flags(), bn.opacity_params(brem_implementation=brem),
            bn.gauss_legendre(nq), np.logspace(-1., 2.5, ne))
    whole = bn.spectral_opacities(e, m, *args, precision=precision)
    for n in (1, 16, 90, 300):
        part = bn.spectral_opacities(e[:, :n].contiguous(), m[:, :n].contiguous(), *args,
                                     precision=precision)
        assert torch.equal(whole[:, :n], part), n
