"""A point's sums do not depend on how many threads share its cells or on which phases share
a launch: the same points in a call small enough for the wide forms and the joint launch of
pair, brem and NES and in a large one, for every brem kernel, each subset of the
reactions, fewer cells than threads, and several rounds of them."""

import pytest

import bns_nurates_gb300 as bn

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("brem", [0, 1, 2])
@pytest.mark.parametrize("nq,stim", [(2, 1), (5, 0), (10, 1), (20, 1)])
@pytest.mark.parametrize("pair,use_brem,nes", [(1, 1, 0), (1, 1, 1), (0, 1, 1), (1, 0, 0)])
def test_cell_forms_agree_bitwise(cuda, nq, stim, brem, pair, use_brem, nes):
    torch = cuda
    eos, m1 = bn.synthetic_points(31, 700)
    e, m = torch.from_numpy(eos).cuda(), torch.from_numpy(m1).cuda()
    args = (bn.opacity_flags(1, pair, use_brem, nes, 1), bn.opacity_params(brem_implementation=brem),
            bn.gauss_legendre(nq))
    large = bn.m1_opacities(e, m, *args, stim_abs=stim)
    small = bn.m1_opacities(e[:, :90].contiguous(), m[:, :90].contiguous(), *args, stim_abs=stim)
    assert torch.equal(large[:, :90], small)
