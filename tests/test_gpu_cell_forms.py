"""A point's sums do not depend on the launch form, beyond test_gpu_cells.py: the large call
has more points than any one-point-per-CTA form takes (5 per SM), so that the joint launch
of pair, brem and NES meets the two-warp NES kernel, and brem alone runs, whose wide kernel
no other small FP64 call launches."""

import pytest

import bns_nurates_gb300 as bn

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("brem", [0, 1, 2])
@pytest.mark.parametrize("nq,stim", [(2, 1), (5, 0), (10, 1), (20, 1)])
@pytest.mark.parametrize("pair,use_brem,nes", [(0, 1, 0), (1, 1, 1), (0, 1, 1)])
def test_forms_agree_bitwise(cuda, nq, stim, brem, pair, use_brem, nes):
    torch = cuda
    large = 6 * torch.cuda.get_device_properties(0).multi_processor_count
    eos, m1 = bn.synthetic_points(32, large)
    e, m = torch.from_numpy(eos).cuda(), torch.from_numpy(m1).cuda()
    args = (bn.opacity_flags(1, pair, use_brem, nes, 1), bn.opacity_params(brem_implementation=brem),
            bn.gauss_legendre(nq))
    whole = bn.m1_opacities(e, m, *args, stim_abs=stim)
    for n in (1, 90, 400):
        part = bn.m1_opacities(e[:, :n].contiguous(), m[:, :n].contiguous(), *args, stim_abs=stim)
        assert torch.equal(whole[:, :n], part), n
