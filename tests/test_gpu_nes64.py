"""The FP64 NES/NPS kernel's forms against the CPU oracle: a point per CTA
(small launches) and per warp, both stimulated-absorption modes, neglected
blocking, quadrature orders at the edges of a warp's item count, and given
distributions whose thin-part exponent differs from the reconstruction's 0.6.
Tolerances are those of test_gpu_parity.py."""

import numpy as np
import pytest

import bns_nurates_gb300 as bn
from test_gpu_parity import assert_close, gpu_grey, grey_probes, oracle_grey

pytestmark = pytest.mark.gpu

NES = (0, 0, 0, 1, 0)


@pytest.fixture(scope="module")
def port_fma():
    import oracle
    return oracle.port_fma()


@pytest.mark.parametrize("batch", [16, 1024, 1041])
@pytest.mark.parametrize("nq,stim,nbb,cf", [(1, 1, 0, None), (4, 0, 0, None), (7, 1, 1, None),
                                            (10, 0, 1, 0.55), (20, 1, 0, None), (12, 1, 0, 0.7)])
def test_nes64_forms(cuda, port, port_fma, batch, nq, stim, nbb, cf):
    eos, m1 = bn.synthetic_points(77, batch)
    pars = (1, 0, 1, 1, 1, 0, 1, nbb)
    distr = port.distr_from_m1(eos, m1)
    if cf is not None:
        distr[21] = cf   # c_f of one species
    sub = [np.ascontiguousarray(a[:, :16]) for a in (eos, m1, distr)]
    got = gpu_grey(cuda, eos, m1, NES, pars, nq, stim=stim, distr=distr)[:, :16]
    args = (sub[1], NES, pars, nq)
    want = oracle_grey(port, sub[0], *args, stim=stim, distr=sub[2])
    pr = grey_probes(port, port_fma, sub[0], *args, stim=stim, distr=sub[2])
    assert_close(got, want, pr, what=f"batch {batch} nq {nq}")


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("nq,stim", [(1, 1), (5, 0), (12, 1), (20, 1)])
def test_nes_forms_agree_bitwise(cuda, precision, nq, stim):
    """A point's NES sums do not depend on how many warps share it: the same
    points in a call small enough for a point per CTA and in a large one."""
    torch = cuda
    eos, m1 = bn.synthetic_points(78, 1600)
    e, m = torch.from_numpy(eos).cuda(), torch.from_numpy(m1).cuda()
    q = bn.gauss_legendre(nq)
    args = (bn.opacity_flags(*NES), bn.opacity_params(), q)
    large = bn.m1_opacities(e, m, *args, stim_abs=stim, precision=precision)
    small = bn.m1_opacities(e[:, :100].contiguous(), m[:, :100].contiguous(), *args,
                            stim_abs=stim, precision=precision)
    assert torch.equal(large[:, :100], small)
