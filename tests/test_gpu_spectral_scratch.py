"""Device memory that a spectral call takes from the library's pool.  It is measured in a
process of its own, since the pool keeps what earlier calls took."""

import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = """
import sys
import torch
import bns_nurates_gb300 as bn
ne, precision = int(sys.argv[1]), sys.argv[2]
eos, m1 = bn.synthetic_points(3, 300000)
e, m = torch.from_numpy(eos).cuda(), torch.from_numpy(m1).cuda()
args = (bn.opacity_flags(), bn.opacity_params(), bn.gauss_legendre(2), [10. + k for k in range(ne)])
bn.spectral_opacities(e[:, :8].contiguous(), m[:, :8].contiguous(), *args, precision=precision)
out = torch.empty((16, 300000, ne), dtype=torch.float64, device="cuda")
torch.cuda.synchronize()
free = torch.cuda.mem_get_info()[0]
bn.spectral_opacities(e, m, *args, precision=precision, out=out)
torch.cuda.synchronize()
print(free - torch.cuda.mem_get_info()[0])
"""


@pytest.mark.parametrize("ne", [1, 4, 24])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_scratch_of_a_large_call(cuda, ne, precision):
    """Two areas of at most 45 MB (include/bns_nurates_gb300.h), in the pool's granules of
    up to 32 MB."""
    got = subprocess.run([sys.executable, "-c", CHILD, str(ne), precision], cwd=ROOT,
                         capture_output=True, text=True, timeout=300)
    assert got.returncode == 0, got.stderr
    assert int(got.stdout.split()[-1]) <= 2 * 45_000_000 + (32 << 20), got.stdout
