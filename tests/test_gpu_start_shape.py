"""The kernels a plan starts with when nobody autotunes it."""
import pytest

import helpers
from fwi_cuda_gb300 import engine

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nz,nx,nshot", [(61, 91, 4), (301, 601, 4)])  # fits the chip; above 500 000 points
@pytest.mark.parametrize("opt", [dict(block=(32, 8)), dict(block=(32, 2), chains=2), dict(chains=1), dict(chains=2),
                                 dict(chains=4)])
def test_block_and_chains_given_are_used(gpu, nz, nx, nshot, opt):
    sv, _, _ = helpers.case(nz=nz, nx=nx, nshot=nshot, nt=4, surf_offset=0)
    for autotune in (False, True):
        with engine.Plan(sv, precision=32, autotune=autotune, **opt) as p:
            assert p.shape == ("direct", 1, opt.get("block", (32, 4))[1])
            assert p.chains == opt.get("chains", 1)
