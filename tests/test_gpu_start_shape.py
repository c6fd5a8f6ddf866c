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


@pytest.mark.parametrize("nz,nx,nshot,shape", [
    (40, 4000, 8, ("direct", 1)), (64, 2000, 12, ("direct", 1)), (64, 2000, 32, ("tma", 4)), (32, 2000, 80, ("direct", 1)),
    (80, 2000, 5, ("direct", 1)), (80, 2000, 8, ("tma", 4)), (128, 1000, 4, ("tma", 8)), (128, 1000, 6, ("direct", 1)),
    (129, 1000, 6, ("tma", 4)), (61, 91, 200, ("direct", 1)), (200, 72, 60, ("tma", 4))])
def test_grids_of_few_bands_step_with_the_direct_kernels(gpu, nz, nx, nshot, shape):
    # Fewer than five bands of 16 rows: the tile list took 24 us a step on
    # 40 x 4000, 4 shots, the direct kernels 15.
    sv, _, _ = helpers.case(nz=nz, nx=nx, nshot=nshot, nt=4, npml=4, surf_offset=0)
    with engine.Plan(sv, precision=32) as p:
        assert p.shape[:2] == shape
