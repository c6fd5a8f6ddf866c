"""The storage budget: what it admits depends on the grid and the window's
size, not on the columns the window starts at or the kernels the plan has."""
import numpy as np
import pytest

import helpers
from fwi_cuda_gb300 import _lib, engine

pytestmark = pytest.mark.gpu


def _survey(x1, nt=60):
    sv, true, init = helpers.case(nz=101, nx=201, nshot=2, nt=nt, snap_dt=2, npml=14, surf_offset=0)
    sv.snap_x1, sv.snap_x2 = x1, x1 + 159  # five rows of 32: nothing to spare for an offset
    return sv, true, tuple(0.97 * a for a in init)


def _least(sv, **opt):
    lo, hi = 0.0, 1.0
    for _ in range(40):
        mid = 0.5 * (lo + hi)
        try:
            engine.Plan(sv, hbm_budget_gb=mid, **opt).close()
            hi = mid
        except _lib.PSVError:
            lo = mid
    return hi


@pytest.mark.parametrize("storage", ["full", "checkpoint", "binomial"])
def test_the_least_budget(gpu, storage):
    opt = dict(storage=storage, checkpoint_interval=7)
    least = {_least(_survey(x1)[0], kernels=k, **opt) for x1 in (16, 17, 19) for k in ("any", "direct", "tma")}
    assert len(least) == 1


@pytest.mark.parametrize("kernels", ["any", "tma"])
def test_states_without_room_for_kept_roundings(gpu, kernels):
    sv, true, init = _survey(17, nt=240)
    opt = dict(precision=32, storage="checkpoint", checkpoint_interval=13, kernels=kernels, max_batch=1, autotune=False)
    tight = _least(sv, **opt)
    got, size = [], []
    with engine.Plan(sv, precision=32) as p:
        p.set_model(*true)
        obs = p.forward()
    for gb in (tight, 2.0 * tight):
        with engine.Plan(sv, hbm_budget_gb=gb, **opt) as p:
            assert p.shape[0] == "tma"
            p.set_model(*init)
            p.set_observed(*obs)
            got.append(p.gradient())
            size.append(p.device_bytes)
    assert size[0] < size[1]
    assert got[0][0] == pytest.approx(got[1][0], rel=1e-4)
    for a, b in zip(got[0][1], got[1][1]):
        assert np.abs(a).max() > 0 and helpers.rel_l2(a, b) < 1e-4
