"""Shots of many sources, and arrays of receivers, in the kernels that run many
steps: more in a tile than a CTA has threads, several on one cell, and what
they cost against the direct kernels."""
import numpy as np
import pytest

import helpers
from fwi_cuda_gb300 import engine

pytestmark = pytest.mark.gpu


def _patch(sv, side, copies=1):
    """side x side x copies sources a shot, below and right of the shot's own."""
    n = side * side * copies
    d = np.arange(n) % (side * side)
    sv.z_src = (np.asarray(sv.z_src)[:, None] + d[None] // side).reshape(-1).astype(np.int32)
    sv.x_src = (np.asarray(sv.x_src)[:, None] + d[None] % side).reshape(-1).astype(np.int32)
    sv.src_shot_to_fire = np.repeat(np.asarray(sv.src_shot_to_fire), n)
    for k in ("stf_z", "stf_x"):
        w = np.repeat(np.asarray(getattr(sv, k)), n, axis=0) / n
        setattr(sv, k, w * (1.0 + 0.01 * np.arange(len(w)))[:, None])  # not all alike
    return sv


def _array(sv, step):
    """Receivers on every step-th cell below the surface, off the frame."""
    z, x = np.meshgrid(np.arange(8, sv.nz - 8, step), np.arange(8, sv.nx - 8, step), indexing="ij")
    sv.z_rec, sv.x_rec = z.reshape(-1).astype(np.int32), x.reshape(-1).astype(np.int32)
    return sv


@pytest.mark.parametrize("rpt", [2, 4, 8])
@pytest.mark.parametrize("side,copies,step", [(12, 1, 1), (24, 1, 3), (6, 3, 2), (11, 6, 5), (1, 40, 1)])
def test_dense_points(gpu, rpt, side, copies, step):
    # bars as in test_gpu_loop.py
    sv, true, init = helpers.case(fdorder=4, nz=70, nx=150, nshot=2, nt=150, surf_offset=0)
    sv.x_src = np.array([60, 90], np.int32)
    _array(_patch(sv, side, copies), step)
    init = tuple(0.97 * a for a in init)
    out = []
    for kw in (dict(kernels="direct", rows_per_thread=1), dict(kernels="tma", rows_per_thread=rpt)):
        with engine.Plan(sv, precision=32, **kw) as p:
            if not out:
                p.set_model(*true)
                obs = p.forward()
            p.set_model(*init)
            t = p.forward()
            p.set_observed(*obs)
            L2, g = p.gradient()
            assert kw["kernels"] == "direct" or p.profile_kernels(4)["stress_fwd"] == 0
            out.append((t, L2, g))
    (ta, La, ga), (tb, Lb, gb) = out
    for a, b in zip(ta, tb):
        assert np.abs(a).max() > 0 and helpers.rel_l2(b, a) < 1e-5
    assert Lb == pytest.approx(La, rel=1e-4)
    for a, b in zip(ga, gb):
        assert np.isfinite(a).all() and np.abs(a).max() > 0 and helpers.rel_l2(b, a) < 1e-4


@pytest.mark.parametrize("nz,nx,nshot", [(101, 201, 1), (301, 601, 1), (281, 561, 2), (301, 601, 8)])
@pytest.mark.parametrize("dense", [lambda sv: _patch(sv, 8), lambda sv: _patch(sv, 16), lambda sv: _patch(sv, 30),
                                   lambda sv: _array(sv, 1), lambda sv: _array(sv, 2)],
                         ids=["64 sources", "256 sources", "900 sources", "all cells", "every other cell"])
def test_an_untuned_plan_is_no_slower_than_the_direct_kernels(gpu, nz, nx, nshot, dense):
    sv, true, _ = helpers.case(fdorder=4, nz=nz, nx=nx, nshot=nshot, nt=60, npml=10, surf_offset=0)
    sv.x_src = np.full(nshot, nx // 2, np.int32)
    dense(sv)
    ms = []
    for kw in (dict(), dict(kernels="direct")):
        with engine.Plan(sv, precision=32, autotune=False, **kw) as p:
            p.set_model(*true)
            p.forward()
            t = []
            for _ in range(5):
                p.forward()
                t.append(p.timing()["forward_ms"])
            ms.append(min(t))
    assert ms[0] < 1.1 * ms[1]


@pytest.mark.parametrize("nz,nx,nshot,side,every,shape", [
    (301, 601, 1, 1, 2, ("tma", 8)), (301, 601, 1, 10, 6, ("tma", 8)), (301, 601, 1, 16, 6, ("direct", 1)),
    (301, 601, 1, 1, 1, ("direct", 1)),
    (301, 601, 8, 1, 5, ("tma", 4)), (301, 601, 8, 12, 5, ("tma", 4)), (301, 601, 8, 30, 5, ("direct", 1)),
    (301, 601, 8, 1, 2, ("direct", 1))])
def test_start_shape_of_crowded_tiles(gpu, nz, nx, nshot, side, every, shape):
    sv, true, _ = helpers.case(fdorder=4, nz=nz, nx=nx, nshot=nshot, nt=4, npml=10, surf_offset=0)
    sv.x_src = np.full(nshot, 330, np.int32)
    _array(_patch(sv, side), every)
    with engine.Plan(sv, precision=32) as p:
        assert p.shape[:2] == shape


def test_a_crowded_survey_is_tuned_by_itself(gpu):
    # the choice of a plan with few points does not become a crowded one's
    small, true, init = helpers.case(fdorder=4, nz=301, nx=601, nshot=1, nt=120, npml=10, surf_offset=0)
    dense, _, _ = helpers.case(fdorder=4, nz=301, nx=601, nshot=1, nt=120, npml=10, surf_offset=0)
    _patch(dense, 60)
    us = {}
    for name, sv, kw in (("few", small, {}), ("many", dense, {}),
                         ("direct", dense, dict(kernels="direct", rows_per_thread=1, block=(32, 4)))):
        with engine.Plan(sv, precision=32, **kw) as p:
            p.set_model(*true)
            p.set_observed(*p.forward())
            p.set_model(*init)
            for _ in range(3):
                p.gradient(fetch=False)
            t = p.timing()
            us[name] = t["forward_ms"] + t["adjoint_ms"]
    assert us["many"] < 1.1 * us["direct"]
