"""Many time steps per launch (TMA family, csrc/psv_loop.cu) at the sizes where
it can go wrong: grids of one, two and a few bands of tiles, ragged tiles,
every order, mirrored surface rows, CPML on four sides, subsampled snapshots,
a short last batch, passes of several launches, several plans at once.

Bars against the direct family: both round every operation to 24 bits, about
20 operations a point and step, so over nt steps the traces part by about
6e-8 sqrt(20 nt) < 1e-5 of their norm; a gradient magnifies that by the traces
over their residual, at most ten here (1e-4)."""
import numpy as np
import pytest

import helpers
from fwi_cuda_gb300 import engine
from fwi_cuda_gb300 import survey as S

pytestmark = pytest.mark.gpu


def _both(sv, true, init, rpt, **opt):
    out = []
    obs = None
    for kernels, r in (("direct", 1), ("tma", rpt)):
        with engine.Plan(sv, precision=32, kernels=kernels, rows_per_thread=r, **opt) as p:
            assert p.shape[0] == kernels
            if obs is None:
                p.set_model(*true)
                obs = p.forward()
            p.set_model(*init)
            traces = p.forward()
            p.set_observed(*obs)
            L2, g = p.gradient()
            out.append((traces, L2, g))
    (ta, La, ga), (tb, Lb, gb) = out
    for a, b in zip(ta, tb):
        assert np.abs(a).max() > 0 and helpers.rel_l2(b, a) < 1e-5
    assert Lb == pytest.approx(La, rel=1e-4)
    for a, b in zip(ga, gb):
        assert np.abs(a).max() > 0 and helpers.rel_l2(b, a) < 1e-4


@pytest.mark.parametrize("rpt", [2, 4])
@pytest.mark.parametrize("fdorder,nz,nx", [(2, 16, 65), (4, 31, 63), (6, 47, 131), (8, 41, 129),
                                           (4, 64, 128), (8, 97, 190)])
def test_ragged_grids_with_a_surface(gpu, fdorder, nz, nx, rpt):
    vp = S.layered_vp(nz, nx, 3, 1800.0, 3000.0, np.random.default_rng(nz))
    sv = S.surface_survey(nz, nx, 0.5, 0.5, 150, 5e-5, fdorder=fdorder, npml=3, nshot=2, nrec=12, fc=300.0,
                          snap_dt=2, surf_offset=0)
    _both(sv, S.model_from_vp(vp), S.model_from_vp(0.97 * vp), rpt)  # a residual in the direct waves


@pytest.mark.parametrize("rpt,offset", [(4, 2), (2, 1), (2, 9)])
def test_mirrored_rows(gpu, rpt, offset):
    # 9 rows above the surface do not fit in a tile of 8: that plan steps with
    # the two-launch kernels
    sv, true, init = helpers.case(fdorder=4, nz=61, nx=91, nshot=1, nt=150, surf_offset=offset)
    init = tuple(0.97 * a for a in init)
    _both(sv, true, init, rpt)


@pytest.mark.parametrize("rpt,kw", [(2, dict(fdorder=2, nt=530)), (4, dict(fdorder=8, nt=270, nz=90, nx=75)),
                                    (4, dict(fdorder=4, nt=300, stf_type=0, snap_dt=1))])
def test_cpml_on_four_sides_subsampled_and_batched(gpu, rpt, kw):
    sv, true, init = helpers.crosswell(stencil="holberg", nshot=3, **kw)
    sv.snap_dz = sv.snap_dx = 2
    init = tuple(0.97 * a for a in init)
    _both(sv, true, init, rpt, max_batch=2)


def test_two_plans_at_once(gpu):
    plans, alone = [], []
    try:
        for k, (nz, nx) in enumerate(((61, 91), (130, 200))):
            sv, true, init = helpers.case(nz=nz, nx=nx, nshot=2, nt=200, seed=k + 1)
            p = engine.Plan(sv, precision=32, kernels="tma", rows_per_thread=2)
            plans.append(p)
            p.set_model(*true)
            obs = p.forward()
            p.set_model(*init)
            p.set_observed(*obs)
            L2, g = p.gradient()
            alone.append((L2, g))
            p.reset_gradient()
        L2 = engine.multi_gradient(plans)
        for k, p in enumerate(plans):
            assert L2[k] == alone[k][0]
            for a, b in zip(alone[k][1], p.get_gradient()):
                assert np.array_equal(a, b)
    finally:
        for p in plans:
            p.close()


def test_the_shape_a_plan_starts_with(gpu):
    # 500 000 points of a batch and a surface the loop handles
    for nz, nx, nshot, precision, isurf, family in ((501, 1001, 1, 32, None, "tma"), (301, 601, 2, 32, None, "tma"),
                                                    (301, 601, 4, 32, None, "tma"), (501, 1001, 1, 64, None, "direct"),
                                                    (501, 1001, 1, 32, (40, 0, 0, 0), "direct")):
        sv, _, _ = helpers.case(nz=nz, nx=nx, nshot=nshot, nt=4, surf_offset=0)
        if isurf:
            sv.isurf = isurf
        with engine.Plan(sv, precision=precision) as p:
            assert p.shape[0] == family
