"""Time steps with the wavefields on chip (TMA family, eight rows per thread,
csrc/psv_resident.cu) where it can go wrong: one tile, ragged last tiles of
either axis, tall tiles and two CTAs per SM, every order, mirrored surface
rows, CPML on four sides, more sources or receivers in a tile than lanes, a
short last batch, checkpointed states, passes of several launches, several
plans at once.

Bars as in test_gpu_loop.py: rounding alone parts the families by less than
1e-5 of a trace's norm, ten times that in a gradient."""
import numpy as np
import pytest

import helpers
from fwi_cuda_gb300 import engine
from fwi_cuda_gb300 import survey as S
from test_gpu_loop import _both

pytestmark = pytest.mark.gpu


def _surface(nz, nx, order, nshot, nt=150, nrec=12, rec_spacing=4, **kw):
    vp = S.layered_vp(nz, nx, 3, 1800.0, 3000.0, np.random.default_rng(nz))
    sv = S.surface_survey(nz, nx, 0.5, 0.5, nt, 5e-5, fdorder=order, npml=3, nshot=nshot,
                          nrec=min(nrec, (nx - 10) // rec_spacing), rec_spacing=rec_spacing, fc=300.0,
                          surf_offset=0, **kw)
    return sv, S.model_from_vp(vp), S.model_from_vp(0.97 * vp)


@pytest.mark.parametrize("order,nz,nx,nshot", [
    (2, 16, 31, 1), (4, 31, 33, 2), (6, 47, 131, 2), (8, 41, 129, 2), (4, 64, 128, 1), (8, 97, 190, 2),
    (4, 301, 601, 1),   # tiles of 38 rows
    (2, 330, 288, 3),   # four CTAs on an SM
    (8, 211, 333, 4),   # two quads a thread
    (6, 380, 701, 2)])  # ... in tiles of 64 rows
def test_ragged_grids_with_a_surface(gpu, order, nz, nx, nshot):
    _both(*_surface(nz, nx, order, nshot, snap_dt=2), 8)


@pytest.mark.parametrize("offset", [1, 9])
def test_mirrored_rows(gpu, offset):
    sv, true, init = helpers.case(fdorder=4, nz=61, nx=91, nshot=1, nt=150, surf_offset=offset)
    _both(sv, true, tuple(0.97 * a for a in init), 8)


@pytest.mark.parametrize("kw", [dict(fdorder=2, nt=530), dict(fdorder=8, nt=270, nz=90, nx=75),
                                dict(fdorder=4, nt=300, stf_type=0, snap_dt=1)])
def test_cpml_on_four_sides_subsampled_and_batched(gpu, kw):
    sv, true, init = helpers.crosswell(stencil="holberg", nshot=3, **kw)
    sv.snap_dz = sv.snap_dx = 2
    _both(sv, true, tuple(0.97 * a for a in init), 8, max_batch=2)


def test_more_receivers_and_sources_in_a_tile_than_lanes(gpu):
    sv, true, init = _surface(64, 128, 4, 1, nrec=100, rec_spacing=1, snap_dt=3)
    n = 40  # sources of one shot, some on one cell
    for k in ("z_src", "x_src", "src_shot_to_fire", "stf_z", "stf_x"):
        v = np.asarray(getattr(sv, k))
        setattr(sv, k, np.repeat(v[:1], n, axis=0).copy())
    sv.x_src = np.asarray(sv.x_src) + np.arange(n) % 24
    _both(sv, true, init, 8)


@pytest.mark.parametrize("storage", ["checkpoint", "binomial"])
def test_checkpointed_states(gpu, storage):
    sv, true, init = _surface(97, 130, 8, 2, nt=200, snap_dt=3)
    got = []
    with engine.Plan(sv, precision=32) as p:
        p.set_model(*true)
        obs = p.forward()
    for kw in (dict(storage="full"), dict(storage=storage, checkpoint_interval=17)):
        with engine.Plan(sv, precision=32, kernels="tma", rows_per_thread=8, **kw) as p:
            p.set_model(*init)
            p.set_observed(*obs)
            got.append(p.gradient())
    assert got[0][0] == got[1][0]
    for a, b in zip(got[0][1], got[1][1]):
        assert np.array_equal(a, b)


def test_four_plans_at_once(gpu):
    # the larger grids' waves meet no difference of the models in 200 steps:
    # no residual, 0 / 0 in their gradients whatever the kernels
    plans, alone = [], []
    try:
        for k, (nz, nx) in enumerate(((61, 91), (130, 200), (201, 401), (281, 561))):
            sv, true, init = helpers.case(nz=nz, nx=nx, nshot=1, nt=200, seed=k + 1)
            p = engine.Plan(sv, precision=32, kernels="tma", rows_per_thread=8)
            plans.append(p)
            p.set_model(*true)
            obs = p.forward()
            p.set_model(*init)
            p.set_observed(*obs)
            alone.append((p.gradient(), p.forward()))
            p.reset_gradient()
        L2 = engine.multi_gradient(plans)
        traces = engine.multi_forward(plans)
        for k, p in enumerate(plans):
            assert p.shape[:2] == ("tma", 8)
            assert L2[k] == alone[k][0][0]
            for a, b in zip(alone[k][0][1], p.get_gradient()):
                assert np.array_equal(a, b, equal_nan=True)
            for a, b in zip(alone[k][1], traces[k]):
                assert np.abs(a).max() > 0 and np.array_equal(a, b)
    finally:
        for p in plans:
            p.close()


def test_plans_that_run_together_take_kernels_that_mix(gpu):
    plans = []
    try:
        for k in range(2):
            sv, true, _ = helpers.case(nz=61, nx=91, nshot=1, nt=40, seed=k + 1)
            p = engine.Plan(sv, precision=32)
            plans.append(p)
            p.set_model(*true)
            assert p.shape[:2] == ("tma", 8)
            alone = p.forward()
        traces = engine.multi_forward(plans)
        for p in plans:
            assert p.shape[:2] != ("tma", 8)
        for a, b in zip(alone, traces[1]):
            assert helpers.rel_l2(b, a) < 1e-5
    finally:
        for p in plans:
            p.close()
