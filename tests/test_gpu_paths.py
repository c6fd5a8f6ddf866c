"""The kernels that run many steps, each case with the path that it names:
tiles of 64 columns on chip (two quads of columns a thread, whose CPML memories
go through L1), and checkpointed states of the tile list.

A batch of more than 152 x 2048 points does not fit the chip in tiles of 32
columns (152 SMs, at most 64 rows a CTA); eight rows per thread run on chip or
with a stress launch of their own, which a profile times.  Bars as in
test_gpu_loop.py."""
import numpy as np
import pytest

import helpers
from fwi_cuda_gb300 import engine

pytestmark = pytest.mark.gpu

WIDE = 152 * 2048


def _run(sv, true, init, obs=None, **kw):
    with engine.Plan(sv, precision=32, **kw) as p:
        if obs is None:
            p.set_model(*true)
            obs = p.forward()
        p.set_model(*init)
        traces = p.forward()
        p.set_observed(*obs)
        L2, g = p.gradient()
        steps = p.profile_kernels(4)["stress_fwd"] == 0  # no launch of half a step
        shape = p.shape[:2]
    return obs, traces, L2, g, steps, shape


def _on_chip(sv, true, init, **kw):
    obs, ta, La, ga, _, _ = _run(sv, true, init, kernels="direct", rows_per_thread=1, **kw)
    _, tb, Lb, gb, steps, shape = _run(sv, true, init, obs, kernels="tma", rows_per_thread=8, **kw)
    assert steps and shape == ("tma", 8)
    assert min(sv.nshot, kw.get("max_batch", sv.nshot)) * sv.nz * sv.nx > WIDE
    for a, b in zip(ta, tb):
        assert np.abs(a).max() > 0 and helpers.rel_l2(b, a) < 1e-5
    assert Lb == pytest.approx(La, rel=1e-4)
    for a, b in zip(ga, gb):
        assert np.isfinite(a).all() and np.abs(a).max() > 0 and helpers.rel_l2(b, a) < 1e-4


def _near(sv):
    """Receivers that the short records' waves reach: beside every source."""
    z = np.asarray(sv.z_src)[:, None] + np.array([-9, -2, 5, 12])[None]
    sv.z_rec = z.reshape(-1).astype(np.int32)
    sv.x_rec = np.full(z.size, int(sv.x_src[0]) + 7, np.int32)
    return sv


def _slow(model):
    """Moduli ten per cent lower: all three scaled alike would leave the field
    of a velocity source, and so the residual, as it is."""
    lam, mu, rho = model
    return 0.9 * lam, 0.9 * mu, rho


@pytest.mark.parametrize("kw", [dict(fdorder=2, nt=270), dict(fdorder=8, nt=150, nx=301),
                                dict(fdorder=4, nt=150, stf_type=0, snap_dt=1), dict(fdorder=6, nt=100, nz=391)])
@pytest.mark.parametrize("step", [1, 2])
def test_wide_tiles_cpml_on_four_sides_and_a_short_last_batch(gpu, kw, step):
    sv, true, init = helpers.crosswell(stencil="holberg", nshot=5, **dict(dict(nz=337, nx=329), **kw))
    sv.snap_dz = sv.snap_dx = step
    _near(sv)
    _on_chip(sv, true, _slow(init), max_batch=4 if sv.nx < 320 else 3)


def test_wide_tiles_with_more_receivers_and_sources_than_lanes(gpu):
    sv, true, init = helpers.case(nz=401, nx=801, nshot=1, nt=120, snap_dt=3, surf_offset=2)
    sv.x_rec = np.arange(100, 740, dtype=np.int32)
    sv.z_rec = np.full(640, sv.isurf[0] + 2, np.int32)
    n = 90  # sources of the shot, some on one cell
    for k in ("z_src", "src_shot_to_fire", "stf_z", "stf_x"):
        setattr(sv, k, np.repeat(np.asarray(getattr(sv, k))[:1], n, axis=0))
    sv.x_src = (np.asarray(sv.x_src)[:1] + np.arange(n) % 40).astype(np.int32)
    _on_chip(sv, true, _slow(init))


@pytest.mark.parametrize("rpt", [2, 4, 8])
@pytest.mark.parametrize("storage", ["checkpoint", "binomial"])
def test_checkpointed_states(gpu, rpt, storage):
    sv, true, init = helpers.case(nz=301, nx=601, nshot=2, nt=170, snap_dt=3, fdorder=8, surf_offset=0)
    kw = dict(kernels="tma", rows_per_thread=rpt)
    obs, _, La, ga, steps, shape = _run(sv, true, _slow(init), storage="full", **kw)
    assert steps and shape == ("tma", rpt) and sv.nshot * sv.nz * sv.nx > WIDE
    _, _, Lb, gb, steps, shape = _run(sv, true, _slow(init), obs, storage=storage, checkpoint_interval=17,
                                      checkpoint_slots=4 if storage == "binomial" else 0, **kw)
    assert steps and shape == ("tma", rpt) and La == Lb
    for a, b in zip(ga, gb):
        assert np.isfinite(a).all() and np.abs(a).max() > 0 and np.array_equal(a, b)


def test_wide_tiles_through_the_drop_in(gpu):
    sv, true, init = helpers.crosswell(stencil="holberg", nshot=1, fdorder=4, nz=577, nx=601, nt=150, snap_dt=5)
    _near(sv)
    assert sv.nz * sv.nx > WIDE
    lam, mu, rho = true
    mzx, rzp, rxp = np.zeros_like(mu), np.zeros_like(mu), np.zeros_like(mu)
    mzx[:-1, :-1] = 4 / (1 / mu[:-1, :-1] + 1 / mu[:-1, 1:] + 1 / mu[1:, :-1] + 1 / mu[1:, 1:])
    rzp[:-1, :-1] = 2 / (rho[:-1, :-1] + rho[1:, :-1])
    rxp[:-1, :-1] = 2 / (rho[:-1, :-1] + rho[:-1, 1:])
    names = ("a", "b", "K", "a_half", "b_half", "K_half")
    snap = (sv.snap_z1, sv.snap_z2, sv.snap_x1, sv.snap_x2, sv.snap_dt, 1, 1)

    def call(precision, grad, src, stf, stf_type, history=None):
        return engine.kernel_PSV(0, sv.nt, sv.nz, sv.nx, sv.dt, sv.dx, sv.dz, sv.surf, sv.isurf, sv.hc, sv.fdorder,
                                 lam, mu, mzx, rzp, rxp, grad, sv.pml_z, [getattr(sv, n + "_z") for n in names],
                                 sv.pml_x, [getattr(sv, n + "_x") for n in names], len(src[0]), stf_type, *stf,
                                 *src, np.zeros(len(src[0]), np.int32), 0 if grad else sv.nrec, 0, sv.z_rec, sv.x_rec,
                                 not grad, snap, history=history, stencil=sv.stencil, precision=precision)

    out = []
    for precision in (64, 32):
        f = call(precision, False, (sv.z_src, sv.x_src), (sv.stf_z, sv.stf_x), sv.stf_type)
        h = out[0][0]["history"] if out else f["history"]
        t = out[0][0] if out else f
        b = call(precision, True, (sv.z_rec, sv.x_rec), (t["rtf_uz"], t["rtf_ux"]), 0, history=h)
        out.append((f, b))
    (fa, ba), (fb, bb) = out
    for k in ("vz", "vx", "uz", "ux", "szz", "szx", "sxx", "We", "rtf_uz", "rtf_ux", "mem_vx_x", "mem_szz_z"):
        assert np.abs(fa[k]).max() > 0 and helpers.rel_l2(fb[k], fa[k]) < 1e-5, k
    for k in fa["history"]:
        assert helpers.rel_l2(fb["history"][k], fa["history"][k]) < 1e-5, k
    for k in ("grad_lam", "grad_mu", "grad_rho", "uz", "We"):
        assert np.abs(ba[k]).max() > 0 and helpers.rel_l2(bb[k], ba[k]) < 1e-4, k


def test_on_chip_plans_at_once_with_a_residual(gpu):
    plans, alone = [], []
    try:
        for k, (nz, nx, nshot) in enumerate(((61, 91, 1), (130, 200, 2), (281, 561, 2))):
            sv, true, init = helpers.case(nz=nz, nx=nx, nshot=nshot, nt=150, seed=k + 1, surf_offset=0)
            p = engine.Plan(sv, precision=32, kernels="tma", rows_per_thread=8)
            plans.append(p)
            p.set_model(*true)
            obs = p.forward()
            p.set_model(*_slow(init))
            p.set_observed(*obs)
            alone.append(p.gradient())
            p.reset_gradient()
        L2 = engine.multi_gradient(plans)
        for k, p in enumerate(plans):
            assert L2[k] == alone[k][0] > 0
            for a, b in zip(alone[k][1], p.get_gradient()):
                assert np.isfinite(a).all() and np.abs(a).max() > 0 and np.array_equal(a, b)
    finally:
        for p in plans:
            p.close()
