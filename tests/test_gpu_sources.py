"""Shots of many sources through the tile list (csrc/psv_loop.cu): more in a
tile than lanes, several on one cell, and what a line of them costs."""
import numpy as np
import pytest

import helpers
from fwi_cuda_gb300 import engine
from test_gpu_loop import _both

pytestmark = pytest.mark.gpu


def _line(sv, n, cells):
    """n sources a shot on `cells` neighbouring cells from the shot's own."""
    x = np.asarray(sv.x_src)[:, None] - cells // 2 + np.arange(n)[None] % cells
    sv.x_src = x.reshape(-1).astype(np.int32)
    sv.z_src = np.repeat(np.asarray(sv.z_src), n)
    sv.src_shot_to_fire = np.repeat(np.asarray(sv.src_shot_to_fire), n)
    for k in ("stf_z", "stf_x"):
        w = np.repeat(np.asarray(getattr(sv, k)), n, axis=0)
        setattr(sv, k, w * (1.0 + 0.01 * np.arange(len(w)))[:, None])  # not all alike
    return sv


@pytest.mark.parametrize("rpt", [2, 4])
@pytest.mark.parametrize("n,cells", [(33, 33), (70, 9), (40, 1)])
def test_sources_on_shared_cells(gpu, rpt, n, cells):
    sv, true, init = helpers.case(fdorder=4, nz=70, nx=150, nshot=2, nt=150, surf_offset=0)
    _both(_line(sv, n, cells), true, tuple(0.97 * a for a in init), rpt)


def test_a_line_of_sources_costs_little(gpu):
    # half of a shot's tiles along x hold 60 sources each
    us = []
    for n in (1, 300):
        sv, true, _ = helpers.case(fdorder=4, nz=301, nx=601, nshot=8, nt=200, npml=20, surf_offset=0)
        if n > 1:
            sv.x_src = np.full(sv.nsrc, 300, np.int32)
            _line(sv, n, n)
        with engine.Plan(sv, precision=32, kernels="tma", rows_per_thread=4) as p:
            p.set_model(*true)
            p.forward()
            t = []
            for _ in range(5):
                p.forward()
                t.append(p.timing()["forward_ms"])
            us.append(min(t))
    assert us[1] < 1.6 * us[0]
