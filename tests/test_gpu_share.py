"""Plans that run alone, together (psv_multi_*) and alone again: together they
step with kernels that mix, alone with their own, whatever came before."""
import numpy as np
import pytest

import helpers
from fwi_cuda_gb300 import _lib, engine

pytestmark = pytest.mark.gpu


def _plans(n, **opt):
    out = []
    for k in range(n):
        sv, true, init = helpers.case(nz=61, nx=91, nshot=1, nt=120, seed=k + 1)
        p = engine.Plan(sv, precision=32, **opt)
        out.append((p, true, tuple(0.97 * a for a in init)))
    return out


def _same(a, b):
    return all(np.abs(x).max() > 0 and np.array_equal(x, y) for x, y in zip(a, b))


def test_alone_after_together_is_alone_again(gpu):
    plans = _plans(2)
    try:
        before = []
        for p, true, init in plans:
            p.set_model(*true)
            before.append(p.forward())
            assert p.shape[:2] == ("tma", 8)
        together = engine.multi_forward([p for p, *_ in plans])
        for p, *_ in plans:
            assert p.shape == ("direct", 1, 4)  # as such a plan starts without the chip to itself
        again = engine.multi_forward([p for p, *_ in plans])
        for k, (p, true, init) in enumerate(plans):
            assert _same(p.forward(), before[k]) and p.shape[:2] == ("tma", 8)
            assert _same(again[k], together[k])
            p.set_model(*init)
            p.set_observed(*before[k])
        alone, L2 = [], []
        for p, *_ in plans:
            L, g = p.gradient()
            alone.append(g)
            L2.append(L)
            shape = p.shape
            p.reset_gradient()
        both = engine.multi_gradient([p for p, *_ in plans])
        for k, (p, *_) in enumerate(plans):
            assert both[k] == pytest.approx(L2[k], rel=1e-4)
            for a, b in zip(alone[k], p.get_gradient()):
                assert np.abs(a).max() > 0 and helpers.rel_l2(b, a) < 1e-4
            p.reset_gradient()
            L, g = p.gradient()
            assert L == L2[k] and _same(g, alone[k]) and p.shape == shape
    finally:
        for p, *_ in plans:
            p.close()


def test_together_first(gpu):
    # the second shape is built before the first has run
    plans = _plans(2, storage="checkpoint", checkpoint_interval=11)
    try:
        for p, true, init in plans:
            p.set_model(*true)
        obs = engine.multi_forward([p for p, *_ in plans])
        for (p, true, init), o in zip(plans, obs):
            p.set_observed(*o)
            p.set_model(*init)
        L2 = engine.multi_gradient([p for p, *_ in plans])
        for k, (p, *_) in enumerate(plans):
            together = p.get_gradient()
            p.reset_gradient()
            L, g = p.gradient()
            assert L == pytest.approx(L2[k], rel=1e-4)
            for a, b in zip(g, together):
                assert np.abs(a).max() > 0 and helpers.rel_l2(b, a) < 1e-4
    finally:
        for p, *_ in plans:
            p.close()


def test_a_refused_call_changes_no_plan(gpu):
    plans = _plans(2)
    try:
        (p, true, _), (r, *_) = plans
        p.set_model(*true)
        with pytest.raises(_lib.PSVError, match="twice"):
            engine.multi_forward([p, p])
        assert p.shape[:2] == ("tma", 8)
        with pytest.raises(_lib.PSVError, match="no model"):
            engine.multi_forward([p, r])
        assert r.shape[:2] == ("tma", 8)
        p.forward()
        assert p.shape[:2] == ("tma", 8)
        assert len(engine.multi_forward([p])) == 1 and p.shape[:2] == ("tma", 8)  # one plan is alone
    finally:
        for p, *_ in plans:
            p.close()
