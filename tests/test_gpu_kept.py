"""What a context keeps between calls (captured steps, factors, buffers) against the same call made afresh.

Comparisons are bitwise where both routes launch the same kernels on the same values.
"""
import numpy as np
import pytest

from td1c_b200 import workloads as W

from .helpers import oracle_tables, oracle_state

WL = dict(W.MIXED_SMALL, igauge=1, split_type=1)


def _context(wl=WL, **kw):
    from oracle.oracle import Oracle
    from td1c_b200.hprod import HProd
    o = Oracle(wl)
    rad, ang = oracle_tables(o)
    h = HProd(wl, rad, ang, **kw)
    orb, cic = oracle_state(o)
    h.set_wfn0(orb, cic)
    return h, orb, cic


class _State:
    """Device buffers that are reset in place, so that every run of a step works on the same addresses."""

    def __init__(self, orb, cic):
        import torch
        self.torch = torch
        self.x0, self.c0 = torch.from_numpy(orb.reshape(-1).copy()).cuda(), torch.from_numpy(cic.copy()).cuda()
        self.x, self.c = self.x0.clone(), self.c0.clone()

    def run(self, h, step, **kw):
        self.x.copy_(self.x0)
        self.c.copy_(self.c0)
        self.torch.cuda.synchronize()
        step(self.x.data_ptr(), self.c.data_ptr(), **kw)
        h.sync()
        return np.concatenate([self.x.cpu().numpy(), self.c.cpu().numpy()])


def _steps(h):
    return {
        "rk4": lambda x, c, use_graph=True: h.rk4_dev(x, c, 30.0, 0.002, 3, use_graph=use_graph),
        "split2": lambda x, c, use_graph=True: h.split2_dev(x, c, 30.0, 0.004, 3, use_graph=use_graph),
        "etdrk2": lambda x, c, use_graph=True: h.etdrk2_dev(x, c, 30.0, 0.004, 3, use_graph=use_graph),
        "etdrk4": lambda x, c, use_graph=True: h.etdrk4_dev(x, c, 30.0, 0.004, 3, use_graph=use_graph),
    }


KINDS = ["rk4", "split2", "etdrk2", "etdrk4"]


@pytest.mark.gpu
@pytest.mark.parametrize("kind", KINDS)
def test_captured_step_after_another_frozen_core(cuda_ok, kind):
    h, orb, cic = _context()
    try:
        s, step = _State(orb, cic), _steps(h)[kind]
        before = s.run(h, step)
        h.set_wfn0(0.7 * orb, cic)
        after = s.run(h, step)  # no other call in between that would build the new factors
        assert np.array_equal(after, s.run(h, step, use_graph=False))
        assert not np.array_equal(after, before)
    finally:
        h.final()


@pytest.mark.gpu
@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("change", ["split", "mixed_external"])
def test_captured_step_after_a_change_of_setting(cuda_ok, kind, change):
    h, orb, cic = _context()
    try:
        s, step = _State(orb, cic), _steps(h)[kind]
        if change == "mixed_external":
            h.set_mixed(2)
        before = s.run(h, step)
        if change == "split":
            h.set_split(2)
        else:
            h.set_mixed(0)
            h.set_mf_external(True)  # W and int2e stay as the last step left them
        after = s.run(h, step)
        assert np.array_equal(after, s.run(h, step, use_graph=False))
        assert not np.array_equal(after, before)
    finally:
        h.final()


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["split2", "etdrk2", "etdrk4"])
def test_captured_step_after_its_factor_slot_was_taken(cuda_ok, kind):
    """More one-body factors than the context keeps, built between two runs of a captured step: narrow and wide
    bands (short and long steps) take the places of the step's own."""
    h, orb, cic = _context()
    try:
        s, step = _State(orb, cic), _steps(h)[kind]
        first = s.run(h, step)
        y = s.x0.clone()
        for k in range(32):
            h.h1itr_dev(y.data_ptr(), np.zeros(9), 0.001 * 1.2 ** k, maxcyc=1)
        assert np.array_equal(s.run(h, step), first)
    finally:
        h.final()


@pytest.mark.gpu
def test_captured_step_after_another_restart_state(cuda_ok):
    h, orb, cic = _context()
    try:
        s = _State(orb, cic)
        for kind in KINDS:
            step = _steps(h)[kind]
            d = 0.5 * s.c0
            h.rk4_reset(s.x0.data_ptr(), s.c0.data_ptr())
            before = s.run(h, step)
            h.rk4_reset(s.x0.data_ptr(), d.data_ptr())
            after = s.run(h, step)
            assert np.array_equal(after, s.run(h, step, use_graph=False))
            assert not np.array_equal(after, before)
    finally:
        h.final()


@pytest.mark.gpu
def test_learned_steps_after_another_frozen_core(cuda_ok):
    """With a bound of zero no prediction stands, so the learned steps are the exact ones."""
    h, orb, cic = _context()
    try:
        s = _State(orb, cic)
        h.set_learned(None, bound=0.0)

        def learned(x, c):
            h.split2_learned_dev(x, c, 30.0, 0.004, 12)

        def exact(x, c):
            h.split2_dev(x, c, 30.0, 0.004, 12, use_graph=False)
        assert np.array_equal(s.run(h, learned), s.run(h, exact))
        h.set_wfn0(0.7 * orb, cic)
        assert np.array_equal(s.run(h, learned), s.run(h, exact))
    finally:
        h.final()
