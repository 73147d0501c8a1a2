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


SECOND = {
    "larger": dict(WL, nfe=15, rmax=28.0, rmask=22.0, lmax1=7, lmax2=14),
    "other_elements": dict(WL, ndvr=10, nfe=6, rmax=11.0, rmask=8.0),
    "more_orbitals": dict(W.NE_SMALL, split_type=1),
}


def _ensemble(h, wl, x, c):
    import ctypes

    def one(t, v):
        return (t * 1)(v)
    d = ctypes.c_double
    rc = h.lib._lib.td1c_gpu_ensemble_split2(1, one(ctypes.c_int, h.ctx_id), one(ctypes.c_void_p, x), one(ctypes.c_void_p, c),
                                             one(d, 30.0), one(d, 0.004), 3, one(d, wl["fint"]), one(d, wl["wlen"]),
                                             one(d, wl["numcyc"]), one(d, wl["cep"]), 20, 1e-10, ctypes.byref(d(0.0)))
    assert rc == 0


def _everything(h, wl, orb, cic):
    """One call of each kind that keeps something in the context."""
    s, out = _State(orb, cic), {}
    lf = np.zeros(9)
    lf[2], lf[5], lf[8] = 0.8, 0.1, 0.8
    out["htot"] = np.concatenate([v.reshape(-1) for v in h.htot(1.0, lf, orb, cic)])
    for kind, step in _steps(h).items():
        out[kind] = s.run(h, step)
        assert np.array_equal(out[kind], s.run(h, step))
    out["ensemble"] = s.run(h, lambda x, c: _ensemble(h, wl, x, c))
    out["dipole"] = np.array([h.dipole_dev(s.x.data_ptr(), s.c.data_ptr())])
    out["dipole3"] = np.concatenate(h.dipole3_dev(s.x.data_ptr(), s.c.data_ptr(), lf))
    out["learned"] = s.run(h, lambda x, c: h.split2_learned_dev(x, c, 30.0, 0.004, 12))
    for mode in (1, 3):
        h.set_mixed(mode)
        out["mixed%d" % mode] = s.run(h, _steps(h)["split2"])
    h.set_time_kind(0)
    out["relax"] = s.run(h, lambda x, c: h.relax_etdrk2_dev(x, c, 0.01, 3))
    h.set_time_kind(1)
    h.set_mixed(0)
    return out


@pytest.mark.gpu
@pytest.mark.parametrize("name", sorted(SECOND))
def test_second_init_of_a_context(cuda_ok, name):
    """The default context bound and initialised again without hprod_final_, to other sizes and back: every call
    does what it does in a fresh context, and the settings made before the second init hold."""
    refs = {}
    for key, wl in (("first", WL), ("second", SECOND[name])):
        h, orb, cic = _context(wl, new_context=True)
        try:
            refs[key] = _everything(h, wl, orb, cic)
        finally:
            h.final()
    h = None
    try:
        for key, wl in (("first", WL), ("second", SECOND[name]), ("first", WL)):
            h, orb, cic = _context(wl)
            got = _everything(h, wl, orb, cic)
            for k, v in refs[key].items():
                assert np.array_equal(got[k], v), (key, k)
        h.set_mixed(1)  # the tensor-core plans are built at once, or by the next init
        h, orb, cic = _context(WL)
        assert np.array_equal(_State(orb, cic).run(h, _steps(h)["split2"]), refs["first"]["mixed1"])
    finally:
        h.final()


@pytest.mark.gpu
def test_repeated_rhs_of_a_state_on_an_8_byte_boundary(cuda_ok):
    """The orbitals may start on any 8-byte boundary, in the first call and in every repeated one."""
    import torch
    h, orb, cic = _context()
    try:
        x = torch.from_numpy(orb.reshape(-1).view(np.float64).copy()).cuda()
        odd = torch.zeros(x.numel() + 1, dtype=torch.float64, device="cuda")
        odd[1:] = x
        assert x.data_ptr() % 16 == 0 and odd[1:].data_ptr() % 16 == 8
        c = torch.from_numpy(cic.copy()).cuda()
        y, yc = torch.empty(orb.size, dtype=torch.complex128, device="cuda"), torch.empty_like(c)
        lf = np.zeros(9)
        lf[2] = lf[8] = 0.8

        def call(t):
            y.fill_(float("nan"))
            torch.cuda.synchronize()
            h.htot_dev(1.0, lf, t.data_ptr(), c.data_ptr(), y.data_ptr(), yc.data_ptr())
            h.sync()
            return y.cpu().numpy()
        want = call(x)
        for t in (odd[1:], odd[1:], odd[1:], x, x, x, odd[1:], x):
            assert np.array_equal(call(t), want)
    finally:
        h.final()


@pytest.mark.gpu
@pytest.mark.parametrize("wl", [W.HE_SMALL, W.MIXED_SMALL], ids=lambda w: w["name"])
def test_rhs_of_changing_time_steps_is_replayed(cuda_ok, wl):
    """A time step that changes every two calls costs no capture: the calls take as long as with one time step
    (a capture and an instantiation take ten times as long as a call; the best of several rounds on both sides)."""
    import time
    import torch
    h, orb, cic = _context(wl)
    try:
        x, c = torch.from_numpy(orb.reshape(-1).copy()).cuda(), torch.from_numpy(cic.copy()).cuda()
        y, yc = torch.empty_like(x), torch.empty_like(c)
        lf = np.zeros(9)
        lf[2] = lf[8] = 0.8

        def call(dt):
            h.htot_dev(dt, lf, x.data_ptr(), c.data_ptr(), y.data_ptr(), yc.data_ptr())

        def best(dts):
            out = []
            for _ in range(7):
                h.sync()
                t = time.perf_counter()
                for dt in dts:
                    call(dt)
                h.sync()
                out.append(time.perf_counter() - t)
            return min(out)
        torch.cuda.synchronize()
        one = best([1.0] * 24)
        two = best([0.25, 0.25, 0.5, 0.5] * 6)
        assert two < 3.0 * one, (one, two)
        want = {}
        for dt in (0.25, 1.0, 0.5):
            call(dt)
            h.sync()
            want[dt] = (y.cpu().numpy(), yc.cpu().numpy())
        for dt in (0.25, 0.5):  # powers of two: exact multiples
            assert np.array_equal(want[dt][0], dt * want[1.0][0]) and np.array_equal(want[dt][1], dt * want[1.0][1])
    finally:
        h.final()
