"""GPU paths that are chosen by size, table or call history, each against the oracle or the path beside it.

Tolerances: 1e-10 relative (the suite's bound for FP64 paths against the oracle: condition of the
Poisson and one-body solves times rounding); bitwise where two routes run the same kernels.
"""
import numpy as np
import pytest

from td1c_b200 import workloads as W

from .helpers import oracle_tables, oracle_state, rel_err

TOL = 1e-10


def _pair(wl, tables=None):
    from oracle.oracle import Oracle
    from td1c_b200.hprod import HProd
    o = Oracle(wl)
    o.set_split(wl.get("split_type", 0))
    rad, ang = oracle_tables(o)
    if tables:
        tables(ang)
    h = HProd(wl, rad, ang)
    orb, cic = oracle_state(o)
    o.set_wfn0(orb, cic)
    h.set_wfn0(orb, cic)
    return o, h, orb, cic


def _field(wl):
    lf = np.zeros(9)
    lf[2] = 1.2 if wl["igauge"] == 1 else 0.2
    lf[5], lf[8] = 0.1, lf[2]
    return lf


def _rhs_parity(wl, tables=None):
    o, h, orb, cic = _pair(wl, tables)
    try:
        lf = _field(wl)
        ho, co = o.htot(1.0, lf, orb, cic)
        hg, cg = h.htot(1.0, lf, orb, cic)
        assert rel_err(hg, ho) < TOL and rel_err(cg, co) < TOL, (rel_err(hg, ho), rel_err(cg, co))
        return hg
    finally:
        h.final()


@pytest.mark.gpu
@pytest.mark.parametrize("lmax,nlat", [(1, 0), (4, 10), (5, 11), (8, 17), (8, 20), (12, 25)])
def test_folded_and_dense_transforms(cuda_ok, lmax, nlat):
    """Odd and even theta grids, row counts around the 8-row tiles, larger grids than lmax2 + 1; then the same
    tables with one entry moved by 1e-12 of the largest, which the dense transforms take."""
    wl = W.small(dict(W.MIXED_SMALL, igauge=1), lmax1=lmax, lmax2=2 * lmax, nlat=nlat)
    folded = _rhs_parity(wl)

    def move(ang):
        t = np.array(ang["legf2"])
        t[np.argmax(np.abs(t))] *= 1.0 + 1e-12
        ang["legf2"] = t
    dense = _rhs_parity(wl, move)
    assert rel_err(folded, dense) < TOL


ORBITAL_SETS = {
    "two": ([(1, 0, 0, 1), (2, 0, 0, 1)], 1, 1, 0, 1),
    "three_m": ([(2, 1, -1, 1), (2, 1, 0, 1), (2, 1, 1, 1)], 2, 1, 1, 2),
    "five": ([(1, 0, 0, 0), (2, 0, 0, 1), (2, 1, -1, 1), (2, 1, 0, 1), (2, 1, 1, 1)], 3, 3, 0, 1),  # 15 pairs
    "d_shell": ([(1, 0, 0, -1), (2, 0, 0, 1)] + [(3, 2, m, 1) for m in (-2, -1, 0, 1, 2)], 3, 3, 0, 1),
    "two_dynamic_cores": ([(1, 0, 0, 0), (2, 0, 0, 0), (2, 1, 0, 1), (3, 1, 0, 1), (3, 0, 0, 1), (3, 2, 0, 1), (4, 0, 0, 1)], 4, 4, 0, 1),
}


@pytest.mark.gpu
@pytest.mark.parametrize("name", sorted(ORBITAL_SETS))
@pytest.mark.parametrize("nfe,ndvr", [(1, 10), (2, 7), (5, 12), (9, 8)])
def test_pair_products_and_elements(cuda_ok, name, nfe, ndvr):
    """Orbital sets with |Delta m| up to 4 and partial tiles, on one element (no bridge), two, and element
    sizes with and without unrolled rows."""
    orbitals, na, nb, mtot, smul = ORBITAL_SETS[name]
    _rhs_parity(dict(W.MIXED_SMALL, name=name, orbitals=orbitals, nela=na, nelb=nb, mtot=mtot, smul=smul, znuc=float(na + nb),
                     nfe=nfe, ndvr=ndvr, rmax=2.0 * nfe, rmask=1.6 * nfe, igauge=1))


@pytest.mark.gpu
@pytest.mark.parametrize("igauge", [0, 1])
@pytest.mark.parametrize("nfe,ndvr,dtime", [(1, 10, 0.01), (2, 7, 0.01), (9, 7, 0.005), (9, 8, 3.0), (14, 6, 0.2), (14, 6, 2.0), (6, 20, 0.004)])
def test_one_body_step_band(cuda_ok, igauge, nfe, ndvr, dtime):
    """Grids without a bridge, with one, and steps whose bridge inverse is a narrow band, a wide one, or not
    a band at all (the long steps)."""
    wl = dict(W.MIXED_SMALL, nfe=nfe, ndvr=ndvr, rmax=1.75 * nfe, rmask=1.4 * nfe, igauge=igauge, split_type=1)
    import torch
    o, h, orb, cic = _pair(wl)
    try:
        lf = _field(wl) * (0.01 if dtime > 0.1 else 1.0)  # the correction cycles converge for a short step or a weak field
        wo, no = o.h1itr_prop(lf, dtime, orb, 20, 1e-10)
        d = torch.from_numpy(orb.reshape(-1).copy()).cuda()
        ng = h.h1itr_dev(d.data_ptr(), lf, dtime, 20, 1e-10)
        assert rel_err(d.cpu().numpy(), wo) < TOL and ng == no
        wo, no = o.dpade_prod(lf, dtime, orb, 2.0, 20, 1e-10)
        d = torch.from_numpy(orb.reshape(-1).copy()).cuda()
        ng = h.dpade_dev(d.data_ptr(), lf, dtime, 2.0, 20, 1e-10)
        assert rel_err(d.cpu().numpy(), wo) < TOL and ng == no
    finally:
        h.final()


@pytest.mark.gpu
@pytest.mark.parametrize("maxcyc,thresh", [(0, 1e-10), (1, 0.0), (2, 0.0), (3, 0.0), (4, 0.0), (20, 0.0), (20, 1e-10)])
def test_correction_cycle_limits(cuda_ok, maxcyc, thresh):
    """Cycle limits below, at and above the passes that stand in a row in a captured step (threshold 0: all
    of them run), eager and captured steps alike."""
    import torch
    wl = dict(W.MIXED_SMALL, igauge=1, split_type=1)
    o, h, orb, cic = _pair(wl)
    try:
        wo, co, _ = o.split2(orb, cic, 30.0, 0.004, 3, maxcyc, thresh)
        for graph in (True, False):
            x, c = torch.from_numpy(orb.reshape(-1).copy()).cuda(), torch.from_numpy(cic.copy()).cuda()
            h.split2_dev(x.data_ptr(), c.data_ptr(), 30.0, 0.004, 3, maxcyc=maxcyc, thresh=thresh, use_graph=graph)
            h.sync()
            assert rel_err(x.cpu().numpy(), wo) < TOL and rel_err(c.cpu().numpy(), co) < TOL
    finally:
        h.final()


@pytest.mark.gpu
@pytest.mark.parametrize("wl", [W.HE_SMALL, W.NE_SMALL, W.LENGTH_SMALL], ids=lambda w: w["name"])
def test_rhs_replay(cuda_ok, wl):
    """The captured RHS on other buffers, other fields, and after changes of a setting: bitwise the eager one."""
    import torch
    o, h, orb, cic = _pair(wl)
    try:
        def call(x, c, lf, dt=1.0):
            y, yc = torch.full_like(x, float("nan")), torch.full_like(c, float("nan"))
            torch.cuda.synchronize()
            h.htot_dev(dt, lf, x.data_ptr(), c.data_ptr(), y.data_ptr(), yc.data_ptr())
            h.sync()
            return y.cpu().numpy(), yc.cpu().numpy()
        xs = [torch.from_numpy((orb * s).reshape(-1).copy()).cuda() for s in (1.0, 0.5)]
        cs = [torch.from_numpy(cic.copy()).cuda() for _ in xs]
        lfs = [_field(wl), 0.5 * _field(wl)]
        split = wl.get("split_type", 0)
        first = {}
        for k in range(2):  # alternating settings never repeat, so these are eager
            for sp in (1, split):
                h.set_split(sp)
                first[k, sp] = call(xs[k], cs[k], lfs[k])
        for sp in (1, split, 2):
            h.set_split(sp)
            for rep in range(4):
                got = call(xs[rep % 2], cs[rep % 2], lfs[rep % 2])
                if sp != 2:
                    for a, b in zip(got, first[rep % 2, sp]):
                        assert np.array_equal(a, b)
        h.set_split(split)
        for dt in (0.25, 0.25, 0.25, 1.0, 1.0, 1.0):
            a = call(xs[0], cs[0], lfs[0], dt)[0]
            assert rel_err(a, dt * first[0, split][0]) < 1e-14
    finally:
        h.final()


@pytest.mark.gpu
def test_host_call_of_a_large_state(cuda_ok):
    """A state above the size from which host copies go through the pinned ring (and not a multiple of its
    pieces): bitwise the device call, frozen-core rows zero, repeated calls included."""
    import torch
    wl = W.small(W.NE_CAS, rmax=30.0, ndvr=20, nfe=21, lmax1=19, lmax2=38, rmask=24.0)
    from td1c_b200 import basis
    from td1c_b200.hprod import HProd
    from td1c_b200.wfn import seeded_orbitals, seeded_cic
    rad, ang = basis.build(wl)
    h = HProd(wl, rad, ang)
    try:
        tb = h.ci_tables()
        orb = seeded_orbitals(wl, rad["xrad"], rad["wrad"], rad["mask"])
        cic = seeded_cic(wl, h.dims["lcic"], tb["stra"], tb["strb"], tb["detoff"], tb["afirst"], tb["acount"])
        h.set_wfn0(orb, cic)
        lf = _field(wl)
        x, c = torch.from_numpy(orb.reshape(-1).copy()).cuda(), torch.from_numpy(cic.copy()).cuda()
        y, yc = torch.empty_like(x), torch.empty_like(c)
        torch.cuda.synchronize()
        h.htot_dev(1.0, lf, x.data_ptr(), c.data_ptr(), y.data_ptr(), yc.data_ptr())
        h.sync()
        for _ in range(3):
            hw, hc = h.htot(1.0, lf, orb, cic)
            assert np.array_equal(hw.reshape(-1), y.cpu().numpy()) and np.array_equal(hc, yc.cpu().numpy())
            assert not np.any(hw[0])
    finally:
        h.final()


@pytest.mark.gpu
def test_ensemble_plan_is_reused_and_renewed(cuda_ok):
    """Ensemble steps on other buffers (the kept step graph), after a new frozen core of one job (a new graph),
    and beside another ensemble of the same jobs: each bitwise the jobs' own steps."""
    import torch
    from td1c_b200.ensemble import DeviceEnsemble
    jobs = [dict(W.HE_SMALL, dt=0.01), dict(W.NE_SMALL, dt=0.01)]
    ens = [DeviceEnsemble(jobs, relax_cycles=0) for _ in range(2)]
    try:
        def check(e, scale):
            a = [[x.clone() for x in e.orb], [x.clone() for x in e.cic]]
            for x in a[0]:
                x *= scale
            b = [[x.clone() for x in v] for v in a]
            torch.cuda.synchronize()
            e.run(3, t0=20.0, orb=a[0], cic=a[1])
            e.run_sequential(3, t0=20.0, orb=b[0], cic=b[1])
            for u, v in zip(a[0] + a[1], b[0] + b[1]):
                assert torch.equal(u, v)
        for e, s in ((ens[0], 1.0), (ens[1], 1.0), (ens[0], 0.9), (ens[0], 1.0), (ens[1], 0.8)):
            check(e, s)
        wfn = ens[0].orb[1].cpu().numpy().copy()
        ens[0].h[1].set_wfn0(0.7 * wfn, ens[0].cic[1].cpu().numpy())
        check(ens[0], 1.0)
        ens[1].final()
        check(ens[0], 0.9)
    finally:
        for e in ens:
            e.final()
