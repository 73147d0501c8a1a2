"""One-body factors: which passes a step takes (folded: one launch per cycle; else two), at every band half-width of the
bridge inverse, on grids with more bridges than one sweep of columns, and when memory is short.

Tolerance against the oracle: 1e-10 relative, the suite's bound for FP64 paths (condition of the one-body
solve times rounding).
"""
import numpy as np
import pytest

from td1c_b200 import workloads as W

from .helpers import oracle_tables, oracle_state, rel_err

TOL = 1e-10
WMAX = 8   # widest band of the folded passes
CYC = 3    # correction cycles asked for, all of them run (threshold 0)
FOLDED, TWO = 1 + CYC + 1, 2 + 2 * CYC + 1  # launches: first pass, cycles, the pass that adds the last correction


def _pair(wl):
    from oracle.oracle import Oracle
    from td1c_b200.hprod import HProd
    o = Oracle(wl)
    o.set_split(1)
    rad, ang = oracle_tables(o)
    h = HProd(wl, rad, ang)
    orb, cic = oracle_state(o)
    o.set_wfn0(orb, cic)
    h.set_wfn0(orb, cic)
    return o, h, rad, orb


def _half_width(h, rad, c, thresh):
    """Largest |row - column| of an entry of the bridge inverse of 1 + c T_l above thresh times its row's diagonal,
    over all l: Schur complement on the bridges, then the inverse of that tridiagonal matrix by substitution (which
    keeps the relative accuracy of entries far below rounding)."""
    nd, nr = rad["ndvr"], rad["nrad"] - 1
    nb = (nr + 1) // nd - 1
    tdiag = h.debug("tdiag", complex_=False).reshape(-1, nr)
    bridge = np.arange(1, nb + 1) * nd - 1
    inner = np.setdiff1d(np.arange(nr), bridge)
    far = 0
    for l in range(tdiag.shape[0]):
        band = np.asarray(rad["radk"] if l == 0 else rad["radk0"]).reshape(rad["nrad"] + 1, 2 * nd + 1)
        m = np.zeros((nr, nr), complex)
        for r in range(nr):
            for q in range(max(0, r - nd), min(nr, r + nd + 1)):
                m[r, q] = c * (tdiag[l, r] if r == q else band[r + 1, nd + q - r])
        m += np.eye(nr)
        s = m[np.ix_(bridge, bridge)] - m[np.ix_(bridge, inner)] @ np.linalg.solve(m[np.ix_(inner, inner)], m[np.ix_(inner, bridge)])
        d, up, lo = np.diag(s).copy(), np.diag(s, 1), np.diag(s, -1)
        for i in range(1, nb):
            d[i] -= lo[i - 1] / d[i - 1] * up[i - 1]
        inv = np.zeros((nb, nb), complex)
        for col in range(nb):
            y = np.zeros(nb, complex)
            y[col] = 1.0
            for i in range(col + 1, nb):
                y[i] = -lo[i - 1] / d[i - 1] * y[i - 1]
            x = 0.0
            for i in range(nb - 1, -1, -1):
                x = (y[i] - (up[i] * x if i + 1 < nb else 0.0)) / d[i]
                inv[i, col] = x
        mag = np.abs(inv.real) + np.abs(inv.imag)
        above = mag > thresh * np.diag(mag)[:, None]
        far = max(far, max(abs(i - j) for i, j in zip(*np.nonzero(above))))
    return far


def _step(h, orb, lf, dtime):
    import torch
    d = torch.from_numpy(orb.reshape(-1).copy()).cuda()
    before = h.launch_count()
    h.h1itr_dev(d.data_ptr(), lf, dtime, CYC, 0.0)
    return d.cpu().numpy(), h.launch_count() - before


def _field(wl, scale=0.01):
    lf = np.zeros(9)
    lf[2] = lf[8] = scale * (1.2 if wl["igauge"] == 1 else 0.2)
    return lf


@pytest.mark.gpu
@pytest.mark.parametrize("igauge", [0, 1])
@pytest.mark.parametrize("ndvr,nfe", [(3, 24), (7, 14), (20, 12)])
def test_every_band_half_width(cuda_ok, igauge, ndvr, nfe):
    """Step sizes whose bridge inverse has half-widths up to 8 and beyond: the folded passes up to 8, the two-launch ones beyond."""
    wl = dict(W.MIXED_SMALL, nfe=nfe, ndvr=ndvr, rmax=0.25 * nfe * ndvr, rmask=0.2 * nfe * ndvr, igauge=igauge, split_type=1)
    o, h, rad, orb = _pair(wl)
    try:
        steps = {}
        for dtime in 10.0 ** np.linspace(-4.5, 1.0, 221):
            w = _half_width(h, rad, 0.5j * dtime, 2.0 ** -64)
            if w not in steps and w == _half_width(h, rad, 0.5j * dtime, 2.0 ** -63) == _half_width(h, rad, 0.5j * dtime, 2.0 ** -65):
                steps[w] = float(dtime)
        assert set(range(4, WMAX + 1)) <= set(steps) and max(steps) > WMAX
        lf = _field(wl)
        for w, dtime in steps.items():
            want, _ = o.h1itr_prop(lf, dtime, orb, CYC, 0.0)
            got, launches = _step(h, orb, lf, dtime)
            assert launches == (FOLDED if w <= WMAX else TWO), (w, launches)
            assert rel_err(got, want) < TOL, w
    finally:
        h.final()


@pytest.mark.gpu
@pytest.mark.parametrize("ndvr,nfe,dtime,launches", [(2, 150, 1e-4, FOLDED), (3, 70, 5e-4, FOLDED), (21, 4, 0.004, TWO), (24, 3, 0.004, TWO)])
def test_grids_of_many_bridges_and_of_long_elements(cuda_ok, ndvr, nfe, dtime, launches):
    """More bridges than columns of the inverse at a time (32 for these elements), and elements that only the
    two-launch passes take."""
    wl = dict(W.MIXED_SMALL, nfe=nfe, ndvr=ndvr, rmax=0.25 * nfe * ndvr, rmask=0.2 * nfe * ndvr, split_type=1)
    o, h, _, orb = _pair(wl)
    try:
        lf = _field(wl, 1.0)
        want, _ = o.h1itr_prop(lf, dtime, orb, CYC, 0.0)
        got, n = _step(h, orb, lf, dtime)
        assert n == launches
        assert rel_err(got, want) < TOL
    finally:
        h.final()


@pytest.mark.gpu
def test_memory_of_a_factor_goes_with_the_elements(cuda_ok):
    """150 elements, 16 multipoles: a factor's arrays are 3 MB, where the whole bridge inverse alone would be 5.7."""
    import torch
    wl = dict(W.HE_SMALL, nfe=150, ndvr=2, rmax=75.0, rmask=60.0, lmax1=15, lmax2=30, split_type=1)
    o, h, _, orb = _pair(wl)
    try:
        _step(h, orb, _field(wl), 1e-4)
        torch.cuda.synchronize()
        free = torch.cuda.mem_get_info()[0]
        _step(h, orb, _field(wl), 2e-4)
        assert free - torch.cuda.mem_get_info()[0] <= 4 << 20
    finally:
        h.final()


def _take(n):
    """n bytes of device memory from the driver, or None."""
    import ctypes
    p = ctypes.c_uint64()
    f = ctypes.CDLL("libcuda.so.1").cuMemAlloc_v2
    f.argtypes = [ctypes.POINTER(ctypes.c_uint64), ctypes.c_size_t]
    return p.value if f(ctypes.byref(p), n) == 0 else None


def _give(ps):
    import ctypes
    f = ctypes.CDLL("libcuda.so.1").cuMemFree_v2
    f.argtypes = [ctypes.c_uint64]
    while ps:
        p = ps.pop()
        assert not p or f(p) == 0


@pytest.mark.gpu
def test_factor_without_memory_for_the_folded_passes(cuda_ok):
    """With room for the two-launch arrays of a factor (20 MB) but not for the folded ones beside them (45 MB), the
    two-launch passes run, and no error is left behind."""
    import torch
    wl = dict(W.HE_TDHF, nfe=60, rmax=120.0, rmask=96.0, lmax1=47, lmax2=94, split_type=1)
    from td1c_b200 import basis
    from td1c_b200.hprod import HProd
    from td1c_b200.wfn import seeded_orbitals
    rad, ang = basis.build(wl)
    h = HProd(wl, rad, ang)
    hog = []
    try:
        orb = seeded_orbitals(wl, rad["xrad"], rad["wrad"], rad["mask"])
        h.set_wfn0(orb, np.ones(1, complex))
        lf = _field(wl, 1.0)
        dtime = 0.002
        want, n = _step(h, orb, lf, dtime)
        assert n == FOLDED
        x, c = torch.from_numpy(orb.reshape(-1).copy()).cuda(), torch.ones(1, dtype=torch.complex128, device="cuda")
        _, n = _step(h, orb, lf, 500.0)  # loads the two-launch kernels: the inverse of a long step is no band
        assert n == TWO
        h.set_wfn0(orb, np.ones(1, complex))
        h.final()
        h = HProd(wl, rad, ang)
        h.set_wfn0(orb, np.ones(1, complex))
        h.h1itr_dev(x.data_ptr(), lf, 0.5 * dtime)  # the scratch of the passes
        torch.cuda.synchronize()
        d = torch.from_numpy(orb.reshape(-1).copy()).cuda()
        torch.cuda.empty_cache()
        hog.append(_take(torch.cuda.mem_get_info()[0] - (1 << 30)))
        for size in (36 << 20, 2 << 20):  # then nothing of either size is left
            while True:
                p = _take(size)
                if not p:
                    break
                hog.append(p)
        _give([hog.pop(1)])  # 36 MB
        before = h.launch_count()
        h.h1itr_dev(d.data_ptr(), lf, dtime, CYC, 0.0)
        assert h.launch_count() - before == TWO
        h.sync()
        _give(hog)
        assert rel_err(d.cpu().numpy(), want) < TOL
        h.split2_dev(x.data_ptr(), c.data_ptr(), 30.0, 0.004, 2)
        h.sync()
        _, n = _step(h, orb, lf, 2 * dtime)
        assert n == FOLDED
    finally:
        _give(hog)
        h.final()
