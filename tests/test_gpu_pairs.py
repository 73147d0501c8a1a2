"""Right-hand sides over the numbers of orbital pairs, element sizes and element numbers at which the Poisson passes for
few pairs and the int2e products change their tiling, against the oracle.

Tolerance: 1e-10 relative, the suite's bound for FP64 paths against the oracle (condition of the Poisson and
one-body solves times rounding).
"""
import numpy as np
import pytest

from td1c_b200 import workloads as W

from .helpers import oracle_tables, oracle_state, rel_err

TOL = 1e-10
SHELLS = [(n, l, m) for n in range(1, 7) for l in range(min(n, 3)) for m in range(-l, l + 1)]


def _workload(nfc, nact, **kw):
    """nfc frozen and nact active orbitals (distinct shells), two active electrons."""
    orbitals = [s + (-1,) for s in SHELLS[:nfc]] + [s + (1,) for s in SHELLS[nfc:nfc + nact]]
    mtot = 2 * orbitals[-1][2] if nact == 1 else 0
    return dict(W.MIXED_SMALL, name="fc%d_act%d" % (nfc, nact), orbitals=orbitals, nela=nfc + 1, nelb=nfc + 1, mtot=mtot, smul=1,
                znuc=float(2 * nfc + 2), igauge=1, **kw)


def _parity(wl, npair=None):
    from oracle.oracle import Oracle
    from td1c_b200.hprod import HProd
    o = Oracle(wl)
    o.set_split(wl.get("split_type", 0))
    rad, ang = oracle_tables(o)
    h = HProd(wl, rad, ang)
    try:
        orb, cic = oracle_state(o)
        o.set_wfn0(orb, cic)
        h.set_wfn0(orb, cic)
        if npair:
            assert h.dims["npair"] == npair
        lf = np.zeros(9)
        lf[2], lf[5], lf[8] = 1.2, 0.1, 1.2
        ho, co = o.htot(1.0, lf, orb, cic)
        hg, cg = h.htot(1.0, lf, orb, cic)
        # (H - E) c: relative to the sums that are subtracted (with one determinant the difference is zero)
        scale = max(np.abs(co).max(), abs(h.energies()["ene_act"]) * np.abs(cic).max())
        err = rel_err(hg, ho), float(np.abs(cg - co).max() / scale)
        assert max(err) < TOL, err
        return h.debug("int2e") if h.dims["nact"] else None
    finally:
        h.final()


PAIRS = [(0, 1, 1), (1, 1, 2), (0, 2, 3), (3, 1, 4), (1, 2, 5), (2, 2, 7), (7, 1, 8), (1, 3, 9), (2, 3, 12), (1, 4, 14), (0, 5, 15),
         (15, 1, 16), (2, 4, 18)]


@pytest.mark.gpu
@pytest.mark.parametrize("nfc,nact,npair", PAIRS, ids=["%d" % p[2] for p in PAIRS])
def test_pairs(cuda_ok, nfc, nact, npair):
    """1 to 16 pairs around the tiles of four, and 18, which the staged passes take."""
    _parity(_workload(nfc, nact, ndvr=8, nfe=7, rmax=14.0, rmask=11.0), npair)


@pytest.mark.gpu
@pytest.mark.parametrize("ndvr", range(2, 26))
def test_every_element_size(cuda_ok, ndvr):
    """Every element size of the passes (one instance each), 2 pairs and 3 elements."""
    _parity(_workload(1, 1, ndvr=ndvr, nfe=3, rmax=6.0, rmask=5.0), 2)


@pytest.mark.gpu
@pytest.mark.parametrize("nfe", [1, 2, 9, 80, 81, 82, 150])
def test_element_numbers(cuda_ok, nfe):
    """No bridge, one, a full tile of eight; the depth of 80 bridges that stands in registers, and beyond it."""
    _parity(_workload(1, 2, ndvr=3, nfe=nfe, rmax=0.5 * nfe + 1.0, rmask=0.4 * nfe + 0.8), 5)


@pytest.mark.gpu
@pytest.mark.parametrize("nact", [8, 9, 10, 11])
def test_int2e_products_over_several_sets_of_warps(cuda_ok, nact):
    """Active orbitals of one m: one block of 8 to 16 tiles a side.  A set of warps holds 16 items of 2 x 4 tiles: up to
    8 tiles a side (8 orbitals) one set, then two (9 to 11 orbitals: 11, 13 and 16 tiles)."""
    orbitals = [(n, 0, 0, 1) for n in range(1, nact + 1)]
    wl = dict(W.MIXED_SMALL, name="s%d" % nact, orbitals=orbitals, nela=1, nelb=1, mtot=0, smul=1, znuc=2.0, igauge=1, ndvr=12, nfe=6,
              rmax=14.0, rmask=11.0)
    g = _parity(wl).reshape((nact,) * 4)  # [l][k][j][i]
    big = np.abs(g).max()
    assert np.abs(g - g.transpose(1, 0, 3, 2).conj()).max() < 1e-12 * big  # (ij|kl) = conj((ji|lk))
