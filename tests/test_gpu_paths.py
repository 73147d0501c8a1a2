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
