"""The framework's work, as cases that can be timed and whose results can be compared.

A case is one call (or one short propagation) that a user of the package makes:

  rhs        one right-hand side on device buffers (HProd.htot_dev): what an integrator of the user's
             own calls four times per step
  rhs_host   the drop-in hprod_htot_ on host buffers (HProd.htot), energies included: what td1c's host
             code calls
  split2     a few time steps of the default propagator (HProd.split2_dev), in FP64 or in the mixed
             form, optionally followed by the dipole that the propagation prints
  relax      cycles of the imaginary-time relaxation that makes every start state
             (HProd.relax_etdrk2_dev)
  ensemble   steps of several independent small jobs together (ensemble.DeviceEnsemble.run)

Sizes: FEDVR grids of 8 to 80 elements of 8 to 21 points, lmax1 5 to 63 (lmax2 = 2 lmax1), 1 to 9
active orbitals: the workloads of td1c_b200/workloads.py, the ensemble's job ranges, and odd sizes
between them.  Orbitals are seeded smooth functions r^(l+1) exp(-zeta r) with an admixture in the next
l, orthonormalised within each m; CI vectors are seeded, normalised and (for singlets) symmetric.
"""
import functools
import math

import numpy as np
import torch

SHELLS = [(2, 0, 0), (2, 1, -1), (2, 1, 0), (2, 1, 1), (3, 0, 0), (3, 1, -1), (3, 1, 0), (3, 1, 1), (3, 2, 0)]


def listed():
    def case(name, kind, atom, nact, nfe, ndvr, lmax, gauge=1, mixed=0, steps=0, phase=0.0, dipole=False, jobs=0):
        return dict(name=name, kind=kind, atom=atom, nact=nact, nfe=nfe, ndvr=ndvr, lmax=lmax, gauge=gauge, mixed=mixed,
                    steps=steps, phase=phase, dipole=dipole, jobs=jobs)
    return [
        # the smallest call: a small box for a quick look, where launches are all the time
        case("rhs_he_tiny", "rhs", "he", 0, 8, 8, 5),
        # He TDHF at its working size, as an integrator of the user's own calls it
        case("rhs_he", "rhs", "he", 0, 40, 20, 23),
        # Ne TD-CASSCF at its working size, the same
        case("rhs_ne", "rhs", "fc", 9, 60, 20, 47),
        # an open shell with a frozen and a dynamic core in the length gauge, on a grid of odd sizes
        case("rhs_open_length", "rhs", "open", 4, 37, 12, 21, gauge=0),
        # the drop-in call from td1c's host code: a small closed-shell box, and Ne at its working size
        case("host_core_small", "rhs_host", "dc", 4, 11, 7, 7, gauge=0),
        case("host_ne", "rhs_host", "fc", 9, 60, 20, 47),
        # a stretch of a He trajectory at the peak of the pulse, then the printed dipole
        case("split2_he", "split2", "he", 0, 40, 20, 23, steps=8, phase=0.5, dipole=True),
        # Ne steps on the rising edge of the pulse, in FP64 and in the mixed form
        case("split2_ne", "split2", "fc", 9, 60, 20, 47, steps=3, phase=0.2),
        case("split2_ne_mixed", "split2", "fc", 9, 60, 20, 47, mixed=1, steps=3, phase=0.2),
        # the largest job of the ensemble's range, at the peak
        case("split2_largest", "split2", "fc", 9, 80, 20, 63, steps=3, phase=0.5),
        # making a start state: a small active space on a middling grid
        case("relax_c", "relax", "fc", 5, 33, 20, 26, steps=3),
        # a parameter scan of small atoms stepped together
        case("ensemble_small", "ensemble", "mix", 0, 12, 20, 9, steps=4, phase=0.3, jobs=6),
    ]


def draw(rng):
    """One more case of the same ranges: sizes spread over their logarithm, odd ones among them."""
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    kind = rng.choice(["rhs", "rhs", "rhs_host", "split2", "split2", "split2", "relax", "ensemble"])
    if kind == "ensemble":
        return dict(kind=kind, atom="mix", nact=0, nfe=log_int(8, 24), ndvr=20, lmax=log_int(5, 15), gauge=1, mixed=0,
                    steps=rng.randint(1, 4), phase=rng.uniform(0.05, 0.6), dipole=False, jobs=rng.randint(2, 6))
    atom = rng.choice(["he", "fc", "fc", "fc", "dc", "open"])
    nact = 0 if atom == "he" else (rng.randint(5, 9) if atom == "fc" else rng.randint(3, 6))
    split = kind == "split2"
    return dict(kind=kind, atom=atom, nact=nact, nfe=log_int(8, 80), ndvr=rng.choice([7, 8, 10, 12, 16, 20, 20, 20]),
                lmax=log_int(5, 63), gauge=rng.choice([1, 1, 0]), mixed=rng.choice([0, 0, 1]) if split else 0,
                steps=rng.randint(1, 3) if kind in ("split2", "relax") else 0, phase=rng.uniform(0.05, 0.6) if split else 0.0,
                dipole=split and rng.random() < 0.3, jobs=0)


# ---------------------------------------------------------------------------------------------------
# workloads and seeded states
# ---------------------------------------------------------------------------------------------------
def _workload(atom, nact, nfe, ndvr, lmax, gauge, split, seed, icomp=1):
    fc, mtot, smul = (1, 0, 0, -1), 0, 1
    if atom == "he":
        orbitals, nela, nelb, z = [(1, 0, 0, 0)], 1, 1, 2.0
    elif atom == "fc":  # frozen 1s, up to eight active electrons
        orbitals = [fc] + [s + (1,) for s in SHELLS[:nact]]
        n = min(4, nact)
        nela = nelb = 1 + n
        if n == nact:  # one determinant: its M
            mtot = 2 * sum(s[2] for s in SHELLS[:nact])
        z = float(2 * nela)
    else:  # frozen 1s, dynamic 2s, active 2p 3s 3p; "open": one more alpha than beta electron, M = 1
        orbitals = [fc, (2, 0, 0, 0)] + [s + (1,) for s in SHELLS[1:1 + nact]]
        n = max(1, nact // 2 - 1)
        nela, nelb = 2 + n + (atom == "open"), 2 + n
        if atom == "open":
            mtot, smul = 1, 2
        z = float(nela + nelb)
    rmax = 2.0 * nfe * ndvr / 20.0
    return dict(name="%s_%d" % (atom, nact), znuc=z, rmin=0.0, rmax=rmax, ndvr=ndvr, nfe=nfe, lmax1=lmax, lmax2=2 * lmax, nlat=0,
                orbitals=orbitals, nela=nela, nelb=nelb, mtot=mtot, smul=smul, igauge=gauge, icomp=icomp, rmask=0.8 * rmax,
                mask_cos_order=4.0, fint=5.0e14 if gauge == 1 else 1.0e14, wlen=800.0, numcyc=3.0, cep=0.0, dt=0.004,
                split_type=split, seed=seed)


def _workloads(case, seed):
    """The workloads of a case: one, or the jobs of an ensemble (drawn from the case's sizes and the seed's pulses)."""
    if case["kind"] != "ensemble":
        split = 0 if case["kind"] in ("rhs", "rhs_host") else 1
        return [_workload(case["atom"], case["nact"], case["nfe"], case["ndvr"], case["lmax"], case["gauge"], split, seed,
                          icomp=0 if case["kind"] == "relax" else 1)]
    shape, pulse, out = np.random.RandomState(case["jobs"] * 1000 + case["nfe"]), np.random.RandomState(seed % (1 << 31)), []
    for j in range(case["jobs"]):
        nact, nfe = int(shape.randint(0, 6)), int(shape.randint(max(6, case["nfe"] * 2 // 3), case["nfe"] + 1))
        lmax = int(shape.randint(max(4, case["lmax"] * 2 // 3), case["lmax"] + 1))
        wl = _workload("fc" if nact >= 2 else "he", nact, nfe, case["ndvr"], lmax, 1, 1, seed + j)
        out.append(dict(wl, fint=float(10.0 ** pulse.uniform(13.0, 14.7)), wlen=float(pulse.uniform(400, 1600)),
                        cep=float(pulse.uniform(0, 360))))
    return out


def _start_time(wl, phase):
    return phase * wl["numcyc"] * 2.0 * math.pi / (1239.84190 / (wl["wlen"] * 27.2113845))


def _fields(wl, seed):
    """lfield of a single right-hand side: A and E of a strong pulse."""
    u = np.random.RandomState(seed % (1 << 31)).uniform(0.5, 1.0, 2)
    lf = np.zeros(9)
    if wl["igauge"] == 1:
        lf[2] = lf[8] = 2.0 * u[0]
        lf[5] = 0.1 * u[1]
    else:
        lf[2] = lf[5] = 0.1 * u[0]
    return lf


def _orbitals(wl, grid):
    rng = np.random.Generator(np.random.Philox(wl["seed"]))
    r, sw, mask = grid["x"], np.sqrt(grid["w"]), grid["mask"]
    nr, nl, n = len(r), wl["lmax1"] + 1, len(wl["orbitals"])
    orb = np.zeros((n, nl, nr), dtype=np.complex128)
    for f, (sh, l, m, _t) in enumerate(wl["orbitals"]):
        g = rng.standard_normal((6, 2)) @ np.array([1.0, 1.0j])
        z = wl["znuc"] / sh * np.array([1.0, 0.75, 0.5, 0.35])
        orb[f, l] = (g[:4, None] * np.exp(-z[:, None] * r)).sum(0) * r ** (l + 1) * sw * mask
        if l + 1 < nl:  # the next channel, so that every l of the path is at work
            orb[f, l + 1] = 0.05 * g[4] * np.exp(-z[0] * r) * r ** (l + 2) * sw * mask
        for _ in range(2):
            for k in range(f):
                if wl["orbitals"][k][2] == m:
                    orb[f] -= orb[k] * np.vdot(orb[k], orb[f])
            orb[f] /= np.linalg.norm(orb[f])
    return orb


def _strings(wl):
    """Alpha and beta strings sorted by (M, mask) and the determinants (alpha, beta) in vector order."""
    act = [o for o in wl["orbitals"] if o[3] == 1]
    ncore = len(wl["orbitals"]) - len(act)

    def strings(nel):
        s = [b for b in range(1 << len(act)) if bin(b).count("1") == nel]
        return sorted((sum(o[2] for k, o in enumerate(act) if b >> k & 1), b) for b in s)
    a, b = strings(wl["nela"] - ncore), strings(wl["nelb"] - ncore)
    dets = [(i, j) for j, (mb, _) in enumerate(b) for i, (ma, _) in enumerate(a) if ma + mb == wl["mtot"]]
    return [x[1] for x in a], [x[1] for x in b], np.array(dets)


def _ci(wl):
    if not any(o[3] == 1 for o in wl["orbitals"]):
        return np.ones(1, dtype=np.complex128)
    a, b, dets = _strings(wl)
    rng = np.random.Generator(np.random.Philox(wl["seed"] + 1000))
    c = np.zeros((len(a), len(b)), dtype=np.complex128)
    c[dets[:, 0], dets[:, 1]] = rng.standard_normal((len(dets), 2)) @ np.array([1.0, 1.0j])
    if wl["nela"] == wl["nelb"]:
        c = 0.5 * (c + c.T)
    c = c[dets[:, 0], dets[:, 1]]
    return c / np.linalg.norm(c)


# ---------------------------------------------------------------------------------------------------
# what a user's program holds, and one pass
# ---------------------------------------------------------------------------------------------------
@functools.lru_cache(maxsize=16)
def _tables(nfe, ndvr, lmax, rmax, rmask, order, mmax):
    from td1c_b200 import basis
    return basis.fedvr(0.0, rmax, ndvr, nfe, rmask, order), basis.sph(lmax, 2 * lmax, mmax, 2 * mmax)


def _tables_of(wl):
    mmax = max(abs(o[2]) for o in wl["orbitals"])
    return _tables(wl["nfe"], wl["ndvr"], wl["lmax1"], wl["rmax"], wl["rmask"], wl["mask_cos_order"], mmax)


class _State:
    """A context with its bound tables, the start state on the device and the working copy."""

    def __init__(self, case, seed):
        from td1c_b200.hprod import HProd
        self.case, self.h, self.ens = case, None, None
        wls = _workloads(case, seed)
        states = [(_orbitals(wl, _grid(wl)), _ci(wl)) for wl in wls]
        if case["kind"] == "ensemble":
            from td1c_b200.ensemble import DeviceEnsemble
            it = iter(states)
            self.ens = DeviceEnsemble(wls, tables=_tables_of, state=lambda h, wl: next(it), relax_cycles=0)
            self.start = [x.clone() for x in self.ens.orb + self.ens.cic]
            self.t0 = [_start_time(wl, case["phase"]) for wl in wls]
            return
        wl, (orb, cic) = wls[0], states[0]
        self.wl, self.h = wl, HProd(wl, *_tables_of(wl), new_context=True)
        self.h.set_wfn0(orb, cic)
        self.lf = _fields(wl, seed)
        if case["kind"] == "rhs_host":
            self.orb, self.cic = orb, cic
            return
        self.y0, self.c0 = torch.from_numpy(orb).cuda(), torch.from_numpy(cic).cuda()
        self.y, self.c = torch.empty_like(self.y0), torch.empty_like(self.c0)
        if case["mixed"]:
            self.h.set_mixed(case["mixed"])
        self.t0 = _start_time(wl, case["phase"])
        self.stream = torch.cuda.ExternalStream(self.h.stream())

    def __del__(self):
        try:
            for h in ([self.h] if self.h else []) + (self.ens.h if self.ens else []):
                h.final()
        except Exception:
            pass


def prepare(case, seed):
    return _State(case, int(seed))


def run(s):
    case = s.case
    if case["kind"] == "ensemble":
        for x, x0 in zip(s.ens.orb + s.ens.cic, s.start):
            x.copy_(x0)
        s.ens.run(case["steps"], t0=s.t0)
        return {"orb": list(s.ens.orb), "cic": list(s.ens.cic)}
    if case["kind"] == "rhs_host":
        hw, hc = s.h.htot(1.0, s.lf, s.orb, s.cic)
        return {"hwfn": hw, "hcic": hc, "energies": np.array(list(s.h.energies().values()))}
    if case["kind"] == "rhs":
        s.h.htot_dev(1.0, s.lf, s.y0.data_ptr(), s.c0.data_ptr(), s.y.data_ptr(), s.c.data_ptr())
        return {"hwfn": s.y, "hcic": s.c}
    with torch.cuda.stream(s.stream):
        s.y.copy_(s.y0)
        s.c.copy_(s.c0)
    if case["kind"] == "relax":
        ene = s.h.relax_etdrk2_dev(s.y.data_ptr(), s.c.data_ptr(), 0.01, case["steps"])
        return {"orb": s.y, "cic": s.c, "energy": ene}
    s.h.split2_dev(s.y.data_ptr(), s.c.data_ptr(), s.t0, s.wl["dt"], case["steps"])
    out = {"orb": s.y, "cic": s.c}
    if case["dipole"]:
        out["dipole"] = s.h.dipole_dev(s.y.data_ptr(), s.c.data_ptr())
    return out


def work(case):
    """Bytes: the state in and out of every right-hand side and one-body solve.  Operations: the
    contractions of a right-hand side, four of them per split step and three per relaxation cycle (one
    is the energy's), and the one-body solves element by element."""
    byt = flo = 0.0
    for wl in _workloads(case, 1):
        nr, l1, l2 = wl["nfe"] * wl["ndvr"] - 1, wl["lmax1"] + 1, wl["lmax2"] + 1
        orbs = wl["orbitals"]
        nf, nc = len(orbs), sum(o[3] == -1 for o in orbs)
        na, nd = sum(o[3] == 1 for o in orbs), len(orbs) - nc
        npair = nd * (nd + 1) // 2 + nd * nc
        m = [o[2] for o in orbs if o[3] == 1]
        quads = sum(1 for i in range(na) for j in range(i + 1) for k in range(na) for q in range(na) if m[i] + m[k] == m[j] + m[q])
        state = 16.0 * nr * l1 * nf
        rhs_b = 2 * state
        # transforms between l and theta need half of a dense product each: the functions have a parity
        rhs_f = 2.0 * nr * (npair * 2 * l2 * l2 + 3 * nd * l1 * l2) + 8.0 * quads * nr * 2 * l2 + 4.0 * nr * npair * l2 * wl["ndvr"]
        rhs_f += 8.0 * nr * l1 * nd * wl["ndvr"] * 2
        n = {"rhs": 1, "rhs_host": 1, "split2": 4 * case["steps"], "ensemble": 4 * case["steps"], "relax": 3 * case["steps"]}[case["kind"]]
        half = {"split2": 2 * case["steps"], "ensemble": 2 * case["steps"], "relax": 2 * case["steps"]}.get(case["kind"], 0)
        byt += n * rhs_b + half * 2 * state
        flo += n * rhs_f + half * 3 * 8.0 * nr * l1 * nd * wl["ndvr"] * 3
    return {"bytes": byt, "flops": flo}


# ---------------------------------------------------------------------------------------------------
# the same results in 64 bits by dense linear algebra, from the definitions
# ---------------------------------------------------------------------------------------------------
def _legendre(n, x):
    """P_n and P_n' at x."""
    p0, p1 = np.ones_like(x), x
    for k in range(2, n + 1):
        p0, p1 = p1, ((2 * k - 1) * x * p1 - (k - 1) * p0) / k
    return p1, n * (p0 - x * p1) / np.where(np.abs(x) == 1, 1, 1 - x * x)


@functools.lru_cache(maxsize=16)
def _lobatto(n):
    k = np.arange(1, n - 1)
    off = np.sqrt(k * (k + 2.0) / ((2 * k + 1.0) * (2 * k + 3.0)))  # Jacobi matrix of the (1, 1) weight
    x = np.linalg.eigvalsh(np.diag(off, 1) + np.diag(off, -1)).astype(np.longdouble)
    for _ in range(4):  # zeros of P_n' by Newton's method: (1 - x^2) P_n'' = 2 x P_n' - n (n + 1) P_n
        p, d = _legendre(n, x)
        x = x - d * (1 - x * x) / (2 * x * d - n * (n + 1) * p)
    x = np.concatenate([[-1], x, [1]]).astype(np.longdouble)
    return x, 2 / (n * (n + 1) * _legendre(n, x)[0] ** 2)


def _grid(wl):
    """Points (without the ends), weights and mask of the FEDVR grid."""
    n, ne = wl["ndvr"], wl["nfe"]
    x01, w01 = _lobatto(n)
    h = wl["rmax"] / ne
    x = np.concatenate([(h * e + h / 2 * (x01[:-1] + 1)) for e in range(ne)])
    w = np.zeros(n * ne + 1, dtype=np.longdouble)
    for e in range(ne):
        w[n * e: n * e + n + 1] += w01 * (h / 2)
    x, w = x[1:].astype(float), w[1:-1].astype(float)
    arg = np.clip((x - wl["rmask"]) / (wl["rmax"] - wl["rmask"]), 0.0, 1.0)
    return dict(x=x, w=w, mask=np.cos(0.5 * np.pi * arg) ** (1.0 / wl["mask_cos_order"]))


def _derivative(n):
    """f_m'(x_k) of the Lobatto shape functions on [-1, 1]."""
    x, w = _lobatto(n)
    d = np.zeros((n + 1, n + 1), dtype=np.longdouble)
    for m in range(n + 1):
        for k in range(n + 1):
            if m != k:
                sel = [q for q in range(n + 1) if q not in (m, k)]
                d[m, k] = np.prod((x[k] - x[sel]) / (x[m] - x[sel])) / (x[m] - x[k])
    d[0, 0], d[n, n] = -0.5 / w[0], 0.5 / w[n]
    return d


def _theta_tables(lmax, mmax):
    """Gauss-Legendre nodes and weights and normalised P_l^m, m = 0 .. mmax: [m][l][theta]."""
    x, _ = np.polynomial.legendre.leggauss(lmax + 1)
    x = x.astype(np.longdouble)
    for _i in range(3):
        p, d = _legendre(lmax + 1, x)
        x = x - p / d
    w = 2 / ((1 - x * x) * _legendre(lmax + 1, x)[1] ** 2)
    t = np.zeros((mmax + 1, lmax + 1, lmax + 1), dtype=np.longdouble)
    top = np.full(lmax + 1, np.sqrt(np.longdouble(0.5)))
    for m in range(mmax + 1):
        if m > 0:
            top = -np.sqrt(np.longdouble(2 * m + 1) / (2 * m)) * np.sqrt(1 - x * x) * top
        t[m, m] = top
        for l in range(m + 1, lmax + 1):
            f = np.sqrt((4 * np.longdouble(l) ** 2 - 1) / (np.longdouble(l) ** 2 - m * m))
            g = np.sqrt((np.longdouble(l - 1) ** 2 - m * m) / (4 * np.longdouble(l - 1) ** 2 - 1)) if l - 2 >= m else 0
            t[m, l] = f * (x * t[m, l - 1] - (g * t[m, l - 2] if l - 2 >= m else 0))
    return x.astype(float), w, t


def _rc(a, z):
    """Real matrix times complex."""
    return torch.complex(a @ z.real, a @ z.imag)


class _Model:
    def __init__(self, wl):
        self.wl = wl
        dev = self.dev = "cuda" if torch.cuda.is_available() else "cpu"
        T = lambda v: torch.as_tensor(np.asarray(v, dtype=float), device=dev)  # noqa: E731
        g = _grid(wl)
        n, ne, x, w = wl["ndvr"], wl["nfe"], g["x"], g["w"]
        nr = self.nr = len(x)
        self.orbitals, self.m = wl["orbitals"], [o[2] for o in wl["orbitals"]]
        types = [o[3] for o in self.orbitals]
        self.nf, self.nfc, self.nc = len(types), types.count(-1), types.count(-1) + types.count(0)
        self.na = self.nf - self.nc
        self.l1, self.l2 = wl["lmax1"] + 1, wl["lmax2"] + 1
        # radial matrices
        d, w01 = _derivative(n), _lobatto(n)[1]
        h2 = np.longdouble(wl["rmax"]) / ne / 2
        kin = np.zeros((2, nr + 2, nr + 2), dtype=np.longdouble)  # kinetic: l = 0, and without the point r = 0
        der = np.zeros((nr + 2, nr + 2), dtype=np.longdouble)
        for e in range(ne):
            sl = slice(n * e, n * e + n + 1)
            kin[0][sl, sl] += (d * w01) @ d.T / h2 / 2
            kin[1][sl, sl] += (d * np.where((e == 0) & (np.arange(n + 1) == 0), 0, w01)) @ d.T / h2 / 2
            der[sl, sl] += w01[:, None] * d.T
        sq = np.sqrt(np.outer(w, w))
        kin, der = kin[:, 1:-1, 1:-1] / sq, der[1:-1, 1:-1] / sq
        self.der, self.x, self.mask = T(der), T(x), T(np.where(x > wl["rmask"], g["mask"], 1.0))
        ls = np.arange(self.l1)
        self.t_bare = torch.stack([T(kin[0 if l == 0 else 1]) for l in ls])
        diag = -wl["znuc"] / x[None] + ls[:, None] * (ls[:, None] + 1) * 0.5 / x[None] ** 2
        self.t_bare += torch.diag_embed(T(diag))
        # angular tables
        mmax = max(abs(v) for v in self.m)
        cost, wt, tab = _theta_tables(self.l2 - 1, 2 * mmax)
        self.cost = T(cost)
        self.f2, self.b2 = [T(t.T) for t in tab], [T(t * wt) for t in tab]  # to theta, from theta
        self.f1, self.b1 = [T(t[:self.l1].T) for t in tab[:mmax + 1]], [T(t[:self.l1] * wt) for t in tab[:mmax + 1]]
        self.alpha = [T([math.sqrt(((l + 1.0) ** 2 - m * m) / ((2 * l + 1.0) * (2 * l + 3.0))) if l >= abs(m) else 0.0
                         for l in ls]) for m in self.m]
        # Poisson: A_l = l (l + 1) / r^2 + 2 kinetic, and its boundary term
        l = np.arange(self.l2, dtype=np.longdouble)[:, None]
        xl = np.asarray(x, dtype=np.longdouble)[None] / wl["rmax"]
        sw = np.sqrt(w)[None]
        self.rho_x = T((2 * l + 1) / (x * sw) / (2 * np.pi))
        self.rho_t, self.t_x = T(xl ** l / (2 * np.pi)), T(xl ** (l + 1) * sw)  # (r / rmax)^l keeps the products in range
        self.v_x = T(4 * np.pi / (2 * l + 1) / (x * sw))
        k2 = T(2 * kin[0])
        self.chol = torch.stack([torch.linalg.cholesky(k2 + torch.diag(T(float(q * (q + 1)) / x ** 2))) for q in range(self.l2)])
        self.lu = {}
        # one-particle excitations a+_p a_q on the strings
        if self.na:
            sa, sb, dets = _strings(wl)
            self.dets = torch.as_tensor(dets, device=dev)
            self.ea, self.eb = self._excitations(sa), self._excitations(sb)

    def _excitations(self, strings):
        at, n = {s: k for k, s in enumerate(strings)}, self.na
        e = torch.zeros((n, n, len(strings), len(strings)), dtype=torch.complex128)
        for k, s in enumerate(strings):
            for q in range(n):
                if s >> q & 1:
                    for p in range(n):
                        t = s & ~(1 << q)
                        if not t >> p & 1:
                            lo, hi = min(p, q), max(p, q)
                            e[p, q, at[t | 1 << p], k] = -1.0 if bin(t >> lo + 1 & (1 << max(0, hi - lo - 1)) - 1).count("1") & 1 else 1.0
        return e.to(self.dev)

    def poisson(self, rho):
        """Potentials of radial densities rho[pair][l][r]."""
        b = (rho * self.rho_x).permute(1, 2, 0)
        y = torch.cholesky_solve(torch.cat([b.real, b.imag], 2), self.chol)
        y = torch.complex(y[..., :rho.shape[0]], y[..., rho.shape[0]:]).permute(2, 0, 1)
        t = (rho * self.rho_t).sum(-1, keepdim=True)
        return (y + t * self.t_x) * self.v_x

    def set_wfn0(self, orb):
        self.orb0 = torch.as_tensor(orb, device=self.dev)
        self.t, self.e_fc = self.t_bare.clone(), 0.0
        if not self.nfc:
            return
        og = torch.stack([_rc(self.f1[abs(self.m[f])], self.orb0[f]) for f in range(self.nfc)])
        fc = torch.stack([_rc(self.b1[abs(self.m[f])], og[f]) for f in range(self.nfc)])
        rho = torch.zeros((1, self.l2, self.nr), dtype=torch.complex128, device=self.dev)
        for f in range(self.nfc):
            l = self.orbitals[f][1]
            rho[0, 0] += (2 * l + 1) * self.orb0[f, l].abs() ** 2
        j = self.poisson(rho)[0, 0].real
        e, gg = 0.0, [j * o for o in og]
        for i in range(self.nfc):
            e += 2 * torch.vdot(fc[i].reshape(-1), self.kinetic(fc[i:i + 1], self.t_bare)[0].reshape(-1)).real
            for k in range(self.nfc):
                mm = abs(self.m[i] - self.m[k])
                w = _rc(self.f2[mm], self.poisson(_rc(self.b2[mm], og[k].conj() * og[i])[None])[0])
                gg[i] = gg[i] - w * og[k]
            e += torch.vdot(fc[i].reshape(-1), _rc(self.b1[abs(self.m[i])], gg[i]).reshape(-1)).real
        self.e_fc = float(e)
        self.t = self.t + torch.diag(j)

    def kinetic(self, o, t):
        z = o.permute(1, 2, 0)
        return _rc(t, z).permute(2, 0, 1)

    def laser(self, zf, o, length, which):
        h = torch.zeros_like(o)
        for f in which:
            a = self.alpha[f][:-1, None]
            lo, up = o[f, :-1], o[f, 1:]
            if length:
                h[f, :-1] += zf * a * self.x * up
                h[f, 1:] += zf * a * self.x * lo
            else:
                dw = _rc(self.der, o[f].T).T
                c = torch.arange(1, self.l1, device=self.dev, dtype=torch.float64)[:, None] / self.x
                h[f, :-1] += -1j * zf * a * (dw[1:] + c * up)
                h[f, 1:] += -1j * zf * a * (dw[:-1] - c * lo)
        return h

    def reg_inverse(self, a):
        d, u = torch.linalg.eigh(a)
        return (u * (d / (d * d + 1e-15))) @ u.conj().T

    def htot(self, dtime, lf, wfn, cic, split):
        nf, nfc, nc, na, m = self.nf, self.nfc, self.nc, self.na, self.m
        length, icomp = self.wl["igauge"] == 0, self.wl["icomp"]
        orb = wfn.clone()
        og = [_rc(self.f1[abs(m[f])], (self.orb0 if f < nfc else orb)[f]) for f in range(nf)]
        for f in range(nfc):
            if length:
                orb[f] = self.orb0[f]
            else:
                og[f] = og[f] * torch.exp(-1j * lf[8] * self.cost[:, None] * self.x)
                orb[f] = _rc(self.b1[abs(m[f])], og[f])
        og = torch.stack(og)
        # density matrices
        if na:
            c = torch.zeros((self.ea.shape[2], self.eb.shape[2]), dtype=torch.complex128, device=self.dev)
            c[self.dets[:, 0], self.dets[:, 1]] = cic
            dv = self.ea @ c + c @ self.eb.transpose(-1, -2)
            flat = dv.reshape(na * na, -1)
            den1 = (flat @ c.reshape(-1).conj()).reshape(na, na).T.contiguous()  # den1[x, y] = <E_yx>
            den2 = torch.einsum("ak,bk->ab", flat.conj(), flat).reshape(na, na, na, na).transpose(2, 3).clone()  # [p, q, r, s]
            for p in range(na):
                den2[p, :, :, p] -= den1.T
            ma = torch.tensor(m[nc:], device=self.dev)
            rden = self.reg_inverse(den1)
        # one-body part
        h0 = self.kinetic(orb, self.t)
        h1 = self.laser(lf[2], orb, length, range(nf))
        if nfc and not length:
            h1 += self.laser(lf[5], orb, True, range(nfc))
        # pair densities and potentials
        g, v2 = torch.zeros_like(orb), torch.zeros_like(orb)
        pairs = [(a, b) for b in range(nf) for a in range(max(b, nfc), nf)]
        at = {p: k for k, p in enumerate(pairs)}
        rho = torch.stack([_rc(self.b2[abs(m[b] - m[a])], og[a].conj() * og[b]) for a, b in pairs])
        v = self.poisson(rho)
        pot = torch.stack([_rc(self.f2[abs(m[b] - m[a])], v[k]) for k, (a, b) in enumerate(pairs)])
        W = lambda a, b: pot[at[a, b]] if (a, b) in at else pot[at[b, a]].conj()  # noqa: E731
        gg, vg = torch.zeros_like(og), torch.zeros_like(og)
        for i in range(nfc, nf):
            for j in range(nfc):
                gg[i] -= W(j, i) * og[j]
            for j in range(nfc, nc):
                gg[i] += 2 * W(j, j) * og[i] - W(j, i) * og[j]
        act = range(nc, nf)
        if na and nc > nfc:
            coul = sum(den1[k - nc, j - nc] * W(j, k) for j in act for k in act)
            for i in range(nfc, nc):
                vg[i] += coul * og[i]
                for j in act:
                    wd = sum(-0.5 * den1[k - nc, j - nc] * og[k] for k in act if m[k] == m[j])
                    vg[i] += wd * W(j, i)
        if na and self.wl["nela"] + self.wl["nelb"] - 2 * nc >= 2:
            allw = torch.stack([W(k, l) for k in act for l in act]).reshape(na * na, -1)
            rule = ma[:, None, None, None] + ma[None, None, :, None] == ma[None, :, None, None] + ma[None, None, None, :]  # i j k l
            d2 = den2.permute(1, 0, 3, 2) * rule  # [i, j, k, l] = den2(j, i, l, k)
            tw = torch.zeros_like(og[nc:])
            for i in range(na):
                d2v = (d2[i].reshape(na, na * na) @ allw).reshape(na, *og.shape[1:])
                tw[i] = (d2v * og[nc:]).sum(0)
            same = (ma[:, None] == ma[None, :])
            vg[nc:] = torch.einsum("ik,i...->k...", rden * same, tw)
        for i in range(nfc, nf):
            g[i], v2[i] = _rc(self.b1[abs(m[i])], gg[i]), _rc(self.b1[abs(m[i])], vg[i])
        # integrals and energies
        dot = lambda a, b: torch.einsum("ilr,jlr->ij", a.conj(), b)  # noqa: E731
        eq = torch.tensor([[a == b for b in m] for a in m], device=self.dev)
        f01 = dot(orb, g + h1 + h0) * eq
        fock = f01 + dot(orb, v2) * eq
        e_dc = float(sum((f01[i, i] + torch.vdot(orb[i].reshape(-1), (h0 + h1)[i].reshape(-1))).real for i in range(nfc, nc)))
        e_act = 0.0
        if na:
            up = torch.triu(f01[nc:, nc:])
            int1 = up + torch.triu(up, 1).conj().T
            r = torch.stack([rho[at[i, j]] if i >= j else torch.zeros_like(rho[0]) for i in act for j in act]).reshape(na * na, -1)
            vv = torch.stack([v[at[k, l]] if k >= l else v[at[l, k]].conj() for k in act for l in act]).reshape(na * na, -1)
            int2 = (r @ vv.T).reshape(na, na, na, na)
            rule = ma[:, None, None, None] + ma[None, None, :, None] == ma[None, :, None, None] + ma[None, None, None, :]
            int2 = int2 * rule
            low = torch.ones((na, na), dtype=torch.bool, device=self.dev).tril()[:, :, None, None]
            int2 = torch.where(low, int2, int2.permute(1, 0, 3, 2).conj())
            e_act = float(((int1 * den1.T).sum() + 0.5 * (int2 * den2.permute(1, 0, 3, 2)).sum()).real)
        # constraint matrix
        tf = dtime if icomp == 0 else 1j * dtime
        X = torch.zeros((nf, nf), dtype=torch.complex128, device=self.dev)
        X[nfc:nc, nfc:nc], X[nc:, nc:] = fock[nfc:nc, nfc:nc], fock[nc:, nc:]
        X[:nfc, nfc:] = (dot(h0 + h1, orb) * eq + dot(orb, g + v2) * eq)[:nfc, nfc:]
        if na and nc > nfc:
            X[nc:, nfc:nc], X[nfc:nc, nc:] = fock[nc:, nfc:nc], fock[nfc:nc, nc:]
        X = X * tf
        if na and nc > nfc and 2 * na != self.wl["nela"] + self.wl["nelb"] - 2 * nc:
            hole = self.reg_inverse(2 * torch.eye(na, device=self.dev, dtype=torch.complex128) - den1)
            b = -tf * (hole @ (2 * fock[nc:, nfc:nc] - den1 @ fock[nfc:nc, nc:].conj().T))
            X[nc:, nfc:nc] += b
            X[nfc:nc, nc:] -= b.conj().T
        h = g + v2
        if split != 1:
            h = h + h1
        if split == 0:
            h = h + h0
        hw = -tf * h + torch.einsum("jlr,ji->ilr", orb, X * eq)
        hw[:nfc] = 0
        hc = torch.zeros_like(cic)
        if na:
            k1 = int1 - 0.5 * torch.einsum("prrq->pq", int2)
            sig = torch.einsum("rs,rsab->ab", k1, dv)
            tv = (int2.reshape(na * na, na * na) @ flat).reshape(dv.shape)
            sig = sig + 0.5 * ((self.ea @ tv).sum((0, 1)) + (tv @ self.eb.transpose(-1, -2)).sum((0, 1)))
            hc = -tf * (sig[self.dets[:, 0], self.dets[:, 1]] - e_act * cic)
        e = [self.e_fc, e_dc, self.e_fc + e_dc, e_act, self.e_fc + e_dc + e_act]
        return hw, hc, e

    # one-body propagation: (1 + c T)^-1 with the laser by correction cycles
    def inverse(self, c, o):
        if c not in self.lu:
            eye = torch.eye(self.nr, device=self.dev, dtype=torch.complex128)
            self.lu = {k: v for k, v in list(self.lu.items())[-1:]}
            self.lu[c] = [torch.linalg.lu_factor(eye + c * self.t[l]) for l in range(self.l1)]
        out = torch.zeros_like(o)
        for l in range(self.l1):
            out[:, l] = torch.linalg.lu_solve(*self.lu[c][l], o[:, l].T).T
        return out

    def cycles(self, c, lf, o, first):
        length, dyn = self.wl["igauge"] == 0, range(self.nfc, self.nf)
        o = self.inverse(c, o)
        total = o.clone()
        for _ in range(20):
            if math.sqrt(float((o[first:].abs() ** 2).sum()) / self.nf) < 1e-10:
                break
            o = self.inverse(c, -c * self.laser(lf[2], o, length, dyn))
            total = total + o
        return total

    def crank_nicolson(self, lf, dt, y):
        c = 0.5j * dt
        h = self.kinetic(y, self.t) + self.laser(lf[2], y, self.wl["igauge"] == 0, range(self.nf))
        o = y.clone()
        o[self.nfc:] -= c * h[self.nfc:]
        out = self.cycles(c, lf, o, 0)
        out[:self.nfc] = y[:self.nfc]
        return out

    def pade(self, lf, dt, y):
        out = self.cycles(dt / 2.0, lf, y, self.nfc)
        out[:self.nfc] = y[:self.nfc]
        return out

    def field(self, t):
        wl = self.wl
        om = 1239.84190 / (wl["wlen"] * 27.2113845)
        f0, cep = math.sqrt(wl["fint"] / 3.50944506E+16), wl["cep"] / 180.0 * math.pi
        last = wl["numcyc"] * 2 * math.pi / om
        env = lambda s: math.sin(math.pi * s / last) ** 2 * math.sin(om * s + cep) if 0 < s < last else 0.0  # noqa: E731
        lf = [0.0] * 9
        if wl["igauge"] == 0:
            lf[2] = lf[5] = f0 * env(t)
            lf[8] = f0 / om * env(t)
        else:
            d = 2 * math.pi / (1239.84190 / (800.0 * 27.2113845)) / 100000.0
            lf[2] = lf[8] = f0 / om * env(t)
            lf[5] = -f0 / om * sum(k * (env(t + j * d) - env(t - j * d)) for j, k in ((1, 0.75), (2, -0.15), (3, 1 / 60))) / d
        return lf

    def split2(self, y, c, t0, steps):
        dt = self.wl["dt"]
        for s in range(steps):
            t = t0 + dt * s
            y = self.crank_nicolson(self.field(t + 0.25 * dt), 0.5 * dt, y)
            y0, c0, yt, ct = y, c, y, c
            for node, weight, nxt in ((0, 1 / 6, 0.5), (0.5, 1 / 3, 0.5), (0.5, 1 / 3, 1.0), (1.0, 1 / 6, 0.0)):
                ky, kc, _ = self.htot(1.0, self.field(t + node * dt), yt, ct, 1)
                y, c = y + dt * weight * ky, c + dt * weight * kc
                yt, ct = y0 + dt * nxt * ky, c0 + dt * nxt * kc
            y = self.crank_nicolson(self.field(t + 0.75 * dt), 0.5 * dt, y)
            y = torch.cat([y[:self.nfc], y[self.nfc:] * self.mask])
        return y, c

    def relax(self, y, c, dt, cycles):
        lf, ene = [0.0] * 9, []
        for _ in range(cycles):
            hy, hc, e = self.htot(1.0, lf, y, c, 1)
            ene.append(e[4])
            w1y, w1c = self.pade(lf, dt, 2 * y + dt * hy) - y, c + dt * hc
            ky, kc, _e = self.htot(1.0, lf, w1y, w1c, 1)
            y, c = w1y + self.pade(lf, dt, (ky - hy) * (0.5 * dt)), w1c + (kc - hc) * (0.5 * dt)
            c = c / torch.linalg.norm(c)
            for i in range(self.nfc, self.nf):
                for j in range(i):
                    if self.m[j] == self.m[i]:
                        y[i] = y[i] - y[j] * torch.vdot(y[j].reshape(-1), y[i].reshape(-1))
                y[i] = y[i] / torch.linalg.norm(y[i])
        return y, c, ene

    def dipole(self, y, c):
        z = self.laser(1.0, y, True, range(self.nf))
        e = torch.einsum("ilr,jlr->ij", y.conj(), z)
        d = 2 * sum(e[f, f].real for f in range(self.nc))
        if self.na:
            cm = torch.zeros((self.ea.shape[2], self.eb.shape[2]), dtype=torch.complex128, device=self.dev)
            cm[self.dets[:, 0], self.dets[:, 1]] = c
            dv = (self.ea @ cm + cm @ self.eb.transpose(-1, -2)).reshape(self.na * self.na, -1)
            exc = (dv @ cm.reshape(-1).conj()).reshape(self.na, self.na)  # <E_ij>
            ok = torch.tensor([[a == b for b in self.m[self.nc:]] for a in self.m[self.nc:]], device=self.dev)
            d = d + (e[self.nc:, self.nc:] * exc * ok).sum().real
        return float(d)


def exact(case, seed):
    outs = []
    for wl in _workloads(case, int(seed)):
        mo = _Model(wl)
        orb, cic = _orbitals(wl, _grid(wl)), _ci(wl)
        mo.set_wfn0(orb)
        y, c = torch.as_tensor(orb, device=mo.dev), torch.as_tensor(cic, device=mo.dev)
        if case["kind"] in ("rhs", "rhs_host"):
            hw, hc, e = mo.htot(1.0, _fields(wl, int(seed)), y, c, 0)
            if case["kind"] == "rhs":
                return {"hwfn": hw, "hcic": hc}
            return {"hwfn": hw.cpu().numpy(), "hcic": hc.cpu().numpy(), "energies": np.array(e)}
        if case["kind"] == "relax":
            y, c, e = mo.relax(y, c, 0.01, case["steps"])
            return {"orb": y, "cic": c, "energy": np.array(e)}
        y, c = mo.split2(y, c, _start_time(wl, case["phase"]), case["steps"])
        if case["kind"] == "split2":
            out = {"orb": y, "cic": c}
            if case["dipole"]:
                out["dipole"] = mo.dipole(y, c)
            return out
        outs.append((y.reshape(-1), c))
    return {"orb": [o for o, _ in outs], "cic": [c for _, c in outs]}
