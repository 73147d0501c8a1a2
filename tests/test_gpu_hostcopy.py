"""Copies of large host buffers: bitwise what a plain copy brings, for one and several parts of the pinned ring, its
slots in use more than once, two threads at once, page-locked buffers and a bounded number of threads."""
import ctypes
import os
import subprocess
import sys
import threading

import numpy as np
import pytest

from td1c_b200 import workloads as W

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
MB = 1 << 20


def _copies():
    """The library's two copy functions (they are not part of its C interface)."""
    from td1c_b200 import _lib
    lib = _lib.load()
    vp, fns = ctypes.c_void_p, []
    for name in ("_ZN4td1c14host_to_deviceEPvPKvmP11CUstream_st", "_ZN4td1c14device_to_hostEPvPKvmP11CUstream_st"):
        f = getattr(lib, name)
        f.argtypes, f.restype = [vp, vp, ctypes.c_size_t, vp], ctypes.c_int
        fns.append(f)
    return fns


def _round_trip(h2d, d2h, n, seed, pinned=False):
    """Random bytes to the device and back on a stream of their own; True if they come back."""
    import torch
    src = torch.from_numpy(np.random.RandomState(seed).randint(0, 256, n, dtype=np.uint8))
    if pinned:
        src = src.pin_memory()
    dst = torch.zeros(n, dtype=torch.uint8, pin_memory=pinned)
    dev = torch.zeros(n, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    s = torch.cuda.Stream()
    assert h2d(dev.data_ptr(), src.data_ptr(), n, s.cuda_stream) == 0
    if not pinned:
        keep = src.clone()
        src.zero_()  # a pageable buffer is free once the call returns
        src = keep
    assert d2h(dst.data_ptr(), dev.data_ptr(), n, s.cuda_stream) == 0
    s.synchronize()
    return bool(torch.equal(dst, src))


SIZES = [1, 512 * 1024 - 1, 512 * 1024, 2 * MB, 2 * MB + 1, 3 * MB + 12345, 8 * MB, 8 * MB + 1, 9 * MB + 77, 16 * MB, 21 * MB + 5]


@pytest.mark.gpu
@pytest.mark.parametrize("pinned", [False, True])
def test_copies_of_every_number_of_parts(cuda_ok, pinned):
    h2d, d2h = _copies()
    for k, n in enumerate(SIZES):
        assert _round_trip(h2d, d2h, n, k, pinned), n


@pytest.mark.gpu
def test_copies_from_several_threads(cuda_ok):
    """One thread has the ring, the others find it in use."""
    h2d, d2h = _copies()
    bad = []

    def work(t):
        for k in range(6):
            if not _round_trip(h2d, d2h, SIZES[3 + (k + t) % 8], 100 * t + k):
                bad.append((t, k))
    threads = [threading.Thread(target=work, args=(t,)) for t in range(3)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad


@pytest.mark.gpu
@pytest.mark.parametrize("nfe,lmax", [(40, 27), (62, 47), (80, 63)])
def test_host_call_of_several_parts(cuda_ok, nfe, lmax):
    """States of 3.2, 8.6 and 14.7 MB (two parts, the first slot used twice, every slot used twice)."""
    import torch
    from td1c_b200 import basis
    from td1c_b200.hprod import HProd
    from td1c_b200.wfn import seeded_orbitals, seeded_cic
    wl = W.small(W.NE_CAS, rmax=2.0 * nfe, nfe=nfe, lmax1=lmax, lmax2=2 * lmax, rmask=1.6 * nfe)
    rad, ang = basis.build(wl)
    h = HProd(wl, rad, ang)
    try:
        tb = h.ci_tables()
        orb = seeded_orbitals(wl, rad["xrad"], rad["wrad"], rad["mask"])
        cic = seeded_cic(wl, h.dims["lcic"], tb["stra"], tb["strb"], tb["detoff"], tb["afirst"], tb["acount"])
        h.set_wfn0(orb, cic)
        lf = np.zeros(9)
        lf[2], lf[5], lf[8] = 1.2, 0.1, 1.2
        x, c = torch.from_numpy(orb.reshape(-1).copy()).cuda(), torch.from_numpy(cic.copy()).cuda()
        y, yc = torch.empty_like(x), torch.empty_like(c)
        torch.cuda.synchronize()
        h.htot_dev(1.0, lf, x.data_ptr(), c.data_ptr(), y.data_ptr(), yc.data_ptr())
        h.sync()
        for _ in range(3):
            hw, hc = h.htot(1.0, lf, orb, cic)
            assert np.array_equal(hw.reshape(-1), y.cpu().numpy()) and np.array_equal(hc, yc.cpu().numpy())
    finally:
        h.final()


THREADS = """
import os, sys, torch
sys.path.insert(0, %r)
from tests.test_gpu_hostcopy import _copies, _round_trip
h2d, d2h = _copies()
pinned = sys.argv[1] == "pinned"
assert _round_trip(h2d, d2h, 100, 0, False) and _round_trip(h2d, d2h, 100, 0, True)
torch.set_num_threads(1)
before = len(os.listdir("/proc/self/task"))
assert _round_trip(h2d, d2h, 9 << 20, 1, pinned)
print(len(os.listdir("/proc/self/task")) - before)
""" % ROOT


@pytest.mark.gpu
@pytest.mark.parametrize("kind,limit,most", [("pinned", "", 0), ("pageable", "1", 0), ("pageable", "3", 2), ("pageable", "", 7)])
def test_threads_of_the_host_copies(cuda_ok, kind, limit, most):
    """Page-locked buffers start none; pageable ones the number asked for."""
    env = dict(os.environ, OMP_NUM_THREADS="1", TD1C_HOST_THREADS=limit)
    r = subprocess.run([sys.executable, "-c", THREADS, kind], env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    started = int(r.stdout.split()[-1])
    want = min(most, len(os.sched_getaffinity(0)) - 1) if not limit else most
    assert started == want, (started, want)
