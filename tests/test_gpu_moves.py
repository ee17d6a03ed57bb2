"""What the handles' and engines' uploads and downloads wait for, and the
drivers' calls on host arrays of every kind."""
import ctypes as C
import threading
import time

import numpy as np
import pytest
import torch

from mlau_gb300 import ics

pytestmark = pytest.mark.gpu


def test_a_small_upload_does_not_wait_for_queued_steps(gpu_lib):
    """Arrays of 51 kB fit the driver's staging, so the call returns while the
    steps queued before it run (some 40 ms; the call takes microseconds)."""
    M = gpu_lib
    st, m = ics.turbulence_3d(n=12, ny=12, nz=8, mach=0.1, seed=1)
    ptrs = (C.POINTER(C.c_double) * 8)(*[M._ptr(st[k]) for k in M.VARS])
    with M.Sim(3, st["ro"].shape, dx=m["dx"], dy=m["dy"], dz=m["dz"], gamma=m["gamma"]) as s:
        s.upload(st)
        s.step(1e-6, 64)
        s.sync()
        s.step(1e-6, 64)
        t0 = time.perf_counter()
        assert M.lib().mlau_sim_upload(s._h, ptrs) == 0
        t1 = time.perf_counter()
        s.sync()
        t2 = time.perf_counter()
    assert t1 - t0 < 0.25 * (t2 - t0), (t1 - t0, t2 - t0)


class Load:
    """An engine whose step holds every SM for some 2 ms (FP32-split) or 30 ms
    (FP64), stepping in a thread of its own."""

    def __init__(self, M, precision):
        self.b = M.Batch.open(8 * 520 * 520, 8, precision=precision)
        for k in range(8):
            st, m = ics.turbulence_2d(n=512, seed=k, vrms=0.3)
            self.b.add(st, m["dx"], m["dy"], m["gamma"], "mlau", 0.3, 1e9)
        self.step_ms = self.b.run(4, steps_per_graph=4)[1] / 4
        self.stop = threading.Event()
        self.th = threading.Thread(target=self.loop)

    def loop(self):
        while not self.stop.is_set():
            self.b.run(4, steps_per_graph=4)

    def __enter__(self):
        self.th.start()
        return self

    def __exit__(self, *a):
        self.stop.set()
        self.th.join()
        self.b.close()


def median_ms(f, n=20):
    ms = []
    for _ in range(n):
        t0 = time.perf_counter()
        f()
        ms.append((time.perf_counter() - t0) * 1e3)
    return np.median(ms)


@pytest.mark.parametrize("precision", [0, 1])
def test_moves_do_not_wait_for_another_engines_step(gpu_lib, precision):
    M = gpu_lib
    st, m = ics.turbulence_2d(n=128, seed=9)
    with M.Batch.open(136 * 136, 1) as b, Load(M, precision) as load:
        k = b.add(st, m["dx"], m["dy"], m["gamma"], "mlau", 0.3, 1.0)
        ms = median_ms(lambda: (b.upload(k, st), b.download(k)))
        got = b.download(k)
    assert all(np.array_equal(got[v], st[v]) for v in got)
    assert ms < 0.5 * load.step_ms, (ms, load.step_ms)


def test_small_kernels_run_beside_the_fp64_engine(gpu_lib):
    """The FP64 engine's step leaves registers for a warp of other streams'
    kernels: an operator's 16 launches take less than one of its steps."""
    M = gpu_lib
    st, m = ics.turbulence_2d(n=112, seed=9)
    with M.Sim(2, st["ro"].shape, dx=m["dx"], dy=m["dy"], gamma=m["gamma"], odr=2) as s, Load(M, 0) as load:
        s.upload(st)
        ms = median_ms(lambda: (s.viscous(1e-3, 1e-9), s.sync()), 8)
    assert ms < 0.5 * load.step_ms, (ms, load.step_ms)


def _array(a, shift, pinned):
    n = a.size
    b = torch.empty(n + 2, dtype=torch.float64, pin_memory=True).numpy() if pinned else np.empty(n + 2)
    off = ((shift * 8 - b.ctypes.data) % 16) // 8
    b = b[off:off + n].reshape(a.shape)
    b[...] = a
    return b


@pytest.mark.parametrize("pinned", [False, True, "mixed"])
@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("shape", [(4, 4), (13, 9), (120, 248), (121, 247), (292, 293), (504, 1016), (505, 1017)])
def test_driver_calls_equal_the_handle(gpu_lib, shape, shift, pinned):
    """Arrays up to the sizes at which the moves change (256 KB, 4 MB) and above, at 16 bytes
    and 8 beyond, ordinary and pinned: the same bits as upload, step, download."""
    M = gpu_lib
    st, m = ics.turbulence_2d(n=shape[1], ny=shape[0], seed=3, vrms=0.4)
    M.set_scheme(2, 1, "lhlld", 1)
    try:
        with M.Sim(2, st["ro"].shape, dx=m["dx"], dy=m["dy"], gamma=m["gamma"], odr=1, flux="lhlld",
                   nrk=1) as s:
            s.upload(st)
            s.step(1e-3, 1)
            want = s.download()
        h = {k: _array(st[k], shift, pinned is True or (pinned == "mixed" and v % 2))
             for v, k in enumerate(M.VARS)}
        ny, nx = st["ro"].shape
        M.mhd_fd_ct_2d(*[h[k] for k in M.VARS], 1e-3, m["dx"], m["dy"], nx, ny, 4, 4, m["gamma"])
        assert all(np.array_equal(h[k], want[k]) for k in M.VARS)
    finally:
        M.release_dropin()
        M.set_scheme(2, 2, "lhlld", 3)
