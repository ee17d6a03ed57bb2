"""The FP32-split step's CT curl: the EMF difference on the integer pipe
(csrc/emf_diff.cuh) against doubles, and the update's cell numbering."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from mlau_gb300 import ics

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("emf") / "libemf.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC",
                    "-I" + os.path.join(ROOT, "mlau_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "c", "emf_diff_check.cpp"), "-o", out], check=True)
    f = C.CDLL(out).emf_diff_check
    f.argtypes, f.restype = [C.c_int, C.c_long, C.c_long], C.c_long
    return f


@pytest.mark.parametrize("kind", [0, 1, 2, 3])
def test_same_bits_as_doubles(check, kind):
    assert check(kind, 500000, 5 + kind) == 0


@pytest.mark.gpu
@pytest.mark.parametrize("prec", [1, 2])
@pytest.mark.parametrize("n", [(4, 9, 5), (31, 5, 4), (33, 12, 7), (130, 6, 5)])
def test_step_commutes_with_periodic_shifts(gpu_lib, n, prec):
    """Every cell is updated once, whatever its place in a block or row: a
    shifted periodic state gives the shifted result, bit for bit."""
    M = gpu_lib
    for odr in (2, 4):
        st, m = ics.turbulence_3d(n=n[0], ny=n[1], nz=n[2], mach=0.3, seed=2, odr=odr)
        core = (slice(4, -4),) * 3
        st = {k: ics.pad_periodic(np.ascontiguousarray(a[core]), 4) for k, a in st.items()}

        def run(s0):
            with M.Sim(3, s0["ro"].shape, dx=m["dx"], dy=m["dy"], dz=m["dz"], gamma=m["gamma"], odr=odr,
                       flux="mlau", precision=prec) as s:
                s.upload(s0)
                s.step(1e-3, 2)
                return {k: a[core] for k, a in s.download().items()}

        ref = run(st)
        shift = (n[2] // 2, 3, n[0] // 2 + 1)
        got = run({k: ics.pad_periodic(np.ascontiguousarray(np.roll(a[core], shift, (0, 1, 2))), 4)
                   for k, a in st.items()})
        assert all(np.array_equal(np.roll(ref[k], shift, (0, 1, 2)), got[k]) for k in ref), odr
