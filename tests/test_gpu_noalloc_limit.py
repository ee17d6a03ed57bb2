"""mlau_fd4c_1d_noalloc at its largest grid, which fills its scratch to the last
double, against the handle API: the same bits."""
import ctypes as C

import numpy as np
import pytest

from mlau_gb300 import ics

pytestmark = pytest.mark.gpu

NX = 16392


@pytest.mark.parametrize("bc,odr,nrk", [("open", 2, 3), ("periodic", 4, 2), ("open", 1, 1)])
def test_largest_grid(gpu_lib, bc, odr, nrk):
    M = gpu_lib
    st, m = ics.riemann_1d(n=NX - 8, seed=4)
    dt = 0.05 * m["dx"]
    kw = dict(dx=m["dx"], gamma=m["gamma"], odr=odr, flux="lhlld", nrk=nrk)
    f = M.lib().mlau_fd4c_1d_noalloc
    d, i = C.c_double, C.c_int
    f.argtypes, f.restype = [C.c_void_p] * 7 + [d, d, d, i, i, d, i, i, i, i, C.c_void_p], i
    with M.Sim(1, (NX,), **kw) as ref, M.Sim(1, (NX,), **kw) as mem:
        for s in (ref, mem):
            s.set_bx(m["bx"])
            s.set_bc(bc)
            s.upload(st)
        v1 = ("ro", "mx", "my", "mz", "en", "by", "bz")
        for _ in range(2):
            assert f(*[mem.device_ptr(k) for k in v1], m["bx"], dt, m["dx"], NX, 4, m["gamma"], odr,
                     M.FLUX["lhlld"], nrk, M.BC1D[bc], mem.stream) == 0
            mem.sync()
            ref.step(dt, 1)
        got, want = mem.download(), ref.download()
    assert all(np.array_equal(got[k], want[k]) for k in want)
